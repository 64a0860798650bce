"""Each kernel alone against a plain PyTorch reference of the same operation, at sizes other than
the tiny models': widths and vocabularies that are no power of two, head sizes in steps of 16,
odd head counts and groups, page sizes, windows, and inputs made so that a fault shows."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _tol(dtype):
    return dict(atol=2e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H", [8, 100, 1536, 3])
def test_embedding(dtype, H):
    from ginfer_b200 import ops
    V = 777
    w = torch.randn(V, H, device=DEV).to(dtype)
    ids = torch.tensor([0, V - 1, 5, 5, 123, 776, 1], dtype=torch.int32, device=DEV)
    assert torch.equal(ops.embedding(ids, w), w[ids.long()])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,eps", [(96, 1e-5), (1536, 1e-6), (130, 1e-3), (5000, 1e-6),
                                   (13000, 1e-6)])
def test_add_rmsnorm(dtype, H, eps):
    from ginfer_b200 import ops
    T = 37
    x32 = torch.randn(T, H, device=DEV) * 3
    delta = (torch.randn(T, H, device=DEV)).to(dtype)
    for gdt in ({torch.float32, dtype}):
        gamma = (1 + 0.1 * torch.randn(H, device=DEV)).to(gdt)
        # residual in fp32 plus a delta in the activation type
        s, n = ops.add_rmsnorm(x32, delta, gamma, eps)
        want_s = x32.double() + delta.double()
        assert s.dtype == torch.float32
        torch.testing.assert_close(s.double(), want_s, atol=1e-6, rtol=1e-6)
        rms = torch.sqrt((want_s ** 2).sum(-1, keepdim=True) / H + eps)
        want_n = want_s * gamma.double() / rms
        torch.testing.assert_close(n.double(), want_n, **_tol(dtype))
        # no delta, activation-typed x (the embedding's output): s is x itself
        xa = x32.to(dtype)
        s2, n2 = ops.add_rmsnorm(xa, None, gamma, eps)
        assert s2 is xa
        xd = xa.double()
        want2 = xd * gamma.double() / torch.sqrt((xd ** 2).sum(-1, keepdim=True) / H + eps)
        torch.testing.assert_close(n2.double(), want2, **_tol(dtype))
        # selected rows only, no sum wanted (the final norm at the rows that want logits)
        rows = torch.tensor([36, 0, 7, 7], dtype=torch.int32, device=DEV)
        s3, n3 = ops.add_rmsnorm(x32, delta, gamma, eps, rows=rows, want_sum=False)
        assert s3 is None
        torch.testing.assert_close(n3.double(), want_n[rows.long()], **_tol(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,rot", [(4, 2, 16, 16), (3, 1, 32, 32), (5, 5, 48, 24),
                                           (12, 2, 128, 128), (2, 1, 64, 0)])
def test_rope_kv_write(dtype, nh, nkv, hd, rot):
    from ginfer_b200 import ops
    T, P, pages_n, maxpos = 19, 4, 11, 300
    qkv = torch.randn(T, (nh + 2 * nkv) * hd, device=DEV).to(dtype)
    orig = qkv.clone()
    positions = torch.randint(0, maxpos, (T,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(pages_n * P, device=DEV)[:T].to(torch.int32)
    slots[3] = -1                                         # a token that is not to be written
    table = None
    if rot:
        half = rot // 2
        inv = 1.0 / (10000.0 ** (torch.arange(half, dtype=torch.float64) / half))
        ang = torch.arange(maxpos, dtype=torch.float64)[:, None] * inv[None, :]
        table = torch.cat([ang.cos(), ang.sin()], 1).float().to(DEV)
    pages = torch.full((2, pages_n, P, nkv, hd), 7.0, device=DEV).to(dtype)
    ops.rope_kv_write(qkv, table, rot, positions, slots, pages, nh, nkv, hd)

    def rotate(x):                                        # x [T, heads, hd], float64
        if not rot:
            return x
        half = rot // 2
        c = table[positions.long(), :half].double()[:, None, :]
        s = table[positions.long(), half:].double()[:, None, :]
        a, b = x[..., :half], x[..., half:rot]
        return torch.cat([a * c - b * s, a * s + b * c, x[..., rot:]], -1)
    o = orig.double()
    q_want = rotate(o[:, :nh * hd].reshape(T, nh, hd))
    k_want = rotate(o[:, nh * hd:(nh + nkv) * hd].reshape(T, nkv, hd))
    v_want = o[:, (nh + nkv) * hd:].reshape(T, nkv, hd)
    tol = _tol(dtype)
    torch.testing.assert_close(qkv[:, :nh * hd].double().reshape(T, nh, hd), q_want, **tol)
    assert torch.equal(qkv[:, (nh + nkv) * hd:], orig[:, (nh + nkv) * hd:])    # v untouched
    flatk = pages[0].reshape(pages_n * P, nkv, hd).double()
    flatv = pages[1].reshape(pages_n * P, nkv, hd).double()
    written = slots >= 0
    torch.testing.assert_close(flatk[slots[written].long()], k_want[written], **tol)
    torch.testing.assert_close(flatv[slots[written].long()], v_want[written], atol=0, rtol=0)
    untouched = torch.ones(pages_n * P, dtype=torch.bool, device=DEV)
    untouched[slots[written].long()] = False
    assert (flatk[untouched] == 7.0).all() and (flatv[untouched] == 7.0).all()
    # without a slot mapping nothing is written (a layer reading another layer's cache)
    pages2 = torch.full_like(pages, 7.0)
    ops.rope_kv_write(orig.clone(), table, rot, positions, None, pages2, nh, nkv, hd)
    assert (pages2 == 7.0).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_silu_mul(dtype):
    from ginfer_b200 import ops
    T, I = 13, 1001
    gu = (torch.randn(T, 2 * I, device=DEV) * 4).to(dtype)
    g, u = gu[:, 0::2].double(), gu[:, 1::2].double()
    want = g / (1 + torch.exp(-g)) * u
    torch.testing.assert_close(ops.silu_mul(gu).double(), want, **_tol(dtype))


@pytest.mark.parametrize("M,N,K", [(2, 8, 9), (1, 389, 96), (130, 2000, 408), (64, 64, 16),
                                   (257, 1001, 1000), (7, 3, 5)])
@pytest.mark.parametrize("bias", [False, True])
def test_gemm_f32_is_true_fp32(M, N, K, bias):
    from ginfer_b200.ops.linear import gemm_f32
    # values with 20 significant bits: a tf32 or bf16 product would lose them
    x = (torch.randn(M, K, device=DEV) * 1024).round() / 1024 + 1.0
    w = (torch.randn(N, K, device=DEV) * 1024).round() / 1024
    b = torch.randn(N, device=DEV) if bias else None
    got = gemm_f32(x, w, b)
    want = x.double() @ w.double().t() + (b.double() if bias else 0)
    torch.testing.assert_close(got.double(), want, atol=2e-5 * math.sqrt(K), rtol=2e-6)
    # a row's result does not depend on the other rows of the batch
    assert torch.equal(gemm_f32(x[:1].contiguous(), w, b), got[:1])


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("N,K,lda", [(33, 68, 68), (129, 64, 80), (1536, 1540, 1540), (4097, 260, 260),
                                     (32800, 132, 136), (40, 515, 519), (31, 4, 4)])
def test_gemm_f32_at_the_edges_of_its_kernels(M, N, K, lda):
    """Every row kernel and tile, with remainders of rows, columns, chunks and cluster shares, rows of
    A apart, 16-byte and 4-byte copies: close to 64 bits, and each row as if it were alone."""
    from ginfer_b200.ops.linear import gemm_f32
    g = torch.Generator(device=DEV).manual_seed(M * 31 + N)
    x = torch.randn(M, lda, device=DEV, generator=g)[:, :K]
    w = torch.randn(N, K, device=DEV, generator=g)
    b = torch.randn(N, device=DEV, generator=g)
    got = gemm_f32(x, w, b)
    # chains of at most K / 4 + 16 FMAs (even or odd k of a segment), their sum, at most 8 segments and the
    # bias: as many roundings of 2^-24, of partial sums that stay below sum |x w|
    bound = (K / 4 + 16 + 10) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t() + b.double().abs())
    assert ((got.double() - (x.double() @ w.double().t() + b.double())).abs() <= bound).all()
    for m in {0, M // 2, M - 1}:
        assert torch.equal(gemm_f32(x[m:m + 1], w, b), got[m:m + 1])


@pytest.mark.parametrize("M", [18, 25, 40, 41, 48, 49, 57, 72, 81, 97, 105, 113, 121, 164])
@pytest.mark.parametrize("N,K", [(130, 100), (1536, 264), (257, 77)])
def test_gemm_f32_multiplies_the_rows_that_are_there(M, N, K):
    """Last tiles with every number of rows a thread, chunks of K that end inside a stage: each row's sums as
    if it were alone."""
    from ginfer_b200.ops.linear import gemm_f32
    g = torch.Generator(device=DEV).manual_seed(M * 31 + N)
    x, w = torch.randn(M, K, device=DEV, generator=g), torch.randn(N, K, device=DEV, generator=g)
    got = gemm_f32(x, w)
    assert torch.equal(torch.cat([gemm_f32(x[m:m + 1], w) for m in range(M)]), got)
    bound = (K / 4 + 26) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    assert ((got.double() - x.double() @ w.double().t()).abs() <= bound).all()


@pytest.mark.parametrize("M", [17, 24, 26, 32, 33])
@pytest.mark.parametrize("N,K", [(130, 100), (1536, 264), (257, 77)])
def test_gemm_f32_around_the_rows_where_its_tiles_change(M, N, K):
    test_gemm_f32_multiplies_the_rows_that_are_there(M, N, K)


@pytest.mark.parametrize("M", [2, 20])
def test_gemm_f32_of_more_than_two_million_columns(M):
    """More tiles of columns than a grid's shorter sides hold."""
    from ginfer_b200.ops.linear import gemm_f32
    N, K = (65536 * 32 if M == 2 else 65536 * 128) + 5, 4
    g = torch.Generator(device=DEV).manual_seed(M)
    x, w = torch.randn(M, K, device=DEV, generator=g), torch.randn(N, K, device=DEV, generator=g)
    got = gemm_f32(x, w)
    for a in (0, N - 1000):
        want, size = (f(x.double()) @ f(w[a:a + 1000].double()).t() for f in (lambda t: t, torch.abs))
        assert ((got[:, a:a + 1000].double() - want).abs() <= 8 * 2.0 ** -24 * size).all()


def _paged_case(B_lens, q_lens, nh, nkv, hd, P, window, dtype, seed=0, spike=True):
    """Random paged cache and queries for requests with kv lengths ``B_lens`` whose last
    ``q_lens`` tokens are this step's queries.  Returns the kernel inputs and the plain result."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    B = len(B_lens)
    total_pages = sum(-(-n // P) for n in B_lens) + 5
    perm = torch.randperm(total_pages, generator=g).tolist()
    W = max(-(-n // P) for n in B_lens) + 2
    table = torch.full((B, W), -1, dtype=torch.int32)
    pages = torch.zeros(2, total_pages, P, nkv, hd)
    ks, vs, qs = [], [], []
    at = 0
    for b, n in enumerate(B_lens):
        k = torch.randn(n, nkv, hd, generator=g)
        v = torch.randn(n, nkv, hd, generator=g)
        q = torch.randn(q_lens[b], nh, hd, generator=g)
        if spike and n > 40:
            # one far key stands out for one query: scale them so that its score dominates
            far = 3 if window == 0 else max(0, n - min(window, n))   # the oldest visible key
            if window < 0:                                           # chunks of -window positions
                far = (n - 1) // -window * -window
            q[-1, 0] = 0
            q[-1, 0, 0] = 30.0
            k[far, 0] = 0
            k[far, 0, 0] = 30.0
        ks.append(k), vs.append(v), qs.append(q)
        for i in range(-(-n // P)):
            page = perm[at]
            at += 1
            table[b, i] = page
            m = min(P, n - i * P)
            pages[0, page, :m] = k[i * P:i * P + m]
            pages[1, page, :m] = v[i * P:i * P + m]
    pages = pages.to(dtype)
    qcat = torch.cat(qs).to(dtype)
    scale = 1.0 / math.sqrt(hd)
    want = []
    for b, n in enumerate(B_lens):
        k = pages[0].double().reshape(-1, nkv, hd)
        v = pages[1].double().reshape(-1, nkv, hd)
        idx = torch.tensor([table[b, c // P] * P + c % P for c in range(n)])
        kk, vv = k[idx], v[idx]
        q = qs[b].to(dtype).double()
        ql = q_lens[b]
        out = torch.empty(ql, nh, hd, dtype=torch.float64)
        for r in range(ql):
            p = n - ql + r
            lo = max(0, p - window + 1) if window > 0 else 0
            if window < 0:
                lo = p // -window * -window
            for h in range(nh):
                kvh = h // (nh // nkv)
                s = (kk[lo:p + 1, kvh] @ q[r, h]) * scale
                out[r, h] = torch.softmax(s, 0) @ vv[lo:p + 1, kvh]
        want.append(out)
    want = torch.cat(want).reshape(-1, nh * hd)
    # windowed layers have given back the pages no query of this step can see
    if window > 0:
        for b, n in enumerate(B_lens):
            first_visible = max(0, n - q_lens[b] - window + 1)
            table[b, :first_visible // P] = -1
    cu = [0]
    for ql in q_lens:
        cu.append(cu[-1] + ql)
    positions = torch.cat([torch.arange(n - ql, n) for n, ql in zip(B_lens, q_lens)])
    seq_of_token = torch.cat([torch.full((ql,), b) for b, ql in enumerate(q_lens)])
    dev = dict(
        q=qcat.reshape(-1, nh * hd).to(DEV), pages=pages.to(DEV), table=table.to(DEV),
        cu=torch.tensor(cu, dtype=torch.int32, device=DEV),
        kv_lens=torch.tensor(B_lens, dtype=torch.int32, device=DEV),
        positions=positions.to(torch.int32).to(DEV),
        seq_of_token=seq_of_token.to(torch.int32).to(DEV))
    return dev, want, scale


def _qkv(dev, nh, nkv, hd):
    """Queries as the first columns of a wider row, as the engine's joined projection has them."""
    T = dev["q"].shape[0]
    qkv = torch.full((T, (nh + 2 * nkv) * hd), float("nan"), dtype=dev["q"].dtype, device=DEV)
    qkv[:, :nh * hd] = dev["q"]
    return qkv


ATT_CASES = [
    # kv lens, q lens, nh, nkv, hd, page, window
    ([70, 5, 130], [70, 5, 130], 4, 2, 16, 16, 0),
    ([200, 64, 1], [3, 64, 1], 3, 1, 32, 8, 0),
    ([300, 129, 77], [100, 1, 77], 5, 5, 48, 4, 33),
    ([515, 260], [2, 260], 12, 2, 128, 16, 0),
    ([700, 90], [65, 90], 6, 3, 64, 16, 100),
    ([1100], [1100], 14, 2, 64, 32, 0),
    # head sizes that are no multiples of 32 or 64, and one of three 64-channel parts
    ([130, 40, 260], [130, 1, 37], 4, 2, 80, 16, 0),
    ([200, 33], [64, 33], 2, 1, 112, 8, 20),
    ([300, 70], [5, 70], 6, 2, 192, 16, 50),
    # a negative window: chunks of that many positions counted from position 0
    ([300, 129, 77], [100, 1, 77], 4, 2, 64, 16, -37),
    ([700, 90], [65, 90], 6, 3, 64, 16, -96),
    ([200, 33], [64, 33], 2, 1, 48, 8, -1),
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("case", ATT_CASES)
def test_paged_attention_simt(dtype, case):
    from ginfer_b200 import ops
    lens, qls, nh, nkv, hd, P, window = case
    dev, want, scale = _paged_case(lens, qls, nh, nkv, hd, P, window, dtype)
    out = ops.paged_attention_simt(_qkv(dev, nh, nkv, hd), dev["pages"], dev["table"],
                                   dev["seq_of_token"], dev["positions"], nh, nkv, hd, scale,
                                   window, P)
    tol = dict(atol=2e-5, rtol=1e-4) if dtype == torch.float32 else dict(atol=1e-2, rtol=2e-2)
    torch.testing.assert_close(out.double().cpu(), want, **tol)


@pytest.mark.parametrize("case", ATT_CASES)
def test_attention_bf16_prefill(case):
    from ginfer_b200.ops import attention_bf16
    lens, qls, nh, nkv, hd, P, window = case
    dev, want, scale = _paged_case(lens, qls, nh, nkv, hd, P, window, torch.bfloat16)
    out = attention_bf16.prefill(_qkv(dev, nh, nkv, hd), dev["pages"], dev["table"], dev["cu"],
                                 dev["kv_lens"], len(lens), max(qls), nh, nkv, hd, scale, window,
                                 P)
    torch.testing.assert_close(out.double().cpu(), want, atol=1e-2, rtol=2e-2)


TC_CASES = [
    # kv lens, q lens, nh, nkv, hd, page, window
    ([515, 260], [2, 260], 12, 2, 128, 16, 0),
    ([700, 90], [65, 90], 6, 3, 64, 16, 100),
    ([1100], [1100], 14, 2, 64, 32, 0),
    ([300, 129, 77, 1000], [300, 1, 77, 129], 4, 4, 128, 8, 0),
    ([640, 400], [128, 400], 2, 1, 128, 16, 200),
    ([2048], [2048], 4, 2, 128, 16, 0),
    # many key tiles per query tile: pairs of CTAs share them (also with a window, and where the
    # second CTA's keys are all behind the window's start for the first rows)
    ([1800, 900], [700, 900], 6, 2, 128, 16, 700),
    ([3000], [130], 4, 1, 64, 8, 0),
    # chunks (a negative window): shorter and longer than a key tile, and of one position
    ([700, 90], [65, 90], 6, 3, 64, 16, -96),
    ([1800, 900], [700, 900], 6, 2, 128, 16, -700),
    ([640, 400], [128, 400], 2, 1, 128, 16, -50),
    ([300], [300], 2, 2, 64, 16, -1),
]


@pytest.mark.parametrize("case", TC_CASES)
def test_attention_tcgen05_prefill(case):
    from ginfer_b200.ops import attention_bf16, gemm_bf16
    lens, qls, nh, nkv, hd, P, window = case
    dev, want, scale = _paged_case(lens, qls, nh, nkv, hd, P, window, torch.bfloat16)
    out = attention_bf16.prefill_tc(_qkv(dev, nh, nkv, hd), dev["pages"], dev["table"], dev["cu"],
                                    dev["kv_lens"], len(lens), max(qls), nh, nkv, hd, scale,
                                    window, P)
    assert out is not None
    gemm_bf16.check_errors()
    torch.testing.assert_close(out.double().cpu(), want, atol=1e-2, rtol=2e-2)


@pytest.mark.parametrize("case", [TC_CASES[1], TC_CASES[5], TC_CASES[6]])
@pytest.mark.parametrize("every", [4, 2])
def test_attention_tcgen05_prefill_with_a_share_of_exponentials_by_polynomial(case, every):
    """The build that computes every n-th exponential of an unmasked tile by a cubic on the FMA
    pipe (off by default) against the oracle and against the default build."""
    from ginfer_b200.ops import attention_bf16, gemm_bf16
    lens, qls, nh, nkv, hd, P, window = case
    dev, want, scale = _paged_case(lens, qls, nh, nkv, hd, P, window, torch.bfloat16)
    args = (_qkv(dev, nh, nkv, hd), dev["pages"], dev["table"], dev["cu"], dev["kv_lens"],
            len(lens), max(qls), nh, nkv, hd, scale, window, P)
    out = attention_bf16.prefill_tc(*args, poly_exp_every=every)
    assert out is not None
    gemm_bf16.check_errors()
    torch.testing.assert_close(out.double().cpu(), want, atol=1e-2, rtol=2e-2)
    plain = attention_bf16.prefill_tc(*args, poly_exp_every=0)
    torch.testing.assert_close(out.float(), plain.float(), atol=1e-2, rtol=2e-2)


DEC_CASES = [
    ([70, 5, 130, 1], 4, 2, 16, 16, 0),
    ([200, 64, 1, 63, 65], 3, 1, 32, 8, 0),
    ([300, 129, 77], 5, 5, 48, 4, 33),
    ([515, 260, 4000], 12, 2, 128, 16, 0),
    ([700, 90], 6, 3, 64, 16, 100),
    ([2049, 17], 40, 2, 64, 16, 0),               # 20 query heads per kv head: two chunks of 16
    ([130, 40, 700], 6, 2, 80, 16, 0),            # five steps of 16 channels
    ([300, 70], 6, 2, 192, 8, 50),
    ([700, 90, 97], 6, 3, 64, 16, -96),           # chunks; the last request sees its own key only
    ([300, 129, 77], 5, 5, 48, 4, -33),
]


@pytest.mark.parametrize("case", DEC_CASES)
@pytest.mark.parametrize("splits", [1, 2, 5, 8, 16, -4])
def test_attention_bf16_decode(case, splits):
    from ginfer_b200.ops import attention_bf16
    lens, nh, nkv, hd, P, window = case
    qls = [1] * len(lens)
    dev, want, scale = _paged_case(lens, qls, nh, nkv, hd, P, window, torch.bfloat16)
    # 2, 4, 8, 16 merge inside a cluster; other counts (and negative ones here) through scratch
    out = attention_bf16.decode(_qkv(dev, nh, nkv, hd), dev["pages"], dev["table"], dev["cu"],
                                dev["positions"], len(lens), nh, nkv, hd, scale, window, P,
                                abs(splits), through_scratch=splits < 0)
    torch.testing.assert_close(out.double().cpu(), want, atol=1e-2, rtol=2e-2)


DEC_TMA_CASES = [   # what the kernel that loads by TMA serves: page sizes and head sizes
    ([300, 64, 1, 65, 129], 8, 1, 128, 8, 0),
    ([1000, 130, 63], 14, 2, 64, 32, 0),
    ([700, 257, 64], 16, 2, 128, 64, 300),
    ([900, 5], 4, 4, 256, 128, 0),
    ([1500, 700], 6, 3, 128, 16, 130),           # a window that starts inside a tile
    ([4100], 18, 2, 64, 16, 0),                   # 9 query heads per kv head: two chunks of 8
    ([300, 70, 8], 4, 2, 256, 8, 0),              # 64 boxes a tile: two for each lane of the loader
    ([600, 70, 9], 6, 2, 192, 16, 40),            # three 64-channel parts a row
    ([1500, 700, 1441], 6, 3, 128, 16, -130),     # chunks that start inside a tile
    ([961, 960], 4, 2, 64, 16, -96),              # the first and the last position of a chunk
]


@pytest.mark.parametrize("case", DEC_TMA_CASES)
@pytest.mark.parametrize("splits", [1, 2, 4, 8, 16])
def test_attention_bf16_decode_with_tiles_by_tma(case, splits):
    """The decode kernel that loads by TMA against the oracle and against the kernel that gathers
    with 16-byte copies (the same arithmetic in another tile layout: equal within rounding)."""
    from ginfer_b200.ops import attention_bf16, gemm_bf16
    lens, nh, nkv, hd, P, window = case
    dev, want, scale = _paged_case(lens, [1] * len(lens), nh, nkv, hd, P, window, torch.bfloat16)
    args = (_qkv(dev, nh, nkv, hd), dev["pages"], dev["table"], dev["cu"], dev["positions"],
            len(lens), nh, nkv, hd, scale, window, P, splits)
    assert attention_bf16.tma_serves(hd, P, splits)
    out = attention_bf16.decode(*args)
    gemm_bf16.check_errors()
    torch.testing.assert_close(out.double().cpu(), want, atol=1e-2, rtol=2e-2)
    other = attention_bf16.decode(*args, use_tma=False)
    torch.testing.assert_close(out.float(), other.float(), atol=1e-2, rtol=2e-2)


@pytest.mark.parametrize("case", [DEC_TMA_CASES[0], DEC_TMA_CASES[2], DEC_TMA_CASES[4],
                                  DEC_TMA_CASES[5], ([9000, 300, 2100], 12, 2, 128, 16, 0)])
@pytest.mark.parametrize("splits,parts", [(8, 2), (8, 5), (4, 3), (1, 4), (8, 16)])
def test_attention_bf16_decode_with_several_clusters_a_request(case, splits, parts):
    """Few requests with many keys: several clusters share a request's keys and a second kernel
    adds their results up.  Against the oracle and against one cluster a request; parts that get
    no key at all (more pieces than tiles) count for nothing."""
    from ginfer_b200.ops import attention_bf16, gemm_bf16
    lens, nh, nkv, hd, P, window = case
    dev, want, scale = _paged_case(lens, [1] * len(lens), nh, nkv, hd, P, window, torch.bfloat16)
    args = (_qkv(dev, nh, nkv, hd), dev["pages"], dev["table"], dev["cu"], dev["positions"],
            len(lens), nh, nkv, hd, scale, window, P, splits)
    out = attention_bf16.decode(*args, parts=parts)
    gemm_bf16.check_errors()
    torch.testing.assert_close(out.double().cpu(), want, atol=1e-2, rtol=2e-2)
    one = attention_bf16.decode(*args)
    torch.testing.assert_close(out.float(), one.float(), atol=1e-2, rtol=2e-2)


@pytest.mark.parametrize("window", [0, 70, -128])
@pytest.mark.parametrize("splits,parts", [(8, 1), (2, 1), (8, 2), (1, 3)])
def test_attention_bf16_decode_of_few_keys(splits, parts, window):
    """Requests whose keys one CTA holds (it writes the result itself) beside requests with one key more, with
    as many as all splits take, with a window and with chunks."""
    from ginfer_b200.ops import attention_bf16, gemm_bf16
    lens, nh, nkv, hd, P = [1, 63, 64, 65, 127, 128, 129, 130, 200, 256, 257, 1030], 6, 2, 64, 16
    dev, want, scale = _paged_case(lens, [1] * len(lens), nh, nkv, hd, P, window, torch.bfloat16)
    out = attention_bf16.decode(_qkv(dev, nh, nkv, hd), dev["pages"], dev["table"], dev["cu"], dev["positions"],
                                len(lens), nh, nkv, hd, scale, window, P, splits, parts=parts)
    gemm_bf16.check_errors()
    torch.testing.assert_close(out.double().cpu(), want, atol=1e-2, rtol=2e-2)


@pytest.mark.parametrize("keys,splits", [(129, 8), (192, 4), (200, 4), (256, 8), (300, 8), (512, 8)])
def test_attention_bf16_decode_gives_a_split_one_tile_while_there_are_splits(keys, splits):
    """Above the keys that one CTA takes and up to a tile a split, the probabilities are rounded against the largest
    score of their warp's sixteen keys, of which it has no more: the same values computed in 64 bits from such
    groups.  (With a second tile a split a warp's probabilities follow its running maximum: about a quarter of the
    bf16 results are then others.)"""
    from ginfer_b200.ops import attention_bf16, gemm_bf16
    nh, nkv, hd, P, B = 12, 2, 128, 16, 4
    g = torch.Generator(device=DEV).manual_seed(keys)
    n = -(-keys // P)
    pages = torch.randn(2, B * n, P, nkv, hd, device=DEV, generator=g).bfloat16()
    table = torch.arange(B * n, device=DEV, dtype=torch.int32).view(B, n)
    qkv = torch.randn(B, (nh + 2 * nkv) * hd, device=DEV, generator=g).bfloat16()
    out = attention_bf16.decode(qkv, pages, table, torch.arange(B + 1, device=DEV, dtype=torch.int32),
                                torch.full((B,), keys - 1, device=DEV, dtype=torch.int32), B, nh, nkv, hd,
                                hd ** -0.5, 0, P, splits).view(B, nh, hd)
    gemm_bf16.check_errors()
    k, v = (t.view(B, n * P, nkv, hd)[:, :keys].double().repeat_interleave(nh // nkv, 2) for t in pages)
    s = torch.einsum("bhd,bkhd->bhk", qkv[:, :nh * hd].view(B, nh, hd).double(), k) * (hd ** -0.5 / math.log(2))
    s = torch.nn.functional.pad(s, (0, -keys % 16), value=-math.inf).unflatten(2, (-1, 16))
    m = s.amax(3, keepdim=True)
    p, weight = torch.exp2(s - m), torch.exp2(m - m.amax(2, keepdim=True))
    v = torch.nn.functional.pad(v, (0, 0, 0, 0, 0, -keys % 16)).unflatten(1, (-1, 16))
    want = torch.einsum("bhgk,bgkhd->bhd", p.float().bfloat16().double() * weight, v) / (p * weight).sum((2, 3))[..., None]
    # a result that another rounding of fp32 sums moves over the middle between two bf16 values: one in some hundred
    assert (out == want.float().bfloat16()).float().mean() > 0.95


@pytest.mark.parametrize("case", DEC_CASES)
@pytest.mark.parametrize("splits", [1, 4, 8, -3])
@pytest.mark.parametrize("rot_frac", [1.0, 0.5])
def test_attention_bf16_decode_rotates_and_writes_the_cache_itself(case, splits, rot_frac):
    """The decode kernel given unrotated q and k equals the rotation-and-write kernel followed by
    the decode kernel, bit for bit in the cache and in the output."""
    from ginfer_b200 import ops
    from ginfer_b200.ops import attention_bf16
    lens, nh, nkv, hd, P, window = case
    B = len(lens)
    dev, _, scale = _paged_case(lens, [1] * B, nh, nkv, hd, P, window, torch.bfloat16, spike=False)
    g = torch.Generator().manual_seed(5)
    qkv = torch.randn(B, (nh + 2 * nkv) * hd, generator=g).to(torch.bfloat16).cuda()
    rot = int(hd * rot_frac) // 2 * 2
    ang = torch.rand(max(lens) + 1, rot // 2, generator=g) * 6.28
    table = torch.cat([ang.cos(), ang.sin()], dim=1).float().cuda().contiguous()
    slots = torch.tensor([int(dev["table"][b, (n - 1) // P]) * P + (n - 1) % P
                          for b, n in enumerate(lens)], dtype=torch.int32).cuda()
    # separately: rotate q in place, write k and v, then attend
    qkv_a, pages_a = qkv.clone(), dev["pages"].clone()
    ops.rope_kv_write(qkv_a, table, rot, dev["positions"], slots, pages_a, nh, nkv, hd)
    want = attention_bf16.decode(qkv_a, pages_a, dev["table"], dev["cu"], dev["positions"], B, nh,
                                 nkv, hd, scale, window, P, abs(splits),
                                 through_scratch=splits < 0)
    # in one kernel
    pages_b = dev["pages"].clone()
    got = attention_bf16.decode(qkv.clone(), pages_b, dev["table"], dev["cu"], dev["positions"],
                                B, nh, nkv, hd, scale, window, P, abs(splits),
                                through_scratch=splits < 0, rope=(table, rot, True))
    torch.cuda.synchronize()
    assert torch.equal(pages_b, pages_a), "the cache differs"
    assert torch.equal(got, want)
    # without the write, the cache stays as it was
    pages_c = dev["pages"].clone()
    attention_bf16.decode(qkv.clone(), pages_c, dev["table"], dev["cu"], dev["positions"], B, nh,
                          nkv, hd, scale, window, P, abs(splits), through_scratch=splits < 0,
                          rope=(table, rot, False))
    torch.cuda.synchronize()
    assert torch.equal(pages_c, dev["pages"])


def test_attention_refuses_head_sizes_it_cannot_take():
    from ginfer_b200 import ops
    from ginfer_b200.ops import attention_bf16
    assert not attention_bf16.supports(40, 4, 2) and not attention_bf16.supports(272, 4, 2)
    assert attention_bf16.supports(48, 5, 5) and attention_bf16.supports(256, 8, 1)
    dev, _, scale = _paged_case([20], [20], 2, 1, 16, 16, 0, torch.float32, spike=False)
    q = torch.zeros(20, 2 * 272 * 2, device=DEV)
    with pytest.raises(ValueError, match="head sizes up to 256"):
        ops.paged_attention_simt(q, torch.zeros(2, 4, 16, 1, 272, device=DEV), dev["table"],
                                 dev["seq_of_token"], dev["positions"], 2, 1, 272, scale, 0, 16)


@pytest.mark.parametrize("V", [256, 389, 151936, 7])
def test_argmax_lowest_index_wins(V):
    from ginfer_b200 import ops
    x = torch.randn(6, V, device=DEV)
    x[1, V - 1] = 50.0
    x[2, 0] = 50.0
    x[3, [V // 2, V // 3, V - 1]] = 60.0                  # a tie: the lowest index wins
    x[4] = -3.0                                           # all equal: index 0
    x[5, 1] = float("nan")                                # NaN never wins
    got = ops.argmax(x).tolist()
    want = [int(x[0].argmax()), V - 1, 0, V // 3, 0,
            int(torch.where(torch.isnan(x[5]), torch.tensor(-1e30, device=DEV), x[5]).argmax())]
    assert got == want


@pytest.mark.parametrize("V", [389, 5000, 151936])
def test_temperature_sampling_is_the_inverse_cdf(V):
    from ginfer_b200 import ops
    R = 64
    g = torch.Generator(device="cpu").manual_seed(V)
    logits = (torch.randn(R, V, generator=g) * 3).to(DEV)
    temps = torch.full((R,), 0.8, device=DEV)
    temps[0] = 0.0                                        # greedy row inside a sampled batch
    temps[1] = 1e-3                                       # nearly greedy
    u = torch.rand(R, generator=g).to(DEV)
    u[2], u[3] = 0.0, 0.99999994
    got = ops.sample(logits, temps, u).tolist()
    assert got[0] == int(logits[0].argmax()) and got[1] == int(logits[1].argmax())
    for r in range(2, R):
        p = torch.softmax(logits[r].double() / float(temps[r]), -1)
        cdf = torch.cumsum(p, 0)
        want = min(int(torch.searchsorted(cdf, u[r].double())), V - 1)
        if got[r] != want:                                # u within rounding of a CDF step
            lo, hi = sorted((got[r], want))
            assert float(cdf[hi - 1] - cdf[lo]).__abs__() < 1e-5 or \
                abs(float(cdf[lo]) - float(u[r])) < 1e-5, (r, got[r], want)
    # the distribution: many draws of one row follow softmax
    row = torch.tensor([[2.0, 1.0, 0.0, -1.0, 0.5]], device=DEV).repeat(4000, 1)
    us = torch.rand(4000, generator=g).to(DEV)
    picks = ops.sample(row, torch.full((4000,), 0.7, device=DEV), us)
    freq = torch.bincount(picks.long(), minlength=5).double() / 4000
    want = torch.softmax(row[0].double() / 0.7, -1).cpu()
    assert (freq.cpu() - want).abs().max() < 0.03


@pytest.mark.parametrize("K,F,T,E,top", [(8, 2, 1, 1, 1), (72, 34, 40, 3, 2), (1024, 704, 2, 16, 2),
                                         (1416, 136, 33, 5, 3), (4096, 64, 20, 4, 1), (2048, 2112, 9, 32, 4),
                                         (128, 50, 384, 7, 2)])
def test_grouped_products_that_stream_the_weights(K, F, T, E, top):
    """One pair to several tiles of an expert, reductions that are no multiple of a step, fewer weight
    rows than a warp takes, one to eight warps a reduction: against 64 bits."""
    from ginfer_b200.ops import moe
    g = torch.Generator(device=DEV).manual_seed(K + F)
    x = torch.randn(T, K, generator=g, device=DEV).bfloat16()
    up = (torch.randn(E, F, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    gate_up = (torch.randn(E, 2 * F, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    idx = torch.rand(T, E, generator=g, device=DEV).argsort(1)[:, :top].int()
    idx[: T // 2, 0] = 0                                   # a crowded expert (twice in a row is no matter)
    wgt = torch.rand(T, top, generator=g, device=DEV) + 0.2
    plan = moe.Plan(idx, E, "few")
    tok, exp = torch.arange(T, device=DEV).repeat_interleave(top), idx.reshape(-1).long()
    place = plan.pos_of_pair.long()
    eps = 2.0 ** -8                                        # of a rounding to bf16: half of 2^-7, eight digits
    acc = K * 2.0 ** -24                                   # of K sums in fp32, relative to sum |x w|
    z = torch.einsum("pk,pfk->pf", x[tok].double(), up[exp].double()) * wgt.reshape(-1, 1).double()
    size = torch.einsum("pk,pfk->pf", x[tok].double().abs(), up[exp].double().abs()) * wgt.reshape(-1, 1)
    # u = relu(z) is rounded once (and z summed in fp32), u^2 again
    want, off = z.relu() ** 2, (z.abs() * eps + acc * size)
    got = moe.grouped_relu2(x, up, plan, wgt)[place].double()
    assert ((got - want).abs() <= (2 * z.abs() + off) * off + eps * (z.abs() + off) ** 2 + 1e-37).all()
    # the gated form with its clamp far away: s(g) u, s with a slope of at most 1.1
    h = torch.einsum("pk,pfk->pf", x[tok].double(), gate_up[exp].double())
    hs = torch.einsum("pk,pfk->pf", x[tok].double().abs(), gate_up[exp].double().abs())
    gt, u = h[:, 0::2], h[:, 1::2]
    og, ou = gt.abs() * eps + acc * hs[:, 0::2], u.abs() * eps + acc * hs[:, 1::2]
    s = gt * torch.sigmoid(gt)
    got = moe.grouped_glu(x, gate_up, plan, 1e9, 1.0, 0.0)[place].double()
    off = 1.1 * og * (u.abs() + ou) + s.abs() * ou
    assert ((got - s * u).abs() <= off + eps * ((s * u).abs() + off) + 1e-6).all()
    y = moe.grouped_relu2(x, up, plan, wgt)
    down = (torch.randn(E, K, F, generator=g, device=DEV) * F ** -0.5).bfloat16()
    if F % 8 == 0:
        got = moe.grouped_down(y, down, plan)[place].double()
        yp = y[place].double()
        want = torch.einsum("pf,pkf->pk", yp, down[exp].double())
        size = torch.einsum("pf,pkf->pk", yp.abs(), down[exp].double().abs())
        assert ((got - want).abs() <= (F + 8) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("K,N", [(8, 2), (264, 38), (1024, 16), (1032, 34), (2056, 20), (4096, 10)])
@pytest.mark.parametrize("counts", [(1, 2, 3, 4, 0, 5), (8, 9, 0, 1, 1, 1), (0, 0, 20, 0, 0, 0), (0, 0, 0, 0, 0, 1)])
def test_products_of_a_handful_of_pairs(K, N, counts):
    """Tiles of every number of rows, reductions around a batch of 1,024 and a warp's 256, fewer items than
    warps: against 64 bits, and each pair as if it were alone."""
    from ginfer_b200.ops import moe
    g = torch.Generator(device=DEV).manual_seed(K + N)
    E, P = len(counts), sum(counts)
    idx = torch.tensor([e for e, n in enumerate(counts) for _ in range(n)])
    idx = idx[torch.randperm(P, generator=torch.Generator().manual_seed(K))].int().cuda().view(P, 1)
    x = torch.randn(P, K, generator=g, device=DEV).bfloat16()
    up = (torch.randn(E, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    plan = moe.Plan(idx, E, "gemv")
    rows = moe.grouped_down(x[plan.pair_of_pos.long()].contiguous(), up, plan)[plan.pos_of_pair.long()]
    glu = moe.grouped_glu(x, up, plan, 1e9, 1.0, 0.0)[plan.pos_of_pair.long()]
    want = torch.einsum("pk,pnk->pn", x.double(), up[idx[:, 0].long()].double())
    size = torch.einsum("pk,pnk->pn", x.double().abs(), up[idx[:, 0].long()].double().abs())
    # a lane's chain of K / 32 products (rounded up to its 8 k) and five additions across the lanes
    assert ((rows.double() - want).abs() <= (K / 32 + 16) * 2.0 ** -24 * size).all()
    gate, lift = rows[:, 0::2].bfloat16().double(), rows[:, 1::2].bfloat16().double()
    ref = gate / (1 + torch.exp(-gate)) * lift
    assert ((glu.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-30).all()
    for p in {0, P // 2, P - 1}:
        one = moe.Plan(idx[p:p + 1].contiguous(), E, "gemv")
        assert torch.equal(moe.grouped_down(x[p:p + 1], up, one)[0], rows[p])
        assert torch.equal(moe.grouped_glu(x[p:p + 1], up, one, 1e9, 1.0, 0.0)[0], glu[p])


def test_products_of_a_handful_of_pairs_take_any_fp32_result():
    """A result that starts at an odd multiple of four bytes: its values, and nothing beside it."""
    from ginfer_b200.ops import moe
    g = torch.Generator(device=DEV).manual_seed(2)
    x = torch.randn(5, 264, generator=g, device=DEV).bfloat16()
    w = torch.randn(3, 38, 264, generator=g, device=DEV).bfloat16()
    plan = moe.Plan(torch.tensor([[0], [2], [0], [1], [2]], dtype=torch.int32, device=DEV), 3, "gemv")
    place = torch.full((5 * 38 + 2,), 7.0, device=DEV)
    assert place.data_ptr() % 8 == 0
    moe._gemm(x, w, plan, place[1:-1].view(5, 38), 0, 0.0, 0.0, 0.0)
    assert torch.equal(place[1:-1].view(5, 38), moe.grouped_down(x, w, plan))
    assert place[0] == 7 and place[-1] == 7


@pytest.mark.parametrize("E,K,N,counts", [
    (24, 2048, 1026, [1] * 24), (32, 1096, 2050, [0] * 20 + [17, 1, 2, 8, 9, 16, 0, 0, 0, 0, 0, 27]),
    (40, 2120, 1056, [2, 0] * 20), (30, 520, 4034, [3] * 10 + [1] * 20)])
def test_routed_products_of_one_or_two_pairs_an_expert(E, K, N, counts):
    """Equal runs of items over all SMs: runs that begin and end inside a tile or hold several, tiles of up to
    16 pairs and experts of more, reductions and rows that are no multiples of a step: against 64 bits, and the
    same bits for the same pairs in another step of that range."""
    from ginfer_b200.ops import moe
    g = torch.Generator(device=DEV).manual_seed(K + N)
    P = sum(counts)
    assert E <= P <= 2.5 * E and 2 * N * K >= 4 << 20
    idx = torch.tensor([e for e, n in enumerate(counts) for _ in range(n)])
    idx = idx[torch.randperm(P, generator=torch.Generator().manual_seed(K))].int().cuda().view(P, 1)
    x = torch.randn(P, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(E, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    wgt = torch.rand(P, 1, generator=g, device=DEV) + 0.5

    def run(idx, x, wgt):
        plan = moe.Plan(idx, E, "few")
        back = plan.pos_of_pair.long()
        return (moe.grouped_down(x[plan.pair_of_pos.long()].contiguous(), w, plan)[back],
                moe.grouped_glu(x, w, plan, 1e9, 1.0, 0.0)[back], moe.grouped_relu2(x, w, plan, wgt)[back])
    rows, glu, relu2 = run(idx, x, wgt)
    for at in range(0, P, 16):
        e = idx[at:at + 16, 0].long()
        want = torch.einsum("pk,pnk->pn", x[at:at + 16].double(), w[e].double())
        size = torch.einsum("pk,pnk->pn", x[at:at + 16].double().abs(), w[e].double().abs())
        # sums of 16 warps with two accumulators each: chains of K / 32 products at most, of fp32 in the tensor
        # cores (four a step), then 17 additions
        assert ((rows[at:at + 16].double() - want).abs() <= (K / 32 + 40) * 2.0 ** -23 * size).all()
    gate, lift = rows[:, 0::2].bfloat16().double(), rows[:, 1::2].bfloat16().double()
    ref = gate / (1 + torch.exp(-gate)) * lift
    assert ((glu.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-30).all()
    ref = (rows * wgt).bfloat16().double().clamp(min=0) ** 2
    assert ((relu2.double() - ref).abs() <= 2.0 ** -8 * ref).all()
    some = torch.arange(P - 1, -1, -1, device=DEV)[:max(E, P - 3)]
    for a, b in zip((rows, glu, relu2), run(idx[some].contiguous(), x[some].contiguous(), wgt[some].contiguous())):
        assert torch.equal(a[some], b)


@pytest.mark.parametrize("E,K,N,counts", [
    (24, 1288, 2050, [3] * 12 + [2] * 12), (32, 2056, 2114, [0] * 20 + [17, 1, 2, 8, 9, 16, 0, 0, 0, 0, 0, 27]),
    (16, 1288, 4098, [1] * 16), (64, 1280, 1642, [1, 2] * 32)])
def test_routed_products_whose_grid_takes_more_than_a_round(E, K, N, counts):
    """The same where blocks of (tile, weight rows) would come to more than fit at once: that is where equal runs
    of items serve."""
    test_routed_products_of_one_or_two_pairs_an_expert(E, K, N, counts)


@pytest.mark.parametrize("K,F,E,top", [(2048, 1408, 32, 4), (1024, 704, 16, 2), (256, 96, 8, 1)])
@pytest.mark.parametrize("counts", [(1, 2, 3, 5), (24, 25, 40, 100)])
def test_a_pairs_result_does_not_depend_on_the_batch(K, F, E, top, counts):
    """Up to 20 pairs, and up to 16 an expert: the first tokens' rows of a step are those of a shorter step, bit
    for bit."""
    from ginfer_b200.ops import moe
    g = torch.Generator(device=DEV).manual_seed(K)
    T = max(counts)
    x = torch.randn(T, K, generator=g, device=DEV).bfloat16()
    up = (torch.randn(E, 2 * F, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    down = (torch.randn(E, K, F, generator=g, device=DEV) * F ** -0.5).bfloat16()
    idx = torch.rand(T, E, generator=g, device=DEV).argsort(1)[:, :top].int()
    got = []
    for n in counts:
        assert (n * top <= 20) == (counts[0] == 1) and moe.kernel_for(x, n * top, (K, F), (F, K)) == "few"
        plan = moe.Plan(idx[:n].contiguous(), E, "few")
        y = moe.grouped_glu(x[:n], up, plan, 1e9, 1.0, 0.0)
        got.append((y[plan.pos_of_pair.long()], moe.grouped_down(y, down, plan)[plan.pos_of_pair.long()]))
    for n, (y, rows) in zip(counts, got):
        assert torch.equal(y, got[-1][0][:n * top]) and torch.equal(rows, got[-1][1][:n * top])


@pytest.mark.parametrize("H,G,D,Vd,lens,one", [
    (16, 16, 128, 128, [70, 9, 33, 5], 0), (16, 8, 100, 126, [8, 16, 1, 7], 0), (4, 4, 64, 64, [24, 3], 0),
    (2, 1, 40, 31, [17, 8, 9], 0), (3, 3, 128, 32, [1, 1, 1], 0), (2, 2, 96, 48, [9, 15, 8], 1),
    (1, 1, 128, 20, [3, 1, 8, 2, 9, 7, 16, 5] * 20, 0)])
def test_delta_rule_of_several_portions_is_that_of_each(H, G, D, Vd, lens, one):
    """Requests of a step share blocks, the longest first: outputs and states are, bit for bit, those of each
    request in a step of its own (the sums over the rows are one tree, wherever the request is), at lengths
    around the chunks of eight tokens, key sizes with rows that are not there and odd numbers of columns."""
    from types import SimpleNamespace
    from ginfer_b200.ops import delta
    g0 = torch.Generator().manual_seed(D + Vd)
    B, T = len(lens), sum(lens)
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, D, generator=g0), dim=-1).cuda() for _ in "qk")
    v, beta = torch.randn(T, H, Vd, generator=g0).cuda(), torch.rand(T, H, generator=g0).cuda()
    g = torch.rand(*((T, H) if one else (T, H, D)), generator=g0).cuda()
    state0 = torch.randn(B + 1, H * D * Vd + 1, generator=g0).cuda()
    slots = torch.randperm(B + 1, generator=g0)[:B]

    def run(requests):
        state = state0.clone()
        rows = torch.cat([torch.arange(sum(lens[:b]), sum(lens[:b + 1])) for b in requests]).cuda()
        own = [lens[b] for b in requests]
        ctx = SimpleNamespace(num_seqs=len(own), slot_ids=slots[requests].int().cuda(), max_q_len=max(own),
                              cu_seqlens_q=torch.tensor([0] + own).cumsum(0).int().cuda())
        return delta.recurrence(*(t[rows] for t in (q, k, v, g, beta)), state, ctx), state
    o, state = run(list(range(B)))
    for b in range(B):
        o1, state1 = run([b])
        assert torch.equal(o[sum(lens[:b]):sum(lens[:b + 1])], o1)
        assert torch.equal(state[slots[b]], state1[slots[b]])
    assert torch.equal(state[[i for i in range(B + 1) if i not in slots.tolist()]],
                       state0[[i for i in range(B + 1) if i not in slots.tolist()]])


@pytest.mark.parametrize("H,G,D,Vd,lens,one", [
    (16, 16, 128, 128, [7, 30, 8, 1, 16, 9], 0), (8, 4, 64, 62, [9, 2, 17, 8] * 5, 0), (8, 8, 36, 64, [3, 25] * 10, 0),
    (16, 16, 100, 128, [12, 1, 15, 8, 7], 1), (10, 10, 64, 31, [8, 4] * 15, 1)])
def test_delta_rule_of_many_portions(H, G, D, Vd, lens, one):
    """Where the requests' columns fill the device, portions of many tokens and single tokens run on different
    kernels with one order of the sums: a token a step gives the same bits, and the recurrence in 64 bits is
    within the rounding of D terms a sum over the tokens so far (decays below one)."""
    from types import SimpleNamespace
    from ginfer_b200.ops import delta
    g0 = torch.Generator().manual_seed(D + Vd)
    B, T = len(lens), sum(lens)
    assert B * H * -(-Vd // 32) >= 2 * 148
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, D, generator=g0), dim=-1) for _ in "qk")
    v, beta = torch.randn(T, H, Vd, generator=g0), torch.rand(T, H, generator=g0)
    g = torch.rand(*((T, H) if one else (T, H, D)), generator=g0)
    state0 = torch.randn(B, H * D * Vd, generator=g0)
    cu = torch.tensor([0] + lens).cumsum(0)

    def run(rows, own, state, longest):
        ctx = SimpleNamespace(num_seqs=B, slot_ids=torch.arange(B).int().cuda(), max_q_len=longest,
                              cu_seqlens_q=torch.tensor([0] + own).cumsum(0).int().cuda())
        return delta.recurrence(*(t[rows].cuda() for t in (q, k, v, g, beta)), state, ctx).cpu()
    state = state0.clone().cuda()
    o = run(torch.arange(T), lens, state, max(lens))
    if not one:                                    # (single tokens with a decay a head: a kernel of their own)
        n = min(lens)
        alone = state0.clone().cuda()
        for t in range(n):
            rows = cu[:-1] + t
            assert torch.equal(run(rows, [1] * B, alone, 1), o[rows])
    kv = torch.arange(H) // (H // G)
    for b in range(B):
        S = state0[b].double().view(H, D, Vd).clone()
        for t in range(int(cu[b]), int(cu[b + 1])):
            S = (g[t].double()[:, None, None] if one else g[t].double()[:, :, None]) * S
            u = beta[t].double()[:, None] * (v[t].double() - torch.einsum("hdv,hd->hv", S, k[t].double()[kv]))
            S = S + k[t].double()[kv][:, :, None] * u[:, None, :]
            want = torch.einsum("hdv,hd->hv", S, q[t].double()[kv])
            assert (o[t].double() - want).abs().max() <= 2.0 ** -24 * D * 8 * S.abs().max()
        got = state[b].cpu().double().view(H, D, Vd)
        assert (got - S).abs().max() <= 2.0 ** -24 * D * 8 * S.abs().max()


def _delta_step(H, G, D, Vd, lens, one=0):
    from types import SimpleNamespace
    from ginfer_b200.ops import delta
    g0 = torch.Generator(device=DEV).manual_seed(D + Vd + sum(lens))
    B, T = len(lens), sum(lens)
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, D, device=DEV, generator=g0), dim=-1) for _ in "qk")
    v, beta = torch.randn(T, H, Vd, device=DEV, generator=g0), torch.rand(T, H, device=DEV, generator=g0)
    g = torch.rand(*((T, H) if one else (T, H, D)), device=DEV, generator=g0)
    state0 = torch.randn(B, H * D * Vd, device=DEV, generator=g0)

    def step(rows=slice(None), own=lens, host=False):
        ctx = SimpleNamespace(num_seqs=len(own), slot_ids=torch.arange(len(own)).int().to(DEV), max_q_len=max(own),
                              cu_seqlens_q=torch.tensor([0] + list(own)).cumsum(0).int().to(DEV))
        if host:
            ctx.q_lens_host = list(own)
        given = [t[rows] for t in (q, k, v, g, beta)]
        return lambda state: delta.recurrence(*given, state, ctx)
    return step, state0


@pytest.mark.parametrize("H,G,D,Vd,lens", [
    (16, 16, 128, 128, [1] * 20 + [70, 9]), (16, 8, 100, 128, [1] * 20 + [17]), (8, 4, 64, 62, [1] * 40 + [90, 33]),
    (8, 8, 64, 64, [1] * 3 + [40, 5]), (16, 16, 64, 64, [1, 1, 30]), (16, 16, 128, 128, [1] * 30 + [3, 2]),
    (16, 16, 64, 64, [40, 33] * 10), (16, 16, 128, 64, [5, 4] * 20), (32, 32, 64, 64, [20, 17, 16])])
def test_delta_rule_of_single_tokens_in_front_of_portions(H, G, D, Vd, lens):
    """Whatever kernels share a step: known lengths or not, outputs and states are the same bits, and where there are
    many requests those of steps of one token each."""
    step, state0 = _delta_step(H, G, D, Vd, lens)
    states = [state0.clone() for _ in range(3)]
    o = step()(states[0])
    assert torch.equal(o, step(host=True)(states[1])) and torch.equal(*states[:2])
    if min(lens) > 1 and len(lens) * H * -(-Vd // 32) >= 2 * 148:
        at = torch.tensor([0] + lens).cumsum(0)[:-1].to(DEV)
        for t in range(min(lens)):
            assert torch.equal(step(at + t, [1] * len(lens))(states[2]), o[at + t])


@pytest.mark.parametrize("H,D,Vd,B,n,one", [(16, 128, 128, 512, 5, 0), (8, 64, 64, 512, 5, 0), (16, 64, 64, 256, 3, 1)])
def test_delta_rule_of_many_short_portions_costs_no_more_than_its_tokens_one_by_one(H, D, Vd, B, n, one):
    """Hundreds of requests with a handful of tokens each, as one step and as steps of one token: the step reads and
    writes the states once, so it may not take longer (with a third for what the steps do otherwise)."""
    step, state = _delta_step(H, H, D, Vd, [n] * B, one)
    at = torch.arange(B, device=DEV) * n
    whole, parts = step(), [step(at + t, [1] * B) for t in range(n)]

    def timed(steps):
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            torch.cuda._sleep(4000000)               # (the launches of all turns are there when the first begins)
            a.record()
            for _ in range(4):
                for f in steps:
                    f(state)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return sorted(times)[3]
    assert timed([whole]) <= 1.34 * timed(parts)


@pytest.mark.parametrize("H,G,D,Vd,lens", [(2, 1, 12, 20, [16, 1, 7]), (4, 2, 64, 64, [40, 8, 9, 3]),
                                           (2, 2, 128, 128, [33, 17]), (3, 3, 100, 36, [24, 25, 31, 1]),
                                           (2, 1, 256, 48, [65]), (1, 1, 128, 4, [1, 1, 23]),
                                           (8, 8, 128, 100, [17] * 6)])
def test_delta_rule_with_channel_decays(H, G, D, Vd, lens):
    """Portions of one token and of many, decays from none to all gone: outputs and states against the
    recurrence in 64 bits, and equal bit for bit however the portions are cut into steps (a router behind
    the layer makes close calls)."""
    from types import SimpleNamespace
    from ginfer_b200.ops import delta
    g0 = torch.Generator().manual_seed(D + Vd)
    B, T = len(lens), sum(lens)
    q = torch.randn(T, G, D, generator=g0) / D ** 0.5
    k = torch.nn.functional.normalize(torch.randn(T, G, D, generator=g0), dim=-1)
    v, beta = torch.randn(T, H, Vd, generator=g0), torch.rand(T, H, generator=g0)
    g = torch.rand(T, H, D, generator=g0)
    g[:, :, ::3] = 1.0 - g[:, :, ::3] * 0.01
    g[T // 2, :, 1::4] = 1e-30                              # a channel forgets all it held
    state0 = torch.randn(B + 2, H * D * Vd + 8, generator=g0)
    cu = torch.tensor([0] + lens).cumsum(0)
    slots = torch.randperm(B + 2, generator=g0)[:B]
    got = []
    for longest in (max(lens), 0):
        state = state0.clone().cuda()
        ctx = SimpleNamespace(num_seqs=B, slot_ids=slots.int().cuda(), cu_seqlens_q=cu.int().cuda(),
                              max_q_len=longest)
        o = delta.recurrence(q.cuda(), k.cuda(), v.cuda(), g.cuda(), beta.cuda(), state, ctx)
        got.append((o.cpu().double(), state.cpu()))
    # the same portions in two steps, and a token a step
    for at in ([max(n // 2, n - 16) for n in lens], None):
        state, o = state0.clone().cuda(), torch.empty_like(got[0][0])
        for step in range(2 if at else max(lens)):
            lo = [0 if not step else a for a in at] if at else [min(step, n) for n in lens]
            hi = [(at if not step else lens)[b] if at else min(step + 1, n) for b, n in enumerate(lens)]
            live = [b for b in range(B) if hi[b] > lo[b]]
            if len(live) < B and not at:              # (the kernel's lanes are chosen by the requests' number)
                break
            rows = torch.cat([torch.arange(int(cu[b]) + lo[b], int(cu[b]) + hi[b]) for b in live])
            ctx = SimpleNamespace(num_seqs=B, slot_ids=slots.int().cuda(), max_q_len=max(h - a for a, h in zip(lo, hi)),
                                  cu_seqlens_q=torch.tensor([0] + [h - a for a, h in zip(lo, hi)]).cumsum(0).int().cuda())
            part = delta.recurrence(*(t[rows].cuda() for t in (q, k, v, g, beta)), state, ctx).cpu().double()
            o[rows] = part
            assert torch.equal(part, got[0][0][rows])
        if at:
            assert torch.equal(o, got[0][0]) and torch.equal(state.cpu(), got[0][1])
    err = [0.0, 0.0]
    for b in range(B):
        S = state0[slots[b], :H * D * Vd].double().reshape(H, D, Vd).clone()
        kv = torch.arange(H) // (H // G)
        for t in range(int(cu[b]), int(cu[b + 1])):
            S = g[t].double()[:, :, None] * S
            u = beta[t].double()[:, None] * (v[t].double() - torch.einsum("hdv,hd->hv", S, k[t, kv].double()))
            S = S + k[t, kv].double()[:, :, None] * u[:, None]
            want = torch.einsum("hdv,hd->hv", S, q[t, kv].double())
            for i in range(2):
                err[i] = max(err[i], float((got[i][0][t] - want).abs().max()))
        for i in range(2):
            kept = got[i][1][slots[b]]
            err[i] = max(err[i], float((kept[:H * D * Vd].double() - S.reshape(-1)).abs().max()))
            assert torch.equal(kept[H * D * Vd:], state0[slots[b], H * D * Vd:])
    # values of a few units, sums of at most 256 products of unit vectors' channels in fp32
    assert err[0] <= 2e-5 and err[1] <= 2e-5, err
    rest = [s for s in range(B + 2) if s not in slots.tolist()]
    assert torch.equal(got[0][1][rest], state0[rest])


@pytest.mark.parametrize("slots", [[2], [0, 4, 1], list(range(69, -1, -1))])
def test_zero_slots_clears_the_named_slots_of_every_state(slots):
    """States of several types and slot sizes (whole 16 bytes, whole words, and neither), more slots than a
    launch names."""
    n = max(max(slots) + 2, 6)
    states = [torch.ones((n, 7), dtype=torch.int32, device=DEV), torch.ones((n, 1), dtype=torch.int32, device=DEV),
              torch.ones((n, 12345), device=DEV), torch.ones((n, 64), device=DEV),
              torch.ones((n, 3), dtype=torch.bfloat16, device=DEV), torch.ones((n, 5), dtype=torch.int8, device=DEV)]
    from ginfer_b200 import ops
    spans = torch.tensor([[t.data_ptr(), t.stride(0) * t.element_size()] for t in states], device=DEV)
    ops.zero_slots(spans, slots)
    for t in states:
        want = torch.ones(n, dtype=torch.bool, device=DEV)
        want[slots] = False
        assert torch.equal((t == 1).all(dim=1), want) and torch.equal((t == 0).all(dim=1), ~want)


def test_a_storage_clears_the_tensors_it_holds_now():
    """States of other types than the engine's own, and one that has been replaced since the last time."""
    from ginfer_b200.cache.storage import CacheStorage
    from ginfer_b200.parts.base import StateSpec
    st = CacheStorage({0: StateSpec((5, 3)), 1: StateSpec((3,), torch.bfloat16)}, [], [], 16, 4, torch.float32, DEV)
    for again in range(2):
        for t in st.state.values():
            t.fill_(1)
        st.reset_slots([1, 4])
        for t in st.state.values():
            assert t[[1, 4]].eq(0).all() and t[[0, 2, 3]].eq(1).all()
        st.state[0] = torch.empty_like(st.state[0])


@pytest.mark.parametrize("H,G,D,Vd,lens", [(2, 1, 12, 20, [64, 1, 7]), (4, 2, 64, 64, [80, 8, 9]),
                                           (2, 2, 128, 128, [66, 17]), (3, 3, 100, 36, [24, 65, 1]),
                                           (16, 16, 128, 48, [64, 3, 9, 70, 8, 1, 65, 64]), (1, 1, 32, 4, [71])])
def test_linear_attention_with_channel_decays_eight_tokens_at_a_time(monkeypatch, H, G, D, Vd, lens):
    """Rows of a wider projection, chunks whole and cut, one and two columns a lane, decays from none to all
    gone: outputs and states against the recurrence token by token in 64 bits."""
    from types import SimpleNamespace
    from ginfer_b200.ops import decay, delta
    g0 = torch.Generator().manual_seed(D + Vd)
    B, T = len(lens), sum(lens)
    q, k = torch.randn(T, G, D, generator=g0) / D ** 0.5, torch.randn(T, G, D, generator=g0) / D ** 0.5
    v, g = torch.randn(T, H, Vd, generator=g0), torch.rand(T, H, D, generator=g0)
    g[:, :, ::3] = 1.0 - g[:, :, ::3] * 0.01
    g[T // 2, :, 1::4] = 1e-30
    state0 = torch.randn(B + 2, H * D * Vd + 8, generator=g0)
    cu = torch.tensor([0] + lens).cumsum(0)
    slots = torch.randperm(B + 2, generator=g0)[:B]
    wide = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1), torch.ones(T, 4)], 1).cuda()
    qd, kd, vd = wide[:, :G * D], wide[:, G * D:2 * G * D], wide[:, 2 * G * D:2 * G * D + H * Vd]
    state = state0.clone().cuda()
    ctx = SimpleNamespace(num_seqs=B, slot_ids=slots.int().cuda(), cu_seqlens_q=cu.int().cuda(),
                          max_q_len=max(lens), q_lens_host=lens)
    o = decay.recurrence(qd, kd, vd, g.reshape(T, -1).cuda(), state, ctx, H, G, D, Vd)
    o, state = o.cpu().double().reshape(T, H, Vd), state.cpu()
    err, kv = 0.0, torch.arange(H) // (H // G)
    for b in range(B):
        S = state0[slots[b], :H * D * Vd].double().reshape(H, D, Vd).clone()
        for t in range(int(cu[b]), int(cu[b + 1])):
            S = g[t].double()[:, :, None] * S + k[t, kv].double()[:, :, None] * v[t].double()[:, None]
            err = max(err, float((o[t] - torch.einsum("hdv,hd->hv", S, q[t, kv].double())).abs().max()))
        err = max(err, float((state[slots[b], :H * D * Vd].double() - S.reshape(-1)).abs().max()))
        assert torch.equal(state[slots[b], H * D * Vd:], state0[slots[b], H * D * Vd:])
    # values of a few units (a state holds some 200 terms of at most one), fp32 sums of at most 128 of them
    assert err <= 2e-5, err
    # scratch for fewer heads than there are: a group of them after the other, the same bits
    for heads in {1, H // 2 + 1}:
        monkeypatch.setattr(decay, "CHANNELS_MAX_WORDS", delta.chunk_words(T, B, heads, D, 0))
        again = state0.clone().cuda()
        o2 = decay.recurrence(qd, kd, vd, g.reshape(T, -1).cuda(), again, ctx, H, G, D, Vd)
        assert torch.equal(o2.cpu().double().reshape(T, H, Vd), o) and torch.equal(again.cpu(), state)
    rest = [s for s in range(B + 2) if s not in slots.tolist()]
    assert torch.equal(state[rest], state0[rest])


@pytest.mark.parametrize("rule", ["linear", "delta"])
def test_what_is_no_number_stays_with_its_token_and_later_ones(rule):
    """Portions eight tokens at a time: a value that is infinite or no number leaves the outputs of earlier
    tokens, of other columns and of other requests as they were, and is not forgotten by later ones."""
    from types import SimpleNamespace
    from ginfer_b200.ops import decay, delta
    H, D, Vd, lens = 2, 32, 20, [70, 66]
    T, g0 = sum(lens), torch.Generator(device=DEV).manual_seed(5)
    q, k = (torch.randn(T, H, D, generator=g0, device=DEV) * D ** -0.5 for _ in range(2))
    v, beta = torch.randn(T, H, Vd, generator=g0, device=DEV), torch.rand(T, H, generator=g0, device=DEV)
    g = torch.rand(T, H * D if rule == "linear" else H, generator=g0, device=DEV) * 0.5 + 0.5
    ctx = SimpleNamespace(num_seqs=2, slot_ids=torch.tensor([1, 0], dtype=torch.int32, device=DEV), max_q_len=70,
                          cu_seqlens_q=torch.tensor([0, 70, 136], dtype=torch.int32, device=DEV), q_lens_host=lens)

    def run(v):
        state = torch.zeros(2, H * D * Vd, device=DEV)
        if rule == "delta":
            return delta.recurrence(q, k, v, g, beta, state, ctx), state.view(2, H, D, Vd)
        o = decay.recurrence(q.view(T, -1), k.view(T, -1), v.view(T, -1), g, state, ctx, H, H, D, Vd)
        return o.view(T, H, Vd), state.view(2, H, D, Vd)
    want, kept = run(v)
    for at in (3, 37, 64, 69):
        for bad in (float("nan"), float("inf")):
            w = v.clone()
            w[at, 1, 6] = bad
            o, state = run(w)
            hit = torch.zeros(T, H, Vd, dtype=torch.bool, device=DEV)
            hit[at:70, 1, 6] = True
            assert torch.equal(o[~hit], want[~hit]) and not o[hit].isfinite().any()
            away = torch.ones_like(state, dtype=torch.bool)
            away[1, 1, :, 6] = False
            assert torch.equal(state[away], kept[away]) and not state[~away].isfinite().any()


@pytest.mark.parametrize("C", [16, 48, 80, 512])
@pytest.mark.parametrize("lens", [[600], [700, 3, 64], [1000, 520, 1, 65]])
def test_shares_of_a_tokens_keys_are_put_together(C, lens):
    """Latent attention of few tokens over many keys in several shares, some of them empty, latent sizes that
    fill no warp: against 64 bits."""
    from types import SimpleNamespace
    from ginfer_b200.ops import latent
    B, H, page = len(lens), 5, 16
    assert latent.key_splits(B, H, max(lens)) > 1
    g = torch.Generator(device=DEV).manual_seed(C + B)
    W = -(-max(lens) // page)
    pages = torch.randn(B * W, page, 1, C, generator=g, device=DEV).bfloat16()
    table = torch.randperm(B * W, generator=g, device=DEV).int().view(B, W)
    q = torch.randn(H, B, C, generator=g, device=DEV).bfloat16().float()      # (the kernel rounds q to bf16)
    ctx = SimpleNamespace(seq_of_token=torch.arange(B, dtype=torch.int32, device=DEV), max_kv_len=max(lens),
                          positions=torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV))
    out = latent.attention(q, None, pages, None, table, ctx, 0, C ** -0.5, page).double()
    for b, n in enumerate(lens):
        c = pages[table[b].long()].reshape(-1, C)[:n].double()
        p = torch.softmax(q[:, b].double() @ c.t() * C ** -0.5, dim=-1)
        # probabilities and result are rounded to bf16: 2^-8 each, of at most sum p |c|
        assert ((out[:, b] - p @ c).abs() <= 2 * 2.0 ** -8 * (p @ c.abs()) + 1e-6).all()
    # a key that is no number makes its request's outputs none, whichever share it falls into
    for at in (0, lens[0] // 2, lens[0] - 1):
        bad = pages.clone()
        bad[int(table[0, at // page]), at % page, 0, 3] = float("nan")
        got = latent.attention(q, None, bad, None, table, ctx, 0, C ** -0.5, page).double()
        assert got[:, 0].isnan().all() and torch.equal(got[:, 1:], out[:, 1:])


@pytest.mark.parametrize("H,G,D,Vd,B", [(2, 1, 12, 20, 3), (4, 2, 64, 64, 1), (16, 16, 128, 128, 5), (3, 3, 100, 36, 2),
                                        (2, 1, 256, 48, 2), (1, 1, 200, 132, 1), (2, 2, 130, 8, 2), (64, 1, 128, 64, 2)])
@pytest.mark.parametrize("channels", [False, True])
@pytest.mark.parametrize("rule", ["delta", "linear", "scaled"])
def test_one_token_of_every_request_through_its_state(H, G, D, Vd, B, channels, rule):
    """Rows and columns that fill no block, keys of every size class, operands as columns of a wider row, a
    decay a head and a channel: against 64 bits; slots that are not named stay."""
    from types import SimpleNamespace
    from ginfer_b200.ops import delta
    g0 = torch.Generator(device=DEV).manual_seed(D + Vd + B)
    def rnd(*shape):
        return torch.randn(*shape, generator=g0, device=DEV)
    wide = rnd(B, 2 * G * D + H * Vd + 8)
    q, k = wide[:, :G * D], wide[:, G * D:2 * G * D]
    wide[:, :2 * G * D] *= D ** -0.5
    v = wide[:, 2 * G * D:2 * G * D + H * Vd] if G * D % 2 == 0 and wide.shape[1] % 4 == 0 else rnd(B, H * Vd)
    g = torch.rand(B, H * D if channels else H, generator=g0, device=DEV)
    beta, c, skip = torch.rand(B, H, generator=g0, device=DEV), rnd(B, H), rnd(H)
    state0 = rnd(B + 2, H * D * Vd + 8)
    slots = torch.randperm(B + 2, generator=g0, device=DEV)[:B]
    state, o = state0.clone(), torch.empty(B, H * Vd, device=DEV)
    ctx = SimpleNamespace(num_seqs=B, slot_ids=slots.int(),
                          cu_seqlens_q=torch.arange(B + 1, dtype=torch.int32, device=DEV))
    kw = dict(beta=beta) if rule == "delta" else dict(c=c, skip=skip) if rule == "scaled" else {}
    assert delta.state_step(q, k, v, g, state, ctx, H, G, D, Vd, o, **kw)
    kv = torch.arange(H, device=DEV) // (H // G)
    qd, kd = (t.double().reshape(B, G, D)[:, kv] for t in (q, k))
    vd, S = v.double().reshape(B, H, Vd), state0[slots, :H * D * Vd].double().reshape(B, H, D, Vd)
    S = S * (g.double().reshape(B, H, -1)[..., None])
    size = S.abs().sum(2).amax() + 8
    if rule == "delta":
        u = beta.double()[..., None] * (vd - torch.einsum("bhdv,bhd->bhv", S, kd))
    else:
        u = vd * (c.double()[..., None] if rule == "scaled" else 1.0)
    S = S + kd[..., None] * u[:, :, None]
    want = torch.einsum("bhdv,bhd->bhv", S, qd) + (skip.double()[:, None] * vd if rule == "scaled" else 0.0)
    # at most 256 products of a state of a few units and unit vectors' channels, summed in fp32
    tol = 2e-6 * float(size)
    assert float((o.double().reshape(B, H, Vd) - want).abs().max()) <= tol
    got = state[slots]
    assert float((got[:, :H * D * Vd].double() - S.reshape(B, -1)).abs().max()) <= tol
    assert torch.equal(got[:, H * D * Vd:], state0[slots, H * D * Vd:])
    rest = [i for i in range(B + 2) if i not in slots.tolist()]
    assert torch.equal(state[rest], state0[rest])


@pytest.mark.parametrize("rule", ["delta", "linear"])
@pytest.mark.parametrize("lens", [[1, 0, 1], [0, 1], [1, 1, 0, 0]])
def test_requests_without_a_token_keep_their_state(rule, lens):
    """Steps of single tokens in which some requests bring none, the last one among them: as if those were
    not in the step."""
    from types import SimpleNamespace
    from ginfer_b200.ops import decay, delta
    H, D, Vd, B, T = 2, 16, 8, len(lens), sum(lens)
    g0 = torch.Generator(device=DEV).manual_seed(B)
    q, k, v, state0 = (torch.randn(*s, generator=g0, device=DEV)
                       for s in ((T, H, D), (T, H, D), (T, H, Vd), (B + 1, H * D * Vd)))
    g, beta = torch.rand(T, H, generator=g0, device=DEV), torch.rand(T, H, generator=g0, device=DEV)
    got = []
    for who in (range(B), [b for b in range(B) if lens[b]]):
        ctx = SimpleNamespace(num_seqs=len(who), slot_ids=torch.tensor(who, dtype=torch.int32, device=DEV),
                              max_q_len=1, q_lens_host=[lens[b] for b in who],
                              cu_seqlens_q=torch.tensor([0] + [lens[b] for b in who], device=DEV).cumsum(0).int())
        state = state0.clone()
        if rule == "delta":
            o = delta.recurrence(q, k, v, g, beta, state, ctx)
        else:
            o = decay.recurrence(q.view(T, -1), k.view(T, -1), v.view(T, -1), g, state, ctx, H, H, D, Vd)
        got.append((o, state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    for b in range(B + 1):
        assert torch.equal(got[0][1][b], state0[b]) == (b == B or not lens[b])


@pytest.mark.parametrize("T,top,N", [(1, 1, 4), (3, 4, 2048), (5, 6, 516), (2, 9, 37), (40, 2, 130)])
@pytest.mark.parametrize("weighted", [False, True])
def test_pairs_rows_are_added_up_in_the_order_chosen(T, top, N, weighted):
    """Widths of quads and others, more choices than are asked for at a time, choices without a row: equal to
    the sum in that order in 32-bit."""
    from types import SimpleNamespace
    from ginfer_b200.ops import moe
    g = torch.Generator(device=DEV).manual_seed(N)
    y = torch.randn(T * top, N, generator=g, device=DEV)
    pos = torch.randperm(T * top, generator=g, device=DEV).int()
    pos[::5] = -1
    wgt = torch.rand(T, top, generator=g, device=DEV) if weighted else None
    got = moe.combine(y, SimpleNamespace(pos_of_pair=pos, top=top), wgt, T)
    want, size = torch.zeros(T, N, dtype=torch.float64, device=DEV), torch.zeros(T, N, device=DEV)
    for k in range(top):
        p = pos.view(T, top)[:, k].long()
        row = torch.where(p[:, None] >= 0, y[p.clamp(min=0)], 0.0) * (wgt[:, k:k + 1] if weighted else 1.0)
        want, size = want + row.double(), size + row.abs()
    assert ((got.double() - want).abs() <= top * 2.0 ** -23 * size).all()


@pytest.mark.parametrize("H,G,D,Vd,lens", [(8, 1, 128, 64, [64, 65, 200]), (6, 2, 36, 132, [130, 64]), (4, 2, 4, 4, [66]),
                                           (64, 1, 64, 64, [127])])
@pytest.mark.parametrize("norm", [False, True])
def test_heads_that_share_queries_and_keys_share_their_scores(H, G, D, Vd, lens, norm):
    """A chunk at a time with fewer key heads than heads: outputs, states and normalisers are, bit for bit,
    those of the same queries and keys written out for every head."""
    from types import SimpleNamespace
    from ginfer_b200.ops import decay
    g0 = torch.Generator(device=DEV).manual_seed(D + Vd)
    B, T = len(lens), sum(lens)
    q, k, v = (torch.randn(T, n, device=DEV, generator=g0) / D ** 0.5 for n in (G * D, G * D, H * Vd))
    g, c = torch.rand(T, H, device=DEV, generator=g0) ** 0.1, torch.rand(T, H, device=DEV, generator=g0)
    skip = torch.randn(H, device=DEV, generator=g0)
    state0 = torch.randn(B, (H * D * Vd + H * D + 3) // 4 * 4, device=DEV, generator=g0)
    ctx = SimpleNamespace(num_seqs=B, slot_ids=torch.arange(B).int().cuda(), max_q_len=max(lens), q_lens_host=lens,
                          cu_seqlens_q=torch.tensor([0] + lens).cumsum(0).int().cuda())
    got = []
    for heads in (G, H):
        state = state0.clone()
        qh, kh = (t.view(T, G, D).repeat_interleave(heads // G, 1).reshape(T, heads * D) for t in (q, k))
        o = decay.recurrence(qh, kh, v, g, state, ctx, H, heads, D, Vd, k_scale=c, skip=skip,
                             normaliser=H * D * Vd if norm else None)
        got.append((o if norm else (o,)) + (state,))
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("H,C,R,window,portions,broken", [
    (16, 64, 16, 0, [(0, 801)], ()), (16, 272, 16, 900, [(0, 401), (700, 402), (3, 2)], ()),
    (20, 48, 0, 512, [(0, 129), (0, 300), (400, 99)], ()), (3, 512, 32, 1024, [(0, 770)], (66, 300)),
    (16, 16, 16, 0, [(0, 63), (0, 65), (64, 641)], (62, 64))])
def test_latent_attention_of_neighbouring_tokens(H, C, R, window, portions, broken):
    """Tokens in fours that share tiles of keys: the bits of a block a token, with remainders of four, requests
    that meet inside a four, windows that start behind key 0, odd numbers of 32 channels, and keys that are no
    number, which no token in front of them sees."""
    from types import SimpleNamespace
    from ginfer_b200.ops import latent
    page, g = 16, torch.Generator(device=DEV).manual_seed(C + R)
    lens, T = [a + n for a, n in portions], sum(n for _, n in portions)
    pages = [-(-n // page) for n in lens]
    table = torch.zeros(len(lens), max(pages), dtype=torch.int32)
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(C)).int()
    for i, n in enumerate(pages):
        table[i, :n] = order[sum(pages[:i]):sum(pages[:i + 1])]
    c = torch.randn(sum(pages), page, 1, C, device=DEV, generator=g).bfloat16()
    r = torch.randn(sum(pages), page, 1, R, device=DEV, generator=g).bfloat16() if R else None
    for p in broken:
        c.view(-1, C)[int(table[0, p // page]) * page + p % page, ::3] = float("nan")
    q = torch.randn(H, T, C, device=DEV, generator=g) * 3 * C ** -0.5
    qr = torch.randn(T, H, R, device=DEV, generator=g) if R else None
    seq = torch.cat([torch.full((n,), i) for i, (_, n) in enumerate(portions)]).int().cuda()
    pos = torch.cat([torch.arange(a, a + n) for a, n in portions]).int().cuda()
    out = []
    for longest in (max(n for _, n in portions), 0):       # 0: a block a token
        ctx = SimpleNamespace(seq_of_token=seq, positions=pos, max_kv_len=max(lens), max_q_len=longest)
        out.append(latent.attention(q, qr, c, r, table.cuda(), ctx, window, (C + R) ** -0.5, page))
    assert torch.equal(*(torch.nan_to_num(o.float(), nan=1e9) for o in out))
    if broken:
        assert torch.isnan(out[0]).any() and not torch.isnan(out[0][:, :min(broken)]).any()


def test_launches_are_counted_where_their_number_follows_from_the_step():
    """What the counter says of a call is the number of kernels that a graph captures of it, whichever call of a kind
    comes first: chunked recurrences with and without shared scores, latent attention plain, in shares and with
    tokens that share tiles, the delta rule in one kernel, in two, and in chunks."""
    from types import SimpleNamespace
    from cuda.bindings import runtime
    from ginfer_b200 import ops
    from ginfer_b200.ops import decay, delta, latent

    def zeros(*shape, dtype=torch.float32):
        return torch.zeros(shape, dtype=dtype, device=DEV)

    def step(lens):
        B, T = len(lens), sum(lens)
        return T, SimpleNamespace(
            num_seqs=B, slot_ids=torch.arange(B).int().cuda(), max_q_len=max(lens), q_lens_host=lens,
            q_starts_host=[0] * B, cu_seqlens_q=torch.tensor([0] + lens).cumsum(0).int().cuda(),
            seq_of_token=torch.repeat_interleave(torch.arange(B), torch.tensor(lens)).int().cuda(),
            positions=torch.cat([torch.arange(n) for n in lens]).int().cuda(), max_kv_len=max(lens))

    def chunked(H, G):
        T, ctx = step([70, 3])
        q, v, g, state = zeros(T, G * 4), zeros(T, H * 8), zeros(T, H), zeros(2, H * 32)
        return lambda: decay.recurrence(q, q, v, g, state, ctx, H, G, 4, 8)

    def attention(H, lens, keys=0):
        T, ctx = step(lens)
        ctx.max_kv_len = keys or ctx.max_kv_len
        q, c, table = zeros(H, T, 32), zeros(600, 16, 1, 32, dtype=torch.bfloat16), zeros(len(lens), 600, dtype=torch.int32)
        return lambda: latent.attention(q, None, c, None, table, ctx, 0, 1.0, 16)

    def rule(H, D, lens, one):
        T, ctx = step(lens)
        q, v, state = zeros(T, H, D), zeros(T, H, 64), zeros(len(lens), H * D * 64)
        g, beta = zeros(T, H) if one else zeros(T, H, D), zeros(T, H)
        return lambda: delta.recurrence(q, q, v, g, beta, state, ctx)
    calls = [chunked(4, 4), chunked(4, 2), chunked(4, 4), attention(16, [5]), attention(16, [1, 1], 9000),
             attention(16, [801]), attention(16, [5]), rule(16, 128, [9, 9], 0), rule(16, 128, [1] * 20 + [30], 0),
             rule(16, 64, [40, 3], 1), rule(16, 128, [9, 9], 0)]
    counts = []
    for call in calls:
        call()                                       # (libraries and attributes)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            before = ops.launch_count()
            call()
            counted = ops.launch_count() - before
        raw = runtime.cudaGraph_t(graph.raw_cuda_graph())
        err, _, n = runtime.cudaGraphGetNodes(raw)
        err, nodes, n = runtime.cudaGraphGetNodes(raw, n)
        kinds = [runtime.cudaGraphNodeGetType(node)[1] for node in nodes[:n]]
        counts.append((counted, sum(k == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)))
    assert [a for a, _ in counts] == [b for _, b in counts] == [3, 4, 3, 1, 2, 2, 1, 1, 2, 2, 1], counts


def _kernels(call):
    """The names of the kernels that a call launches, as a captured graph has them."""
    from cuda.bindings import driver
    call()                                           # (libraries and attributes)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw, names = driver.CUgraph(graph.raw_cuda_graph()), []
    err, _, n = driver.cuGraphGetNodes(raw)
    err, nodes, n = driver.cuGraphGetNodes(raw, n)
    for node in nodes[:n]:
        if driver.cuGraphNodeGetType(node)[1] != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        err, params = driver.cuGraphKernelNodeGetParams(node)
        err, name = driver.cuFuncGetName(params.func) if int(params.func) else driver.cuKernelGetName(params.kern)
        names.append(name.decode())
    return names


@pytest.mark.parametrize("H,D,Vd,lens,warp", [
    (4, 128, 128, [5], True), (2, 72, 128, [1, 17], True), (2, 72, 128, [1, 1, 17], False), (4, 128, 128, [63], True), (4, 128, 128, [64], False),
    (5, 97, 128, [9], True), (6, 97, 128, [9], False), (5, 65, 128, [30], True), (8, 96, 128, [9], False)])
def test_delta_rule_of_few_columns_and_tokens_takes_a_warp_a_column(H, D, Vd, lens, warp):
    """While every block has an SM of its own and portions are short; the same bits as beside a long portion, where the
    other kernel serves."""
    step, state0 = _delta_step(H, H, D, Vd, lens)
    one = step()
    names = _kernels(lambda: one(state0))
    assert any("delta_recurrence_kernel" in n for n in names) == warp != any("delta_tree_kernel" in n for n in names)
    both, more = _delta_step(H, H, D, Vd, lens + [64])
    less = more[:len(lens)].clone()
    o = both()(more)
    assert torch.equal(both(slice(0, sum(lens)), lens)(less), o[:sum(lens)]) and torch.equal(less, more[:len(lens)])


@pytest.mark.parametrize("E,N,K,pairs,ring", [
    (24, 2048, 1408, 32, False), (24, 2048, 1408, 48, True), (24, 4096, 1280, 28, False), (24, 4096, 1280, 40, True),
    (24, 2112, 2048, 28, True), (32, 2048, 1536, 32, True)])
def test_routed_products_take_equal_runs_where_they_gain(E, N, K, pairs, ring):
    from ginfer_b200.ops import moe
    x, w = torch.zeros(pairs, K, device=DEV).bfloat16(), torch.zeros(E, N, K, device=DEV).bfloat16()
    plan = moe.Plan(torch.arange(pairs, dtype=torch.int32, device=DEV).view(-1, 1) % E, E, "few")
    names = _kernels(lambda: moe.grouped_down(x, w, plan))
    assert any("moe_ring_kernel" in n for n in names) == ring != any("moe_stream_kernel" in n for n in names)
