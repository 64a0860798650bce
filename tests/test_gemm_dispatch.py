"""Which kernel a bfloat16 product of few rows gets (on the host): the one that streams the weights
through registers or the tcgen05 one."""
import pytest
import torch

from ginfer_b200.ops import gemm_bf16

BF, F32 = torch.bfloat16, torch.float32


class _Tcgen05(Exception):
    pass


@pytest.fixture
def kernel(monkeypatch):
    def tcgen05(*_):
        raise _Tcgen05
    monkeypatch.setattr(gemm_bf16, "stream", lambda *a, **k: True)
    monkeypatch.setattr(gemm_bf16, "_dev_state", tcgen05)         # (both asked for on the way to that kernel)
    monkeypatch.setattr(gemm_bf16, "_workspace", tcgen05)

    def of(M, N, K, dtype, **kw):
        try:
            gemm_bf16.gemm(torch.zeros(M, K, dtype=BF), torch.empty(N, K, dtype=BF), None, dtype, **kw)
        except _Tcgen05:
            return "tcgen05"
        return "stream"
    return of


@pytest.mark.parametrize("M, N, K, dtype, epi, want", [
    (1, 256, 64, BF, 0, "stream"), (4, 256, 64, BF, 0, "stream"), (5, 256, 64, BF, 0, "tcgen05"),
    (5, 256, 64, F32, 0, "stream"), (8, 256, 64, F32, 0, "stream"), (9, 256, 64, F32, 0, "tcgen05"),
    (8, 256, 64, BF, 1, "stream"), (8, 256, 64, BF, 2, "stream"), (8, 256, 64, BF, 4, "stream"),
    (9, 256, 64, BF, 2, "tcgen05"),
    (1, 1776, 4096, BF, 0, "stream"), (1, 1777, 4096, BF, 0, "tcgen05"), (8, 1777, 4096, BF, 2, "tcgen05")])
def test_few_rows_and_small_weights_are_streamed(kernel, M, N, K, dtype, epi, want):
    assert kernel(M, N, K, dtype, epi=epi) == want


@pytest.mark.parametrize("kw", [dict(split_k=1), dict(split_k=4), dict(split_k=3, through_workspace=True),
                                dict(through_workspace=True), dict(streamed=False), dict(resid=torch.zeros(2, 256)),
                                dict(scale=gemm_bf16.RowScale(torch.zeros(1, 16), 1e-6))])
def test_what_asks_for_the_other_kernel_gets_it(kernel, kw):
    assert kernel(2, 256, 64, F32, **kw) == "tcgen05"
    assert kernel(2, 256, 64, F32) == "stream"
