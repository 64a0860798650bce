"""Workloads of the engine that its speed and its outputs are measured on.

A pass runs a batch of requests from their prompts to their last output token, through the step
function: prompts go in under a token budget, in portions where they are longer, beside the single
tokens of requests that already decode, as continuous batching orders it.  The token ids are given
(a replayed trace), so every pass does the same work whatever a rounding does to an arg-max.  The
outputs are the logits of every prompt's last token and of every output token.

Weights are drawn from the seed as deep residual models start out: matrices keep the size of what
passes them, a sublayer's last matrix is smaller by the root of the number of sublayers, embeddings
are as large as all that the layers add, norms are near one; decay rates, step sizes, mixing matrices
and routers lie where trained models have them.  So a rounding stays the size of a rounding on its
way to the logits, and an expert is seldom chosen by one.  Every drawn value is one that bfloat16
holds, unless the model runs in 32-bit.
"""
from __future__ import annotations

import hashlib
import math

import torch

PAGE = 16
VOCAB = 32768          # of the designs beside Qwen2, as in the benchmark
F64 = torch.float64


# ----------------------------------------------------------------------------- configurations
def _qwen2(hidden, heads, kv, ff, theta, layers=28, vocab=151936, positions=4096):
    return {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": layers,
            "hidden_size": hidden, "num_attention_heads": heads, "num_key_value_heads": kv,
            "head_dim": hidden // heads, "intermediate_size": ff, "vocab_size": vocab,
            "rope_theta": theta, "rms_norm_eps": 1e-6, "max_position_embeddings": positions,
            "tie_word_embeddings": False, "use_sliding_window": False, "torch_dtype": "bfloat16"}


def _vilepel(width, heads, dim, rank, window, ff, experts, top, expert_ff):
    latent = {"type": "latent_attention", "mixer": {
        "heads": heads, "dim": dim, "rot_dim": dim // 2, "vdim": dim, "kv_rank": rank,
        "scale": (1.5 * dim) ** -0.5, "mask": {"size": window}, "rot": {"base": 10000.0, "dims": dim // 2}}}
    delta = {"type": "channel_delta", "mixer": {"heads": heads, "kv_heads": heads, "dim": dim, "vdim": dim,
                                                "conv": 4, "decay_rank": 64, "gate_rank": 64}}
    dense = {"kind": "dense", "ff": ff, "limit": 7.0}
    moe = {"kind": "moe", "expert": {"ff": expert_ff, "limit": 7.0},
           "router": {"experts": experts, "top": top}}
    turns = [dict(latent, mlp=dense), dict(delta, mlp=moe), dict(latent, mlp=moe), dict(delta, mlp=dense)]
    return {"architecture": "Vilepel", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-5},
            "embedding": {"scale": 1.0}, "torch_dtype": "bfloat16", "layers": turns * 2}


def _zolapel(width, heads, kv, dim, window, experts, top, expert_ff, side):
    layer = {"type": "attention",
             "mixer": {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
                       "mask": {"size": window},
                       "rot": {"base": 500000.0, "dims": dim, "scaling": {
                           "factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}},
             "mlp": {"kind": "moe", "expert": {"ff": expert_ff}, "router": {"experts": experts, "top": top}}}
    return {"architecture": "Zolapel", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-5},
            "residual_mult": 0.5, "token_side": {"dim": side}, "torch_dtype": "bfloat16",
            "loop": {"start": 2, "stop": 4, "times": 2}, "layers": [layer] * 8}


def _pimidra(width, heads, kv, dim, chunk, ff, experts, top, expert_ff, ssd_heads, state):
    attention = {"type": "attention", "mixer": {
        "heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
        "mask": {"size": chunk}, "v_mix": True,
        "rot": {"base": 10000.0, "dims": dim // 2, "scaling": {"factor": 8.0}}}}
    ssd = {"type": "mamba2", "mixer": {"heads": ssd_heads, "vdim": 64, "state": state, "groups": 1,
                                       "conv": 4, "norm_groups": 1}}
    gla = {"type": "gla", "mixer": {"heads": heads, "dim": dim, "vdim": dim, "tau": 16.0, "decay_rank": 16}}
    dense = {"kind": "dense", "ff": ff}
    moe = {"kind": "moe", "expert": {"ff": expert_ff}, "router": {"experts": experts, "top": top}}
    turns = [dict(attention, mlp=dense), dict(ssd, mlp=moe), dict(attention, mlp=moe), dict(gla, mlp=dense)]
    return {"architecture": "Pimidra", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-5},
            "postln_alpha": 2.0, "torch_dtype": "bfloat16", "layers": turns * 2}


def _bapivik(width, heads, kv, dim, rank, q_rank, window, ff):
    def latent(source):
        m = {"heads": heads, "dim": dim, "vdim": dim, "kv_rank": rank, "q_rank": q_rank,
             "scale": dim ** -0.5}
        return {"type": "latent_attention", "mixer": m if source is None else dict(m, kv_from=source)}
    attention = {"type": "attention", "mixer": {
        "heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
        "mask": {"size": window}, "softcap": 30.0, "q_temp": {"coef": 0.25, "every": 256}}}
    linear = {"type": "lightning", "mixer": {
        "heads": heads, "dim": dim, "vdim": dim,
        "decay": [math.exp(-2.0 ** (-3.0 - 5.0 * n / heads)) for n in range(heads)]}}
    layers = []
    for i in (0, 4):
        layers += [latent(None), latent(i), attention, linear]
    return {"architecture": "Bapivik", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-5},
            "max_positions": 8192, "logit_softcap": 30.0, "torch_dtype": "bfloat16",
            "layers": [dict(x, mlp={"kind": "dense", "ff": ff}) for x in layers]}


def _lasizen(width, heads, kv, dim, window, ff):
    attention = {"type": "attention", "mixer": {
        "heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
        "mask": {"size": window},
        "rot": {"base": 500000.0, "dims": dim // 2,
                "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
    delta = {"type": "delta", "mixer": {"heads": heads, "kv_heads": heads, "dim": dim, "vdim": dim, "conv": 4}}
    return {"architecture": "Lasizen", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-5},
            "embedding": {"scale": 1.0}, "logit_scale": 0.5, "torch_dtype": "bfloat16",
            "layers": [dict((attention, delta)[i % 2], mlp={"kind": "dense", "ff": ff}) for i in range(8)]}


def _daburax(width, heads, kv, dim, experts, identity, top, expert_ff):
    retention = {"type": "retention", "mixer": {
        "heads": heads, "dim": dim, "vdim": dim, "rot": {"base": 10000.0, "dims": dim},
        "decay": [1.0 - 2.0 ** (-5.0 - 4.0 * n / heads) for n in range(heads)]}}
    parallel = {"type": "parallel", "mixer": {
        "left": {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
                 "rot": {"base": 10000.0, "dims": dim // 2, "scaling": {"factor": 4.0}}},
        "right": {"heads": heads, "dim": dim, "vdim": dim, "gate_cap": 15.0},
        "left_scale": 1.0, "right_scale": 0.5}}
    mlp = {"kind": "moe", "expert": {"ff": expert_ff}, "shared": {"ff": expert_ff},
           "router": {"experts": experts - identity, "identity": identity, "top": top,
                      "groups": {"count": 4, "keep": 2}}}
    return {"architecture": "Daburax", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-6},
            "streams": 4, "residual_mult": 0.5, "torch_dtype": "bfloat16",
            "embedding": {"scale": 1.0, "bigram": {"buckets": 32749, "mul_prev": 257, "mul_cur": 31}},
            "layers": [dict(parallel if i % 4 == 2 else retention, mlp=mlp) for i in range(8)]}


# the shapes that the benchmark measures, by design and size
CONFIGS = {
    ("qwen2", "1.5b"): lambda: _qwen2(1536, 12, 2, 8960, 10000.0),
    ("qwen2", "7b"): lambda: _qwen2(3584, 28, 4, 18944, 1e6, vocab=152064, positions=8192),
    ("vilepel", "s"): lambda: _vilepel(1024, 8, 64, 256, 512, 2816, 16, 2, 704),
    ("vilepel", "m"): lambda: _vilepel(2048, 16, 128, 512, 1024, 5632, 32, 4, 1408),
    ("zolapel", "s"): lambda: _zolapel(1024, 8, 2, 64, 512, 16, 2, 1056, 64),
    ("zolapel", "m"): lambda: _zolapel(2048, 16, 4, 128, 1024, 32, 4, 2112, 128),
    ("pimidra", "s"): lambda: _pimidra(1024, 8, 2, 64, 512, 2816, 16, 2, 704, 32, 64),
    ("pimidra", "m"): lambda: _pimidra(2048, 16, 4, 128, 1024, 5632, 32, 4, 1408, 64, 128),
    ("bapivik", "s"): lambda: _bapivik(1024, 8, 2, 64, 256, 384, 512, 4224),
    ("bapivik", "m"): lambda: _bapivik(2048, 16, 4, 128, 512, 768, 1024, 8448),
    ("lasizen", "s"): lambda: _lasizen(1024, 8, 2, 64, 512, 4224),
    ("lasizen", "m"): lambda: _lasizen(2048, 16, 4, 128, 1024, 8448),
    ("daburax", "s"): lambda: _daburax(1024, 8, 2, 64, 16, 2, 2, 704),
    ("daburax", "m"): lambda: _daburax(2048, 16, 4, 128, 32, 4, 4, 1408),
}


# ----------------------------------------------------------------------------- the cases
def _case(design, size, requests, prompt_min, prompt_max, outputs, budget=8192, dtype="bfloat16"):
    return {"design": design, "size": size, "dtype": dtype, "requests": requests,
            "prompt_min": prompt_min, "prompt_max": prompt_max, "outputs": outputs, "budget": budget}


def listed():
    return [
        # one chat user: a short question (13 to 19 ids in the published runs), latency of each token
        dict(_case("qwen2", "1.5b", 1, 17, 17, 40), name="chat of one"),
        # the benchmark's headline batch: 8 prompts of 512, decoding
        dict(_case("qwen2", "1.5b", 8, 512, 512, 32), name="batch of 8"),
        # a full engine (64 requests at a time by default) of prompts of uneven length
        dict(_case("qwen2", "1.5b", 64, 33, 321, 24), name="batch of 64"),
        # time to the first token of one 2,048-token prompt
        dict(_case("qwen2", "1.5b", 1, 2048, 2048, 1), name="prompt of 2048"),
        # the 7B shape in service: long and short prompts in portions of 2,048 beside decoding requests
        dict(_case("qwen2", "7b", 8, 130, 4097, 20, budget=2048), name="7b in service"),
        # the 32-bit path (checking a model, or serving one that needs it): ragged prompts and decoding
        dict(_case("qwen2", "1.5b", 3, 19, 101, 6, dtype="float32"), name="32-bit"),
        # every further design at a different point of the range: few and many requests, the first
        # portion of a long prompt and later ones, the smaller and the larger size
        dict(_case("vilepel", "m", 4, 150, 1201, 16), name="vilepel of 4"),
        dict(_case("zolapel", "m", 16, 37, 259, 20), name="zolapel of 16"),
        dict(_case("pimidra", "m", 2, 1500, 1700, 16), name="pimidra of 2"),
        dict(_case("bapivik", "m", 32, 61, 193, 16), name="bapivik of 32"),
        dict(_case("lasizen", "s", 1, 43, 43, 32), name="lasizen of one"),
        dict(_case("daburax", "m", 8, 350, 650, 20, budget=2048), name="daburax of 8"),
    ]


def draw(rng):
    """Another case: Qwen2 as often as the other designs together, batches of 1 to 64, prompts of 8
    to 3,000 tokens, 1 to 40 outputs, 32-bit with small batches only (as it is used)."""
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    while True:
        design = "qwen2" if rng.random() < 0.5 else rng.choice(
            ("vilepel", "zolapel", "pimidra", "bapivik", "lasizen", "daburax"))
        size = ("7b" if rng.random() < 0.2 else "1.5b") if design == "qwen2" else rng.choice("sm")
        full = rng.random() < 0.15 and size != "7b"
        requests = spread(1, 4) if full else spread(1, 64)
        longest = spread(8, 150 if full else 3000)
        shortest = min(longest, spread(8, 1000))
        c = _case(design, size, requests, shortest, longest, spread(1, 8 if full else 40),
                  rng.choice((2048, 8192)), "float32" if full else "bfloat16")
        if sum(lengths(c)) <= (9000 if size == "7b" else 20000) and requests * c["outputs"] <= 1536:
            return c


def lengths(case):
    """The requests' prompt lengths: from the shortest to the longest, evenly on a logarithmic
    scale, every third one from the other end, so that long and short ones mix."""
    n, lo, hi = case["requests"], case["prompt_min"], case["prompt_max"]
    up = [int(round(lo * (hi / lo) ** (i / max(1, n - 1)))) for i in range(n)] if n > 1 else [hi]
    out = []
    while up:
        out.append(up.pop() if len(out) % 3 == 2 else up.pop(0))
    return out


def schedule(case):
    """The steps of a pass: lists of ``(request, first token, tokens, logits wanted)``.  A request
    whose prompt is through brings its next token to every step; the budget that is left goes to
    prompts in order, in portions."""
    prompts, outputs = lengths(case), case["outputs"]
    done = [0] * len(prompts)
    steps = []
    while True:
        left, step = case["budget"], []
        for r, n in enumerate(prompts):
            if n <= done[r] < n + outputs - 1:
                step.append((r, done[r], 1, True))
        left -= len(step)
        for r, n in enumerate(prompts):
            take = min(left, n - done[r])
            if done[r] < n and take > 0:
                step.append((r, done[r], take, done[r] + take == n))
                left -= take
        if not step:
            return steps
        for r, _, n, _ in step:
            done[r] += n
        steps.append(step)


def sequences(case, seed):
    """Token ids of every request: prompt and the outputs that are fed back."""
    g = torch.Generator().manual_seed(int(seed) * 7919 + 11)
    vocab = CONFIGS[case["design"], case["size"]]().get("vocab_size", VOCAB)
    return [torch.randint(0, vocab, (n + case["outputs"] - 1,), generator=g).tolist()
            for n in lengths(case)]


# ----------------------------------------------------------------------------- weights
def weight(case, seed, name, shape, device):
    """The tensor ``name`` of the case's model, in 32-bit."""
    digest = hashlib.sha256(f"{seed}:{name}".encode()).digest()
    g = torch.Generator(device=device).manual_seed(int.from_bytes(digest[:7], "little"))
    leaf = name.rsplit(".", 1)[-1]
    design, streams = case["design"], 4

    def normal(mean, std):
        return torch.randn(shape, generator=g, device=device) * std + mean

    def uniform(lo, hi):
        return torch.rand(shape, generator=g, device=device) * (hi - lo) + lo
    layers = 28 if design == "qwen2" else 8
    if "norm" in leaf or "norm." in name:
        if name == "final.norm" or leaf not in ("norm1", "norm2"):
            mean = 0.0 if leaf == "b" or (name == "final.norm" and design in ("vilepel", "daburax")) else 1.0
            t = normal(0.1 if name.endswith("side.norm") else mean, 0.02)
        else:                      # around zero in two designs; one norms what a sublayer adds
            t = normal({"vilepel": -0.7, "daburax": 0.0}.get(design, 1.0), 0.02)
    elif leaf == "A_log":                                  # rates of 1 to 16
        t = uniform(1.0, 16.0).log()
    elif leaf == "dt_bias":                                # steps of 0.001 to 0.1 through softplus
        t = uniform(math.log(1e-3), math.log(1e-1)).exp().expm1().log()
    elif leaf == "conv" or name.endswith("conv.b"):
        t = uniform(-0.5, 0.5)
    elif name.endswith("a2.b"):                            # most channels are kept
        t = normal(2.0, 1.0)
    elif name.endswith("i.b"):
        t = normal(-1.0, 0.5)
    elif name.endswith("f.b"):
        t = normal(3.0, 1.0)
    elif leaf in ("D", "act", "vmix", "sink", "shift", "ls1", "ls2", "step"):
        lo, hi = {"D": (0.8, 1.2), "act": (0.3, 0.7), "vmix": (0.4, 0.6), "sink": (-1.0, 1.0),
                  "shift": (0.0, 1.0), "ls1": (0.1, 0.2), "ls2": (0.03, 0.07), "step": (-0.03, 0.03)}[leaf]
        t = uniform(lo, hi)
    elif leaf == "dwa":                                    # mostly the layer's own result
        t = normal(0.0, 0.05)
        t[-1] += 1.0
    elif ".hc" in name:                                    # streams that differ and mix a little
        t = normal(1.0 / streams, 0.05) if leaf == "in" else normal(1.0, 0.2)
        if leaf == "mix":
            t = torch.eye(streams, device=device) + (t - 1.0) * 0.25
    elif leaf == "router":                                 # a trained router prefers some experts
        t = normal(0.0, 3.0 * shape[1] ** -0.5)
    elif leaf == "correction":
        t = normal(0.0, 0.01)
    elif leaf in ("embed", "bigram", "pos") or "embed_tokens" in name:
        tied = {"zolapel": 0.2, "bapivik": 0.02}           # the head is the same matrix
        t = normal(0.0, 1.0 if name == "side.embed" else tied.get(design, 1.0))
    elif len(shape) < 2:
        t = normal(0.0, 0.02)
    else:
        last = leaf in ("o", "down") or "o_proj" in name or "down_proj" in name
        sharp = "q_proj" in name or "k_proj" in name       # scores that prefer some keys
        t = normal(0.0, shape[1] ** -0.5 * (1.5 if sharp else (2 * layers) ** -0.5 if last else 1.0))
    return t if case["dtype"] == "float32" else t.to(torch.bfloat16).float()


# ----------------------------------------------------------------------------- through the engine
def prepare(case, seed):
    """A loaded model with its runner and cache (a server that is up) and the requests' tokens."""
    from ginfer_b200 import architectures  # noqa: F401  (registers the designs)
    from ginfer_b200.config.registry import resolve_architecture
    from ginfer_b200.engine import ModelRunner, StepEntry
    from ginfer_b200.parts.model import DecoderModel

    device = torch.device("cuda:0")
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    config = CONFIGS[case["design"], case["size"]]()
    arch = resolve_architecture(config)
    model = DecoderModel(arch.build_plan(arch.config_cls.from_dict(config)))
    tensors = {}
    for s in model.tensor_specs():
        t = weight(case, seed, s.name, s.shape, device)
        tensors[s.name] = t if s.role in ("f32", "norm32") else t.to(dtype)
    model.load(tensors, dtype, device)
    del tensors
    total = [n + case["outputs"] - 1 for n in lengths(case)]
    runner = ModelRunner(model, page_size=PAGE, max_num_seqs=64,
                         max_seq_len=8192 if max(total) > 4096 else 4096,
                         num_pages=sum(-(-n // PAGE) + 1 for n in total) + 8,
                         max_num_batched_tokens=8192, enforce_eager=False)
    runner.warmup()
    ids = sequences(case, seed)
    steps = [[StepEntry(r, ids[r][at:at + n], [n - 1] if want else []) for r, at, n, want in step]
             for step in schedule(case)]
    rows = case["requests"] * case["outputs"]
    logits = torch.empty((rows, runner.vocab_size), dtype=torch.float32, device=device)
    return {"runner": runner, "steps": steps, "logits": logits}


@torch.no_grad()
def run(state):
    runner, out, at = state["runner"], state["logits"], 0
    for entries in state["steps"]:
        logits = runner.step(entries)
        n = logits.shape[0]
        if n:
            out[at:at + n].copy_(logits)       # a step's logits are valid until the next step
            at += n
    for r in {e.request_id for entries in state["steps"] for e in entries}:
        runner.end(r)
    return out


# ----------------------------------------------------------------------------- what a pass needs
def _layers(config):
    """``(mixer type, mixer, feed-forward)`` of every layer run."""
    if "num_hidden_layers" in config:
        m = {"heads": config["num_attention_heads"], "kv_heads": config["num_key_value_heads"],
             "dim": config["head_dim"], "vdim": config["head_dim"]}
        return [("attention", m, {"kind": "dense", "ff": config["intermediate_size"]})] * config["num_hidden_layers"]
    layers = [(x["type"], x["mixer"], x["mlp"]) for x in config["layers"]]
    loop = config.get("loop")
    if loop:
        a, b = loop["start"], loop["stop"]
        layers = layers[:b] + layers[a:b] * (loop["times"] - 1) + layers[b:]
    return layers


def _mixer_size(kind, m, width, design):
    """``(weights, state or cache values a token or request, flops a token beside the weights' and
    flops a key a query sees)``."""
    if kind == "parallel":
        parts = [_mixer_size("attention", m["left"], width, design),
                 _mixer_size("memory", m["right"], width, design)]
        return tuple(sum(p[i] for p in parts) for i in range(5))
    h, d, v = m["heads"], m.get("dim", m.get("state")), m["vdim"]
    if kind == "attention":
        g = m["kv_heads"]
        shared = design in ("zolapel", "bapivik")          # values that are the keys as projected
        return (width * (2 * h * d + g * d * (1 if shared else 2)), 2 * g * d, 0, 0, 4 * h * d)
    if kind == "latent_attention":
        r, rank = m.get("rot_dim", 0), m["kv_rank"]
        q = width * m["q_rank"] + m["q_rank"] * h * d if "q_rank" in m else width * h * (d + r)
        own = 0 if "kv_from" in m else width * (rank + r)
        return (q + own + rank * h * (d + v) + h * v * width, (rank + r) if own else 0, 0, 0,
                2 * h * (d + r + v))
    if kind == "mamba2":
        return (width * (2 * h * v + 2 * d + h) + h * v * width, 0, h * d * v, 6 * h * d * v, 0)
    extra = {"channel_delta": 2, "delta": 3, "gla": 3, "lightning": 3, "retention": 3, "memory": 3}[kind]
    inner = width * h * (2 * d + (extra - 1) * v) + h * v * width
    return (inner, 0, h * d * v, (8 if "delta" in kind else 6) * h * d * v, 0)


def work(case):
    """Weights once a step (of the experts the expected number that its tokens reach), the cache a
    query sees and recurrent states once a step, logits written once; two flops a weight a token,
    the scores and the recurrences."""
    config = CONFIGS[case["design"], case["size"]]()
    width = config.get("hidden_size", config.get("width"))
    vocab = config.get("vocab_size", VOCAB)
    item = 4 if case["dtype"] == "float32" else 2
    nbytes = flops = 0.0
    sizes = [(_mixer_size(kind, m, width, case["design"]), m, mlp) for kind, m, mlp in _layers(config)]
    for step in schedule(case):
        tokens = sum(n for _, _, n, _ in step)
        rows = sum(1 for s in step if s[3])
        nbytes += rows * vocab * 4 + (vocab * width * item if rows else 0) + tokens * width * item
        flops += 2.0 * rows * vocab * width
        for (weights, cached, state, per_token, per_key), m, mlp in sizes:
            nbytes += weights * item + 8.0 * state * len(step)
            flops += tokens * (2.0 * weights + per_token)
            window = (m.get("mask") or {}).get("size", 0)
            for _, start, n, _ in step:
                seen = [min(p + 1, window) if window else p + 1 for p in (start, start + n - 1)]
                nbytes += cached * item * min(start + n, seen[1] + n)
                flops += per_key * n * (seen[0] + seen[1]) / 2
            if mlp["kind"] == "dense":
                mats = 2 if case["design"] in ("bapivik", "lasizen") else 3
                nbytes += mats * width * mlp["ff"] * item
                flops += 2.0 * mats * width * mlp["ff"] * tokens
            else:
                r, mats = mlp["router"], 2 if case["design"] == "zolapel" else 3
                outputs = r["experts"] + r.get("identity", 0)
                reached = r["experts"] * (1.0 - (1.0 - r["top"] / outputs) ** tokens)
                one = mats * width * mlp["expert"]["ff"]
                used = r["top"] * r["experts"] / outputs
                shared = mats * width * mlp["shared"]["ff"] if mlp.get("shared") else 0
                nbytes += (reached * one + shared + outputs * width) * item
                flops += 2.0 * (used * one + shared + outputs * width) * tokens
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """32-bit: measured 1e-6 to 3e-6 off 64 bits.  bfloat16: 2e-3 to 1.2e-2 off, most of it from a
    few roundings a layer, and where feed-forwards are routed from the odd token whose choice of
    experts a rounding decides; two right implementations are up to about 1.4 times that apart."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 0.02 if case["design"] in ("qwen2", "bapivik", "lasizen") else 0.03}


# ----------------------------------------------------------------------------- plain, in 64 bits
class _Plain:
    """The case's model over whole sequences in float64: plain torch, no cache, no batching rules."""

    def __init__(self, case, seed):
        self.case, self.seed = case, seed
        self.config = CONFIGS[case["design"], case["size"]]()
        self.device = torch.device("cuda:0" if torch.cuda.is_available() else "cpu")
        self.ids = sequences(case, seed)
        self.n = [len(s) for s in self.ids]
        self.top = max(self.n)
        tokens = torch.tensor([t for s in self.ids for t in s], device=self.device)
        self.tokens = tokens
        self.place = torch.cat([torch.arange(n, device=self.device) + i * self.top
                                for i, n in enumerate(self.n)])          # rows of the padded batch
        self.pos = torch.cat([torch.arange(n, device=self.device) for n in self.n])
        self.width = self.config.get("hidden_size", self.config.get("width"))
        self.eps = self.config.get("rms_norm_eps") or self.config["norm"]["eps"]

    # tensors and rows
    def w(self, name, *shape):
        return weight(self.case, self.seed, name, shape, self.device).to(F64)

    def lin(self, x, name, out, bias=None):
        y = x @ self.w(name, out, x.shape[-1]).T
        return y if bias is None else y + self.w(bias, out)

    def pad(self, x):
        out = torch.zeros((len(self.n) * self.top,) + x.shape[1:], dtype=x.dtype, device=x.device)
        out[self.place] = x
        return out.view((len(self.n), self.top) + x.shape[1:])

    def flat(self, x):
        return x.reshape((-1,) + x.shape[2:])[self.place]

    def before(self, x, back):
        """The rows ``back`` tokens earlier in the same sequence, zeros before its start."""
        p = self.pad(x)
        out = torch.zeros_like(p)
        if back < self.top:
            out[:, back:] = p[:, :self.top - back]
        return self.flat(out)

    def rms(self, x, w=None):
        y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + self.eps)
        return y if w is None else y * w

    def norm(self, x, name, offset=0.0):
        return self.rms(x, offset + self.w(name, x.shape[-1]))

    def rotate(self, x, freqs, neighbours, mult=1.0):
        n = len(freqs)
        f = torch.tensor(freqs, dtype=torch.float32, device=x.device)
        a = (self.pos.float()[:, None] * f[None, :]).to(F64)[:, None, :]
        c, s = torch.cos(a) * mult, torch.sin(a) * mult
        out = x.clone()
        first = slice(0, 2 * n, 2) if neighbours else slice(0, n)
        second = slice(1, 2 * n, 2) if neighbours else slice(n, 2 * n)
        u, v = x[..., first], x[..., second]
        out[..., first], out[..., second] = u * c - v * s, v * c + u * s
        return out

    @staticmethod
    def freqs(dims, base, factor=1.0):
        return [base ** (-2.0 * i / dims) / factor for i in range(dims // 2)]

    def attend(self, q, k, v, scale, window=0, chunk=0, cap=None, slopes=False, sink=None):
        """``q [N, H, D]``, ``k``, ``v [N, G, .]``, sequence by sequence."""
        H, G = q.shape[1], k.shape[1]
        out = torch.empty(q.shape[0], H, v.shape[2], dtype=F64, device=q.device)
        at = 0
        for n in self.n:
            i = torch.arange(n, device=q.device)
            far = i[:, None] - i[None, :]
            hidden = far < 0
            if window:
                hidden |= far >= window
            if chunk:
                hidden |= (i[:, None] // chunk) != (i[None, :] // chunk)
            for h in range(H):
                g = h // (H // G)
                s = (q[at:at + n, h] @ k[at:at + n, g].T) * scale
                if cap:
                    s = cap * torch.tanh(s / cap)
                if slopes:
                    s = s - 2.0 ** (-8.0 * (h + 1) / H) * far
                s = s.masked_fill(hidden, -math.inf)
                top = s.amax(-1, keepdim=True)
                if sink is not None:
                    top = torch.maximum(top, sink[h])
                e = torch.exp(s - top)
                d = e.sum(-1, keepdim=True)
                if sink is not None:
                    d = d + torch.exp(sink[h] - top)
                out[at:at + n, h] = (e / d) @ v[at:at + n, g]
            at += n
        return out

    def scan(self, q, k, v, decay, beta=None):
        """``S <- decay S + k v^T`` (with ``beta``: the delta rule, ``v`` less what the state already
        answers, times beta), ``o = S^T q``; a decay a token and key channel, or a token."""
        q, k, v = self.pad(q), self.pad(k), self.pad(v)
        decay = self.pad(decay)
        if decay.dim() == 3:
            decay = decay[..., None]
        beta = None if beta is None else self.pad(beta)[..., None]
        B, T, H, D = q.shape
        S = torch.zeros(B, H, D, v.shape[-1], dtype=F64, device=q.device)
        out = torch.empty(B, T, H, v.shape[-1], dtype=F64, device=q.device)
        for t in range(T):
            S = decay[:, t, :, :, None] * S
            u = v[:, t]
            if beta is not None:
                u = beta[:, t] * (u - torch.einsum("bhdv,bhd->bhv", S, k[:, t]))
            S = S + k[:, t, :, :, None] * u[:, :, None, :]
            out[:, t] = torch.einsum("bhdv,bhd->bhv", S, q[:, t])
        return self.flat(out)

    def conv(self, x, name, bias=None):
        w = self.w(name, x.shape[1], 4)
        y = sum(self.before(x, 3 - j) * w[:, j] for j in range(4))
        return torch.nn.functional.silu(y if bias is None else y + self.w(bias, x.shape[1]))

    def experts(self, h, pre, mlp, idx, wgt, one):
        """``sum of wgt * one(expert, rows)`` over the chosen experts; ``one`` gets the rows' weights."""
        out = torch.zeros_like(h)
        for e in range(mlp["router"]["experts"]):
            row, place = torch.nonzero(idx == e, as_tuple=True)
            if row.numel():
                out.index_add_(0, row, one(f"{pre}e{e}.", h[row], wgt[row, place][:, None]))
        return out

    # the model
    def logits(self):
        x = getattr(self, self.case["design"])()
        rows, at = [], 0
        first = {}
        for n, p in zip(self.n, lengths(self.case)):
            first[len(first)] = at + p - 1
            at += n
        seen = dict.fromkeys(first, 0)
        for step in schedule(self.case):           # in the order a pass returns them
            for r, _, _, want in step:
                if want:
                    rows.append(first[r] + seen[r])
                    seen[r] += 1
        return self.head(x[torch.tensor(rows, device=x.device)])

    def head(self, x):
        c, design = self.config, self.case["design"]
        vocab = c.get("vocab_size", VOCAB)
        if design == "qwen2":
            return self.lin(self.norm(x, "model.norm.weight"), "lm_head.weight", vocab)
        if design == "zolapel":
            return self.lin(self.layer_norm(x, "final.norm"), "embed", vocab)
        y = self.norm(x, "final.norm", 1.0 if design in ("vilepel", "daburax") else 0.0)
        if design == "bapivik":
            cap = c["logit_softcap"]
            return cap * torch.tanh(self.lin(y, "embed", vocab) / cap)
        return self.lin(y, "head", vocab) * c.get("logit_scale", 1.0)

    def qwen2(self):
        c, W = self.config, self.width
        H, G, D, ff = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["intermediate_size"]
        x = self.w("model.embed_tokens.weight", c["vocab_size"], W)[self.tokens]
        f = self.freqs(D, c["rope_theta"])
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = self.norm(x, p + "input_layernorm.weight")
            q, k, v = (self.lin(h, f"{p}self_attn.{a}_proj.weight", n * D, f"{p}self_attn.{a}_proj.bias")
                       .view(-1, n, D) for a, n in (("q", H), ("k", G), ("v", G)))
            o = self.attend(self.rotate(q, f, False), self.rotate(k, f, False), v, D ** -0.5)
            x = x + self.lin(o.flatten(1), p + "self_attn.o_proj.weight", W)
            h = self.norm(x, p + "post_attention_layernorm.weight")
            z = torch.nn.functional.silu(self.lin(h, p + "mlp.gate_proj.weight", ff)) \
                * self.lin(h, p + "mlp.up_proj.weight", ff)
            x = x + self.lin(z, p + "mlp.down_proj.weight", W)
        return x

    def vilepel(self):
        W = self.width

        def glu(h, pre, ff, limit):
            g = self.lin(h, pre + "gate", ff).clamp(max=limit)
            u = self.lin(h, pre + "up", ff).clamp(-limit, limit)
            return self.lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), pre + "down", W)

        def latent(h, p, m):
            H, D, R, V, C = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            f = self.freqs(R, m["rot"]["base"])
            q = self.lin(h, p + "q", H * (D + R)).view(-1, H, D + R)
            dkv = self.lin(h, p + "dkv", C + R)
            c = self.norm(dkv[:, :C], p + "dkv.norm")
            kr = self.rotate(dkv[:, None, C:], f, True).expand(-1, H, -1)
            k = torch.cat([self.lin(c, p + "uk", H * D).view(-1, H, D), kr], -1)
            q = torch.cat([q[..., :D], self.rotate(q[..., D:], f, True)], -1)
            v = self.lin(c, p + "uv", H * V).view(-1, H, V)
            return self.lin(self.attend(q, k, v, m["scale"], m["mask"]["size"]).flatten(1), p + "o", W)

        def delta(h, p, m):
            H, D, V = m["heads"], m["dim"], m["vdim"]
            q, k, v = (self.conv(self.lin(h, p + a, H * n), f"{p}{a}.conv").view(-1, H, n)
                       for a, n in (("q", D), ("k", D), ("v", V)))
            q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            a = self.lin(self.lin(h, p + "a1", 64), p + "a2", H * D, p + "dt_bias").view(-1, H, D)
            rate = self.w(p + "A_log", H).exp()[:, None]
            g = torch.exp(-rate * torch.nn.functional.softplus(a))
            o = self.scan(q * D ** -0.5, k, v, g, torch.sigmoid(self.lin(h, p + "b", H)))
            gate = torch.sigmoid(self.lin(self.lin(h, p + "g1", 64), p + "g2", H * V)).view(-1, H, V)
            return self.lin((self.norm(o, p + "norm") * gate).flatten(1), p + "o", W)
        x = self.w("embed", VOCAB, W)[self.tokens]
        for i, L in enumerate(self.config["layers"]):
            p, mlp = f"l{i}.", L["mlp"]
            mix = latent if L["type"] == "latent_attention" else delta
            x = x + self.norm(mix(x, p + "mix.", L["mixer"]), p + "norm1", 1.0)
            if mlp["kind"] == "dense":
                y = glu(x, p + "mlp.", mlp["ff"], mlp["limit"])
            else:
                s = torch.softmax(self.lin(x, p + "mlp.router", mlp["router"]["experts"]), -1)
                wgt, idx = torch.topk(s, mlp["router"]["top"], -1)
                e = mlp["expert"]
                y = self.experts(x, p + "mlp.", mlp, idx, wgt,
                                 lambda q, r, s: s * glu(r, q, e["ff"], e["limit"]))
            x = x + self.norm(y, p + "norm2", 1.0)
        return x

    def layer_norm(self, x, name):
        y = x - x.mean(-1, keepdim=True)
        y = y / torch.sqrt((y * y).mean(-1, keepdim=True) + self.eps)
        return y * self.w(name, x.shape[-1]) + self.w(name + ".b", x.shape[-1])

    def zolapel(self):
        c, W = self.config, self.width
        m, mlp, d = c["layers"][0]["mixer"], c["layers"][0]["mlp"], c["token_side"]["dim"]
        H, G, D, mult = m["heads"], m["kv_heads"], m["dim"], c["residual_mult"]
        sc, n = m["rot"]["scaling"], len(c["layers"])
        f = []
        for v in self.freqs(D, m["rot"]["base"]):
            turns = sc["original"] * v / (2.0 * math.pi)
            keep = min(1.0, max(0.0, (turns - sc["low"]) / (sc["high"] - sc["low"])))
            f.append(keep * v + (1.0 - keep) * v / sc["factor"])
        x = self.w("embed", VOCAB, W)[self.tokens]
        emb = x
        side = self.w("side.embed", VOCAB, n * d)[self.tokens]
        loop, steps = c["loop"], self.w("loop.step", c["loop"]["times"], W)
        order = list(range(loop["stop"])) + list(range(loop["start"], loop["stop"])) * (loop["times"] - 1) \
            + list(range(loop["stop"], n))
        turn = 0
        for i in order:
            if i == loop["start"]:
                x = x + (emb if turn else 0.0) + steps[turn]
                turn += 1
            p = f"l{i}."
            h = self.layer_norm(x, p + "norm1")
            q = self.lin(h, p + "mix.q", H * D).view(-1, H, D)
            k = self.lin(h, p + "mix.k", G * D).view(-1, G, D)
            gate = torch.sigmoid(self.lin(h, p + "mix.g", H))[:, :, None]
            o = self.attend(self.rotate(self.norm(q, p + "mix.q.norm"), f, True),
                            self.rotate(self.norm(k, p + "mix.k.norm"), f, True), k, m["scale"],
                            m["mask"]["size"]) * gate
            x = x + mult * self.w(p + "ls1", W) * self.lin(o.flatten(1), p + "mix.o", W)
            h = self.layer_norm(x, p + "norm2")
            s = torch.sigmoid(self.lin(h, p + "mlp.router", mlp["router"]["experts"]))
            wgt, idx = torch.topk(s, mlp["router"]["top"], -1)
            y = self.experts(h, p + "mlp.", mlp, idx, wgt, lambda q, r, s: self.lin(
                torch.relu(self.lin(s * r, q + "up", mlp["expert"]["ff"])) ** 2, q + "down", W))
            x = x + mult * self.w(p + "ls2", W) * y
            g = torch.nn.functional.gelu(self.lin(x, p + "side.gate", d), approximate="tanh")
            x = x + mult * self.norm(self.lin(g * side[:, i * d:(i + 1) * d], p + "side.proj", W),
                                     p + "side.norm")
        return x

    def pimidra(self):
        W, c = self.width, self.config
        silu = torch.nn.functional.silu
        values = []

        def ssd(h, p, m):
            H, V, N = m["heads"], m["vdim"], m["state"]
            inner = H * V
            z, xbc, dt = self.lin(h, p + "in", 2 * inner + 2 * N + H).split([inner, inner + 2 * N, H], -1)
            xbc = self.conv(xbc, p + "conv", p + "conv.b")
            v, B, C = xbc[:, :inner].view(-1, H, V), xbc[:, inner:inner + N], xbc[:, inner + N:]
            dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias", H))
            decay = torch.exp(-self.w(p + "A_log", H).exp() * dt)
            k = B[:, None, :].expand(-1, H, -1)
            y = self.scan(C[:, None, :].expand(-1, H, -1), k, v * dt[:, :, None], decay)
            y = (y + self.w(p + "D", H)[:, None] * v).flatten(1) * silu(z)
            return self.lin(self.norm(y, p + "norm"), p + "o", W)

        def attention(h, p, m):
            H, G, D = m["heads"], m["kv_heads"], m["dim"]
            f = self.freqs(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"]["factor"])
            q, k, v = (self.lin(h, p + a, n * D, f"{p}{a}.b") for a, n in (("q", H), ("k", G), ("v", G)))
            q, k = self.norm(q, p + "q.norm").view(-1, H, D), self.norm(k, p + "k.norm").view(-1, G, D)
            values.append(v)
            if len(values) > 1:
                lam = self.w(p + "vmix")
                v = (1 - lam) * v + lam * values[0]
            o = self.attend(self.rotate(q, f, False), self.rotate(k, f, False), v.view(-1, G, D),
                            m["scale"], chunk=m["mask"]["size"])
            return self.lin(o.flatten(1), p + "o", W)

        def gla(h, p, m):
            H, D = m["heads"], m["dim"]
            q, k, v = (self.lin(h, p + a, H * D).view(-1, H, D) for a in "qkv")
            z = self.lin(self.lin(h, p + "a1", 16), p + "a2", H * D, p + "a2.b")
            alpha = (torch.nn.functional.logsigmoid(z) / m["tau"]).exp().view(-1, H, D)
            o = self.norm(self.scan(q * D ** -0.5, k, v, alpha), p + "norm").flatten(1)
            return self.lin(o * silu(self.lin(h, p + "g", H * D)), p + "o", W)
        mixers = {"mamba2": ssd, "attention": attention, "gla": gla}
        x = self.w("embed", VOCAB, W)[self.tokens]
        for i, L in enumerate(c["layers"]):
            p, mlp = f"l{i}.", L["mlp"]
            x = self.norm(c["postln_alpha"] * x + mixers[L["type"]](x, p + "mix.", L["mixer"]), p + "norm1")
            if mlp["kind"] == "dense":
                y = self.lin(torch.relu(self.lin(x, p + "mlp.gate", mlp["ff"]))
                             * self.lin(x, p + "mlp.up", mlp["ff"]), p + "mlp.down", W)
            else:
                ff = mlp["expert"]["ff"]
                s, idx = torch.topk(self.lin(x, p + "mlp.router", mlp["router"]["experts"]),
                                    mlp["router"]["top"], -1)
                y = self.experts(x, p + "mlp.", mlp, idx, torch.softmax(s, -1), lambda q, r, s: s * self.lin(
                    silu(self.lin(r, q + "gate", ff)) * self.lin(r, q + "up", ff), q + "down", W))
            x = self.norm(c["postln_alpha"] * x + y, p + "norm2")
        return x

    def bapivik(self):
        W, c = self.width, self.config
        latents = {}

        def linear(h, p, m):
            H, D = m["heads"], m["dim"]
            q, k, v = (torch.nn.functional.silu(self.lin(h, p + a, H * D)).view(-1, H, D) for a in "qkv")
            decay = torch.tensor(m["decay"], dtype=F64, device=h.device).expand(h.shape[0], H)
            o = self.norm(self.scan(q, k, v, decay).flatten(1), p + "norm")
            return self.lin(o * torch.sigmoid(self.lin(h, p + "g", H * D)), p + "o", W)

        def latent(h, p, m, i):
            H, D, R = m["heads"], m["dim"], m["kv_rank"]
            if "kv_from" not in m:
                latents[i] = self.norm(self.lin(h, p + "dkv", R), p + "dkv.norm")
            lat = latents[m.get("kv_from", i)]
            q = self.lin(self.norm(self.lin(h, p + "dq", m["q_rank"]), p + "dq.norm"), p + "uq", H * D)
            k, v = (self.lin(lat, p + a, H * D).view(-1, H, D) for a in ("uk", "uv"))
            o = self.attend(q.view(-1, H, D), k, v, m["scale"])
            o = o * torch.sigmoid(self.lin(h, p + "g", H))[:, :, None]
            return self.lin(o.flatten(1), p + "o", W)

        def attention(h, p, m):
            H, G, D, t = m["heads"], m["kv_heads"], m["dim"], m["q_temp"]
            q = self.norm(self.lin(h, p + "q", H * D).view(-1, H, D), p + "q.norm")
            k = self.lin(h, p + "k", G * D).view(-1, G, D)
            temp = 1.0 + t["coef"] * torch.log(((self.pos + 1) // t["every"]).to(F64) + 1.0)
            o = self.attend(q * temp[:, None, None], self.norm(k, p + "k.norm"), k, m["scale"],
                            m["mask"]["size"], cap=m["softcap"], slopes=True)
            return self.lin(o.flatten(1), p + "o", W)
        x = self.w("embed", VOCAB, W)[self.tokens] + self.w("pos", c["max_positions"], W)[self.pos]
        past = [x]
        for i, L in enumerate(c["layers"]):
            p, m, ff = f"l{i}.", L["mixer"], L["mlp"]["ff"]
            h = self.norm(x, p + "norm1")
            a = latent(h, p + "mix.", m, i) if L["type"] == "latent_attention" else \
                (attention if L["type"] == "attention" else linear)(h, p + "mix.", m)
            x = x + self.norm(a, p + "norm1b")
            u = torch.relu(self.lin(self.norm(x, p + "norm2"), p + "mlp.up", ff, p + "mlp.up.b")) ** 2
            x = x + self.norm(self.lin(u, p + "mlp.down", W, p + "mlp.down.b"), p + "norm2b")
            past.append(x)
            dwa = self.w(p + "dwa", i + 2)
            x = sum(dwa[j] * past[j] for j in range(i + 2))
        return x

    def lasizen(self):
        W, c = self.width, self.config

        def yarn(rot):
            sc, dims = rot["scaling"], rot["dims"]

            def at(turns):
                return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(rot["base"]))
            lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
            out = []
            for i, f in enumerate(self.freqs(dims, rot["base"])):
                ramp = min(1.0, max(0.0, (i - lo) / max(hi - lo, 0.001)))
                out.append(f / sc["factor"] * ramp + f * (1.0 - ramp))
            return out, 0.1 * math.log(sc["factor"]) + 1.0

        def attention(h, p, m):
            H, G, D = m["heads"], m["kv_heads"], m["dim"]
            f, mult = yarn(m["rot"])
            q, k, v = (self.lin(h, p + a, n * D).view(-1, n, D) for a, n in (("q", H), ("k", G), ("v", G)))
            q, k = (self.rms(self.rotate(t, f, False, mult)) for t in (q, k))
            o = self.attend(q, k, v, m["scale"], m["mask"]["size"],
                            sink=torch.zeros(H, dtype=F64, device=h.device))
            return self.lin(o.flatten(1), p + "o", W)

        def delta(h, p, m):
            H, D = m["heads"], m["dim"]
            q, k, v = (self.conv(self.lin(h, p + a, H * D), f"{p}{a}.conv").view(-1, H, D) for a in "qkv")
            q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            g = torch.exp(-self.w(p + "A_log", H).exp() * torch.nn.functional.softplus(
                self.lin(h, p + "a", H, p + "dt_bias")))
            o = self.norm(self.scan(q * D ** -0.5, k, v, g, torch.sigmoid(self.lin(h, p + "b", H))), p + "norm")
            return self.lin(o.flatten(1) * torch.nn.functional.silu(self.lin(h, p + "g", H * D)), p + "o", W)
        x = self.w("embed", VOCAB, W)[self.tokens]
        for i, L in enumerate(c["layers"]):
            p = f"l{i}."
            h = self.norm(x, p + "norm1")
            h = h + (self.before(h, 1) - h) * self.w(p + "shift", W)
            mix = attention if L["type"] == "attention" else delta
            x = x + self.norm(mix(h, p + "mix.", L["mixer"]), p + "norm1b")
            z = self.lin(self.norm(x, p + "norm2"), p + "mlp.up", L["mlp"]["ff"])
            a, b = torch.nn.functional.softplus(self.w(p + "mlp.act", 2))
            neg = z.clamp(max=0.0)
            z = torch.where(z > 0, a * z * z, (0.5 + b) * (torch.expm1(neg) - neg)) + z / 2
            x = x + self.norm(self.lin(z, p + "mlp.down", W), p + "norm2b")
        return x

    def daburax(self):
        W, c = self.width, self.config
        silu = torch.nn.functional.silu

        def retention(h, p, m):
            H, D = m["heads"], m["dim"]
            f = self.freqs(D, m["rot"]["base"])
            q, k, v = (self.lin(h, p + a, H * D).view(-1, H, D) for a in "qkv")
            decay = torch.tensor(m["decay"], dtype=F64, device=h.device).expand(h.shape[0], H)
            o = self.rms(self.scan(self.rotate(q, f, False), self.rotate(k, f, False) * D ** -0.5, v, decay))
            return self.lin(o.flatten(1) * silu(self.lin(h, p + "g", H * D)), p + "o", W)

        def attention(h, p, m):
            H, G, D = m["heads"], m["kv_heads"], m["dim"]
            f = self.freqs(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"]["factor"])
            q, k, v = (self.lin(h, p + a, n * D, f"{p}{a}.b").view(-1, n, D)
                       for a, n in (("q", H), ("k", G), ("v", G)))
            o = self.attend(self.rotate(q, f, True), self.rotate(k, f, True), v, m["scale"],
                            sink=self.w(p + "sink", H))
            return self.lin(o.flatten(1), p + "o", W)

        def memory(h, p, m):
            H, D, cap = m["heads"], m["dim"], m["gate_cap"]
            q, k, v = (self.lin(h, p + a, H * D).view(-1, H, D) for a in "qkv")
            i, f = (cap * torch.tanh(self.lin(h, p + a, H, f"{p}{a}.b") / cap) for a in "if")
            i, f = self.pad(i), self.pad(torch.nn.functional.logsigmoid(f))
            top = torch.zeros_like(i[:, 0])                    # the running maximum starts at zero
            keep, write, tops = torch.empty_like(i), torch.empty_like(i), torch.empty_like(i)
            for t in range(i.shape[1]):
                new = torch.maximum(f[:, t] + top, i[:, t])
                keep[:, t], write[:, t] = torch.exp(f[:, t] + top - new), torch.exp(i[:, t] - new)
                top = tops[:, t] = new
            keep, write, tops = self.flat(keep), self.flat(write), self.flat(tops)
            k = k * write[:, :, None]
            one = torch.ones(v.shape[:2] + (1,), dtype=F64, device=v.device)
            o = self.scan(q * D ** -0.5, k, torch.cat([v, one], -1), keep)
            o = o[..., :-1] / (torch.maximum(o[..., -1:].abs(), torch.exp(-tops)[:, :, None]) + 1e-6)
            o = self.rms(o).flatten(1) * self.w(p + "norm", H * D)
            return self.lin(o * torch.sigmoid(self.lin(h, p + "g", H * D)), p + "o", W)

        def expert(h, p, ff):
            return self.lin(silu(self.lin(h, p + "gate", ff)) * self.lin(h, p + "up", ff), p + "down", W)

        def routed(h, p, mlp):
            r, ff = mlp["router"], mlp["expert"]["ff"]
            outputs = r["experts"] + r["identity"]
            s = torch.softmax(self.lin(h, p + "router", outputs), -1)
            choice = s + self.w(p + "correction", outputs)
            best = choice.view(-1, r["groups"]["count"], outputs // r["groups"]["count"])
            _, kept = torch.topk(best.amax(-1), r["groups"]["keep"], -1)
            closed = torch.ones(best.shape[:2], dtype=torch.bool, device=h.device).scatter_(1, kept, False)
            choice = best.masked_fill(closed[:, :, None], -math.inf).flatten(1)
            _, idx = torch.topk(choice, r["top"], -1)
            wgt = s.gather(1, idx)
            y = self.experts(h, p, mlp, idx, wgt, lambda q, rows, s: s * expert(rows, q, ff))
            y = y + (wgt * (idx >= r["experts"])).sum(-1, keepdim=True) * h       # identities
            return y + expert(h, p + "shared.", mlp["shared"]["ff"]) * torch.sigmoid(
                self.lin(h, p + "shared.sg", 1))
        b = c["embedding"]["bigram"]
        prev = self.before(self.tokens[:, None], 1)[:, 0]
        pair = torch.where(self.pos == 0, b["buckets"],
                           (prev * b["mul_prev"] + self.tokens * b["mul_cur"]) % b["buckets"])
        x = self.w("embed", VOCAB, W)[self.tokens] + self.w("bigram", b["buckets"] + 1, W)[pair]
        n = c["streams"]
        xs = torch.stack([x] * n)
        for i, L in enumerate(c["layers"]):
            p = f"l{i}."

            def sublayer(xs, at, run):
                w_in, w_out, mix = (self.w(f"{p}hc{at}.{a}", *s) for a, s in (
                    ("in", (n,)), ("out", (n,)), ("mix", (n, n))))
                y = run(self.norm(torch.einsum("s,snw->nw", w_in, xs), f"{p}norm{at}", 1.0))
                return torch.einsum("st,snw->tnw", mix, xs) + c["residual_mult"] * w_out[:, None, None] * y
            m = L["mixer"]
            if L["type"] == "retention":
                xs = sublayer(xs, 1, lambda h: retention(h, p + "mix.", m))
            else:
                xs = sublayer(xs, 1, lambda h: m["left_scale"] * attention(h, p + "mix.left.", m["left"])
                              + m["right_scale"] * memory(h, p + "mix.right.", m["right"]))
            xs = sublayer(xs, 2, lambda h: routed(h, p + "mlp.", L["mlp"]))
        return xs.sum(0)


@torch.no_grad()
def exact(case, seed):
    return _Plain(case, seed).logits()
