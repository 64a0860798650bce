"""Gated delta rule with a decay per key channel or per head over per-request state
(``csrc/delta_rule.cu``)."""
from __future__ import annotations

from ctypes import addressof, c_float, c_int, c_void_p

import torch

from . import _Counter, _code, _cuda, _fn, _ok, _p, _stream


MAX_KEY_SIZE = 256        # the recurrence kernel's largest
# Steps with a portion of at least this many tokens take the recurrence with one decay a head eight
# tokens at a time.
CHUNKED_MIN_TOKENS = 16


def prepare(proj: torch.Tensor, b_off: int, a: torch.Tensor, conv_w: torch.Tensor,
            dt_bias: torch.Tensor, A_log: torch.Tensor, state: torch.Tensor, ctx, H: int, G: int,
            D: int, Vd: int, taps: int, conv_off: int):
    """``proj [T, >= 2 G D + H Vd + ...]``: the q | k | v projections first, the ``H`` beta columns
    at ``b_off``; ``a [T, H D]`` fp32: the decay's pre-activation.  Convolves (reading the slots'
    last inputs, and bringing them up to date afterwards), activates, normalises; returns fp32
    ``(q [T, G, D], k [T, G, D], v [T, H, Vd], g [T, H, D], beta [T, H])``."""
    _cuda(proj, a, conv_w, dt_bias, A_log, state)
    T = proj.shape[0]
    assert proj.dim() == 2 and proj.stride(1) == 1
    assert a.dtype == torch.float32 and a.is_contiguous() and a.shape == (T, H * D)
    assert state.dtype == torch.float32 and state.dim() == 2 and state.is_contiguous()
    ch = 2 * G * D + H * Vd
    assert conv_w.dtype == torch.float32 and conv_w.shape == (ch, taps) and conv_w.is_contiguous()
    dev = proj.device
    qn = torch.empty((T, G, D), dtype=torch.float32, device=dev)
    kn = torch.empty_like(qn)
    v = torch.empty((T, H, Vd), dtype=torch.float32, device=dev)
    g = torch.empty((T, H, D), dtype=torch.float32, device=dev)
    beta = torch.empty((T, H), dtype=torch.float32, device=dev)
    f = _fn("delta_rule", "gf_delta_prepare",
            [c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
             c_void_p, c_void_p] + [c_int] * 9 + [c_void_p] * 5 + [c_int, c_void_p],
            kernels=2)
    rc = f(_p(proj), proj.stride(0), int(b_off), _p(a), _p(conv_w), _p(dt_bias), _p(A_log),
           _p(state), _p(ctx.seq_of_token), _p(ctx.cu_seqlens_q), _p(ctx.slot_ids), T,
           ctx.num_seqs, H, G, D, Vd, taps, state.stride(0), int(conv_off), _p(qn), _p(kn), _p(v),
           _p(g), _p(beta), _code(proj.dtype), _stream())
    if rc == -3:
        raise ValueError("the delta-rule kernels need heads to be a multiple of kv heads and key "
                         f"sizes up to 256; got {H} heads, {G} kv heads, key size {D}")
    _ok(rc, "delta_prepare")
    return qn, kn, v, g, beta


def prepare_heads(proj: torch.Tensor, a_off: int, b_off: int, conv_w: torch.Tensor,
                  dt_bias: torch.Tensor, A_log: torch.Tensor, state: torch.Tensor, ctx, H: int,
                  G: int, D: int, Vd: int, taps: int, conv_off: int):
    """The same with one decay a head: ``proj [T, >= 2 G D + H Vd + ...]`` fp32 holds the q | k | v
    projections first, the heads' decay pre-activations at ``a_off`` and the beta columns at
    ``b_off``.  Returns fp32 ``(q [T, G, D], k [T, G, D], v [T, H, Vd], g [T, H], beta [T, H])``."""
    _cuda(proj, conv_w, dt_bias, A_log, state)
    T = proj.shape[0]
    assert proj.dim() == 2 and proj.stride(1) == 1 and proj.dtype == torch.float32
    assert max(a_off, b_off) + H <= proj.shape[1]
    assert state.dtype == torch.float32 and state.dim() == 2 and state.is_contiguous()
    ch = 2 * G * D + H * Vd
    assert conv_w.dtype == torch.float32 and conv_w.shape == (ch, taps) and conv_w.is_contiguous()
    assert dt_bias.dtype == torch.float32 and dt_bias.numel() == H
    assert A_log.dtype == torch.float32 and A_log.numel() == H
    dev = proj.device
    qn = torch.empty((T, G, D), dtype=torch.float32, device=dev)
    kn = torch.empty_like(qn)
    v = torch.empty((T, H, Vd), dtype=torch.float32, device=dev)
    g = torch.empty((T, H), dtype=torch.float32, device=dev)
    beta = torch.empty_like(g)
    f = _fn("delta_rule", "gf_delta_prepare_heads",
            [c_void_p, c_int, c_int, c_int] + [c_void_p] * 7 + [c_int] * 10 + [c_void_p] * 6)
    rc = f(_p(proj), proj.stride(0), int(a_off), int(b_off), _p(conv_w), _p(dt_bias), _p(A_log),
           _p(state), _p(ctx.seq_of_token), _p(ctx.cu_seqlens_q), _p(ctx.slot_ids), T,
           ctx.num_seqs, int(ctx.max_q_len), H, G, D, Vd, taps, state.stride(0), int(conv_off),
           _p(qn), _p(kn), _p(v), _p(g), _p(beta), _stream())
    if rc == -3:
        raise ValueError("the delta-rule kernels need heads to be a multiple of kv heads and key "
                         f"sizes up to {MAX_KEY_SIZE}; got {H} heads, {G} kv heads, key size {D}")
    _ok(rc, "delta_prepare_heads")
    return qn, kn, v, g, beta


def state_step(q, k, v, g, state, ctx, H: int, G: int, D: int, Vd: int, o, c=None, skip=None,
               beta=None) -> bool:
    """One token, or none, of every request (``csrc/state_step.cu``): rows of ``q``, ``k`` (``G D``), ``v``, ``o``
    (``H Vd``), ``g`` (``H`` or ``H D``) and ``c`` (``H``), all fp32 with a row stride; with ``beta [T, H]``
    the delta rule, else ``S <- g S + c k v^T``.  ``False`` where the kernel does not take the case."""
    f = _fn("state_step", "gf_state_step",
            [c_void_p, c_int] * 4 + [c_int, c_void_p, c_int] + [c_void_p] * 3 + [c_int, c_void_p, c_void_p] +
            [c_int] * 5 + [c_void_p, c_int, c_void_p])
    rc = f(_p(q), q.stride(0), _p(k), k.stride(0), _p(v), v.stride(0), _p(g), g.stride(0),
           g.shape[1] // H, _p(c), c.stride(0) if c is not None else 0, _p(skip), _p(beta), _p(state),
           state.stride(0), _p(ctx.cu_seqlens_q), _p(ctx.slot_ids), ctx.num_seqs, H, G, D, Vd, _p(o),
           o.stride(0), _stream())
    if rc == -6:
        return False
    _ok(rc, "state_step")
    return True


def chunk_words(T: int, B: int, heads: int, D: int, one_decay: int) -> int:
    """fp32 words of scratch with which ``heads`` heads of a step go eight tokens at a time."""
    from ctypes import c_longlong

    from .build import load_library
    f = load_library("delta_rule").gf_delta_chunk_words
    f.argtypes, f.restype = [c_int] * 5, c_longlong
    return int(f(T, B, heads, D, one_decay))


def recurrence(qn, kn, v, g, beta, state: torch.Tensor, ctx) -> torch.Tensor:
    """Advance every request's state over its tokens of this step; returns ``o [T, H, Vd]`` fp32.
    ``g``: ``[T, H, D]``, or ``[T, H]`` for one decay a head (long portions then go eight tokens at a
    time, and steps of single tokens on a kernel of their own; with a decay a channel every step goes token
    by token, so that a token's bits do not depend on how the portions are cut)."""
    T, G, D = qn.shape
    H, Vd = v.shape[1], v.shape[2]
    o = torch.empty((T, H, Vd), dtype=torch.float32, device=qn.device)
    f = _fn("delta_rule", "gf_delta_recurrence",
            [c_void_p] * 8 + [c_int] * 6 + [c_void_p, c_int, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p],
            kernels=0)
    one = int(g.dim() == 2)
    scratch, longest = None, int(ctx.max_q_len if one else getattr(ctx, "max_q_len", 0))
    if one and longest == 1 and state_step(qn.view(T, G * D), kn.view(T, G * D), v.view(T, H * Vd),
                                           g.view(T, -1), state, ctx, H, G, D, Vd, o.view(T, H * Vd), beta=beta):
        return o
    if one and longest >= CHUNKED_MIN_TOKENS:
        scratch = torch.empty(chunk_words(T, ctx.num_seqs, H, D, one), dtype=torch.float32,
                              device=qn.device)
    # single tokens in front of portions, as the scheduler orders a mixed step
    singles, q_lens = 0, getattr(ctx, "q_lens_host", ())
    if longest > 1 and len(q_lens) == ctx.num_seqs:
        while singles < len(q_lens) and q_lens[singles] == 1:
            singles += 1
    launches = c_int()
    rc = f(_p(qn), _p(kn), _p(v), _p(g), _p(beta), _p(state), _p(ctx.cu_seqlens_q),
           _p(ctx.slot_ids), ctx.num_seqs, H, G, D, Vd, state.stride(0), _p(o), one,
           _p(scratch), longest, T, singles, addressof(launches), _stream())
    if rc == -3:
        raise ValueError(f"the delta-rule recurrence takes key sizes up to {MAX_KEY_SIZE}, got {D}")
    _ok(rc, "delta_recurrence")
    _Counter.launches += launches.value
    return o


def output(o: torch.Tensor, gate: torch.Tensor, w: torch.Tensor, eps: float,
           dtype: torch.dtype) -> torch.Tensor:
    """``o / rms(o) * w * sigmoid(gate)`` per head; ``[T, H Vd]`` in ``dtype``."""
    _cuda(o, gate, w)
    T, H, Vd = o.shape
    assert gate.stride(1) == 1 and gate.shape == (T, H * Vd) and gate.dtype == dtype
    assert w.dtype == torch.float32 and w.numel() == Vd
    out = torch.empty((T, H * Vd), dtype=dtype, device=o.device)
    f = _fn("delta_rule", "gf_delta_output",
            [c_void_p, c_void_p, c_int, c_void_p, c_float, c_void_p, c_int, c_int, c_int, c_int,
             c_void_p])
    _ok(f(_p(o), _p(gate), gate.stride(0), _p(w), float(eps), _p(out), T, H, Vd, _code(dtype),
          _stream()), "delta_output")
    return out
