"""Chunked HDLA operator: ``chunk_hrdplr_delta_rule`` and its autograd function.

Same names, argument order, defaults and return values as the reference's
``HRDPLR/hrdplr.py:286-318`` (entry point) and ``:101-284`` (``ChunkDPLRDeltaRuleFunction``); the
stage sequence itself runs inside libhdla (``hdla_chunk_fwd`` / ``hdla_chunk_bwd``).
"""
from __future__ import annotations

import ctypes as C
import functools
import os
import warnings
from typing import Optional, Tuple

import torch

from . import _lib

autocast_custom_fwd = functools.partial(torch.amp.custom_fwd, device_type="cuda")
autocast_custom_bwd = functools.partial(torch.amp.custom_bwd, device_type="cuda")


def contiguous(fn):
    """Make every tensor argument contiguous (reference: HRDPLR/utils.py:14-25)."""
    @functools.wraps(fn)
    def wrapper(ctx, *args, **kwargs):
        return fn(ctx,
                  *(i if not isinstance(i, torch.Tensor) else i.contiguous() for i in args),
                  **{k: (v if not isinstance(v, torch.Tensor) else v.contiguous()) for k, v in kwargs.items()})
    return wrapper


def _tc_shape(q, v, RANK_AB: int) -> bool:
    """Whether the bf16 tensor-core pipeline takes this problem (at its own chunk of 64): bf16, rank 2, head dims
    that are multiples of 8 up to 128 (smaller ones fill a prefix of the 128-wide tiles)."""
    T, K, V = q.shape[1], q.shape[-1], v.shape[-1]
    return (q.dtype == torch.bfloat16 and RANK_AB == 2 and K % 8 == 0 and V % 8 == 0 and 8 <= K <= 128
            and 8 <= V <= 128 and T > 32)


def _internal_chunk(q, v, RANK_AB: int, chunk_size: int) -> int:
    """Chunk size actually used.  The operator's result does not depend on the chunk size (it only sets how
    the recurrence is blocked), and the reference layer asks for 16 (HRDPLR/hdla_custom.py:308) only because its
    own backward is limited to that.  Problems the tensor-core pipeline supports are therefore run at its chunk
    of 64 whatever was requested; ``HDLA_HONOR_CHUNK=1`` keeps the requested value."""
    if (os.environ.get("HDLA_HONOR_CHUNK", "0") != "1" and _tc_shape(q, v, RANK_AB)
            and os.environ.get("HDLA_FORCE_SIMT", "0") != "1"):
        return 64
    return chunk_size


def _dims(q, v, a, gk, RANK_AB: int, chunk_size: int, flags: int = 0, cu_seqlens=None) -> _lib.HdlaDims:
    chunk_size = _internal_chunk(q, v, RANK_AB, chunk_size)
    B, T, H, K = q.shape
    if os.environ.get("HDLA_FORCE_SIMT", "0") == "1":      # debugging aid: fp32 CUDA-core pipeline for any dtype
        flags |= _lib.FLAG_FORCE_SIMT
    if os.environ.get("HDLA_FUSED_PREP", "0") == "1":      # one-kernel chunk preparation (see include/hdla.h)
        flags |= _lib.FLAG_FUSED_PREP
    d = _lib.HdlaDims(B, T, H, K, v.shape[-1], RANK_AB, chunk_size, _lib.dtype_code(q.dtype),
                      _lib.dtype_code(gk.dtype), flags)
    if cu_seqlens is not None:
        d.with_seqlens(cu_seqlens)
    return d


def _seq_offsets(cu_seqlens):
    """cu_seqlens (tensor or sequence of ints) -> tuple of python ints, or None.  The library sizes its grids from
    the offsets, so they are needed on the host (a device tensor is copied, which synchronises -- as the
    reference's chunk-index preparation does)."""
    if cu_seqlens is None:
        return None
    if isinstance(cu_seqlens, torch.Tensor):
        cu_seqlens = cu_seqlens.detach().cpu().tolist()
    return tuple(int(x) for x in cu_seqlens)


def _check_shapes(q, k, v, a, b, gk, RANK_AB, initial_state, n_states=None):
    B, T, H, K = q.shape
    if k.shape != q.shape or gk.shape != q.shape:
        raise ValueError(f"k {tuple(k.shape)} and gk {tuple(gk.shape)} must match q {tuple(q.shape)}")
    if v.shape[:3] != q.shape[:3]:
        raise ValueError(f"v {tuple(v.shape)} must be [B, T, H, V] with q {tuple(q.shape)}")
    if a.shape != (B, T * RANK_AB, H, K) or b.shape != a.shape:
        raise ValueError(f"a {tuple(a.shape)} / b {tuple(b.shape)} must be [B, T*RANK_AB, H, K] = "
                         f"{(B, T * RANK_AB, H, K)}")
    if not (a.dtype == b.dtype == q.dtype):
        raise TypeError("a and b must have the dtype of q, k, v")
    N = B if n_states is None else n_states
    if initial_state is not None and initial_state.shape != (N, H, K, v.shape[-1]):
        raise ValueError(f"initial_state {tuple(initial_state.shape)} must be [{N}, H, K, V] = "
                         f"{(N, H, K, v.shape[-1])}")


def workspace_bytes(dims: _lib.HdlaDims, with_backward: bool) -> int:
    n = _lib.load().hdla_chunk_workspace_bytes(C.byref(dims), int(with_backward))
    if n == 0:
        raise RuntimeError(f"unsupported problem: {_lib.last_error()}")
    return n


# ---- device status words ----------------------------------------------------------------------
# The bf16 tensor-core kernels report in the first bytes of the workspace (see include/hdla.h): a device-side wait
# that ran out, a chunk whose total log decay is beyond what the pipeline represents, the largest chunk decay of the
# call.  The protocol -- a copy to pinned memory after every call, looked at when the device is used next, and a
# forward that waits and is rerun on the fp32 pipeline while an overflow is plausible -- is in csrc/binding.cpp.
_warned_fallback = False


def warn_fallback() -> None:
    """Called when a forward call is rerun on the fp32 pipeline: warns the first time."""
    global _warned_fallback
    if not _warned_fallback:
        _warned_fallback = True
        warnings.warn("hdla_impl_b200: a chunk's total log decay exceeds what the bf16 tensor-core pipeline represents; "
                      "such calls are rerun on the fp32 CUDA-core pipeline (correct, much slower)", RuntimeWarning,
                      stacklevel=3)


class _DecayHistory:
    """``["decay"]``: the largest chunk decay seen on a device (None: nothing seen yet); can be set."""

    def __init__(self, index: int):
        self.index = index

    def __getitem__(self, key):
        if key != "decay":
            raise KeyError(key)
        return _lib.native().decay(self.index)

    def __setitem__(self, key, value):
        if key != "decay":
            raise KeyError(key)
        _lib.native().set_decay(self.index, value)


def _status_state(dev) -> _DecayHistory:
    return _DecayHistory(dev.index if isinstance(dev, torch.device) else int(dev))


def check_status(dev=None, wait: bool = False) -> None:
    """Raise if an earlier call on ``dev`` reported a problem. ``wait`` synchronises first."""
    index = -1 if dev is None else (dev.index if isinstance(dev, torch.device) else int(dev))
    _lib.native().status_check(index, bool(wait))


def _post_status(ws: torch.Tensor, dev) -> None:
    """Enqueue the copy of the status words of the call that just used ``ws``."""
    _lib.native().status_post(ws)


def _alloc_ws(nbytes: int, device) -> torch.Tensor:
    return torch.empty(nbytes, dtype=torch.uint8, device=device)


def save_workspace_default() -> bool:
    """Whether forward keeps its intermediates for backward (default) or backward recomputes them
    like the reference does (``HDLA_RECOMPUTE=1``; trades time for activation memory)."""
    return os.environ.get("HDLA_RECOMPUTE", "0") != "1"


def chunk_hrdplr_fwd(q, k, v, a, b, gk, scale, initial_state, output_final_state, RANK_AB, head_first, chunk_size):
    """Forward stage sequence (reference: HRDPLR/hrdplr.py:25-99). Returns ``(o, final_state)``."""
    o, ht, _, _ = _chunk_fwd(q, k, v, a, b, gk, scale, initial_state, output_final_state, RANK_AB, head_first,
                             chunk_size)
    return o, ht


def _chunk_fwd(q, k, v, a, b, gk, scale, initial_state, output_final_state, RANK_AB, head_first, chunk_size,
               _keep_ws: bool = False, cu_seqlens=None):
    """``chunk_hrdplr_fwd`` returning ``(o, final_state, workspace, used_fp32_pipeline)``; with ``_keep_ws`` the
    workspace is sized for, and keeps what, ``hdla_chunk_bwd(HDLA_FLAG_WS_HOLDS_FWD)`` needs."""
    assert head_first is False, "head_first=True is not supported (as in the reference)"
    _lib.require_cuda(q, k, v, a, b, gk, initial_state)
    N = None if cu_seqlens is None else len(cu_seqlens) - 1
    _check_shapes(q, k, v, a, b, gk, RANK_AB, initial_state, N)
    rest = (RANK_AB, float(scale), _state(initial_state), output_final_state,
            _internal_chunk(q, v, RANK_AB, chunk_size), cu_seqlens, bool(_keep_ws))
    r = _lib.native().chunk(*[_plain(t) for t in (q, k, v, a, b, gk)], *rest)
    if r is NotImplemented:
        workspace_bytes(_dims(q, v, a, gk, RANK_AB, chunk_size, 0, cu_seqlens), bool(_keep_ws))      # says why
        raise TypeError("q, k, v must share one dtype, gk and the states must be floating-point tensors")
    return r


def _plain(t):
    """The tensor itself, detached and without its subclass."""
    return t if t is None else t.detach().as_subclass(torch.Tensor)


def _state(t):
    """An initial state as the native path takes it: of a floating-point type (an integer one is converted)."""
    return _plain(t) if t is None or t.is_floating_point() else _plain(t).to(torch.float32)


class ChunkDPLRDeltaRuleFunction(torch.autograd.Function):
    """Autograd wrapper (reference: HRDPLR/hrdplr.py:101-284): forward saves the inputs; backward
    receives ``(do, dht)`` and returns gradients for q,k,v,a,b,gk and the initial state.  (``chunk_hrdplr_delta_rule``
    takes the same steps in native code where its arguments are plain tensors.)"""

    @staticmethod
    @contiguous
    @autocast_custom_fwd
    def forward(ctx, q, k, v, a, b, gk, scale, initial_state, output_final_state, RANK_AB, head_first, chunk_size,
                cu_seqlens=None):
        keep = save_workspace_default() and any(
            isinstance(t, torch.Tensor) and t.requires_grad for t in (q, k, v, a, b, gk, initial_state))
        o, final_state, ctx.ws, ctx.force_simt = _chunk_fwd(q, k, v, a, b, gk, scale, initial_state, output_final_state,
                                                            RANK_AB, head_first, chunk_size, _keep_ws=keep,
                                                            cu_seqlens=cu_seqlens)
        ctx.cu_seqlens = cu_seqlens
        ctx.save_for_backward(q, k, v, a, b, gk, initial_state)
        ctx.head_first = head_first
        ctx.scale = scale
        ctx.chunk_size = chunk_size
        ctx.output_final_state = output_final_state
        ctx.RANK_AB = RANK_AB
        return o.to(q.dtype), final_state

    @staticmethod
    @contiguous
    @autocast_custom_bwd
    def backward(ctx, do, dht):
        q, k, v, a, b, gk, initial_state = ctx.saved_tensors
        ws, ctx.ws = ctx.ws, None
        grads = _lib.native().chunk_backward(*[_plain(t) for t in (q, k, v, a, b, gk)], ctx.RANK_AB, float(ctx.scale),
                                             _state(initial_state), _plain(do), _plain(dht), ws,
                                             _internal_chunk(q, v, ctx.RANK_AB, ctx.chunk_size), ctx.cu_seqlens,
                                             ctx.force_simt)
        dq, dk, dv, da, db, dgk, dh0 = grads
        if dh0 is not None and initial_state.dtype != torch.float32:
            dh0 = dh0.to(initial_state.dtype)
        return dq, dk, dv, da, db, dgk, None, dh0, None, None, None, None, None


def _packed_supported(q, v, RANK_AB: int) -> bool:
    return _tc_shape(q, v, RANK_AB) and os.environ.get("HDLA_FORCE_SIMT", "0") != "1" \
        and os.environ.get("HDLA_HONOR_CHUNK", "0") != "1"


@torch.compiler.disable
def chunk_hrdplr_delta_rule(
    q: torch.Tensor,   # [B, T, H, K]
    k: torch.Tensor,   # [B, T, H, K]
    v: torch.Tensor,   # [B, T, H, V]
    a: torch.Tensor,   # [B, T * RANK_AB, H, K]
    b: torch.Tensor,   # [B, T * RANK_AB, H, K]
    gk: torch.Tensor,  # [B, T, H, K]  log decay
    RANK_AB: int,
    scale: Optional[float] = None,
    initial_state: Optional[torch.Tensor] = None,   # [B, H, K, V]
    output_final_state: bool = False,
    head_first: bool = False,
    chunk_size: int = 32,
    cu_seqlens=None,
) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """Drop-in for the reference's ``chunk_hrdplr_delta_rule`` (HRDPLR/hrdplr.py:286-318).

    ``cu_seqlens`` (an extension; the reference plumbs it only into its chunk kernels, HRDPLR/fwd_triton.py:618-623,
    HRDPLR/bwd_triton.py:919-924): offsets of sequences packed along T in a batch of one, as in
    ``fused_recurrent_dplr_delta_rule``; ``initial_state`` / the final state are then ``[n_seqs, H, K, V]``.  bf16
    problems of the tensor-core pipeline run packed (chunks never straddle two sequences; one scan per sequence
    and head); anything else is computed sequence by sequence."""
    offsets = None if cu_seqlens is None else _seq_offsets(cu_seqlens)
    if head_first is False:
        r = (_lib._native or _lib.native()).chunk(q, k, v, a, b, gk, RANK_AB, scale, initial_state, output_final_state,
                                                  chunk_size, offsets, None)
        if r is not NotImplemented:
            return r
    # what the native path does not take: other problems of a packed batch, tensor subclasses, invalid arguments
    assert q.dtype == k.dtype == v.dtype
    scale = k.shape[-1] ** -0.5 if scale is None else scale
    if offsets is not None:
        if q.shape[0] != 1:
            raise ValueError(f"The batch size is expected to be 1 rather than {q.shape[0]} when using `cu_seqlens`."
                             f"Please flatten variable-length inputs before processing.")
        if initial_state is not None and initial_state.shape[0] != len(offsets) - 1:
            raise ValueError(f"The number of initial states is expected to be equal to the number of input sequences, "
                             f"i.e., {len(offsets) - 1} rather than {initial_state.shape[0]}.")
        if offsets[0] != 0 or offsets[-1] != q.shape[1] or any(y < x for x, y in zip(offsets, offsets[1:])):
            raise ValueError(f"cu_seqlens {offsets} must rise from 0 to T={q.shape[1]}")
        if not _packed_supported(q, v, RANK_AB):
            outs, states = [], []
            for s_, (lo, hi) in enumerate(zip(offsets, offsets[1:])):
                if hi == lo:
                    states.append(initial_state[s_:s_ + 1].float() if initial_state is not None else
                                  q.new_zeros(1, q.shape[2], q.shape[3], v.shape[-1], dtype=torch.float32))
                    continue
                h0 = None if initial_state is None else initial_state[s_:s_ + 1]
                o_s, ht_s = ChunkDPLRDeltaRuleFunction.apply(
                    q[:, lo:hi], k[:, lo:hi], v[:, lo:hi], a[:, lo * RANK_AB:hi * RANK_AB],
                    b[:, lo * RANK_AB:hi * RANK_AB], gk[:, lo:hi], scale, h0, output_final_state, RANK_AB,
                    head_first, chunk_size)
                outs.append(o_s)
                states.append(ht_s)
            return torch.cat(outs, 1), (torch.cat(states, 0) if output_final_state else None)
    o, final_state = ChunkDPLRDeltaRuleFunction.apply(
        q, k, v, a, b, gk, scale, initial_state, output_final_state, RANK_AB, head_first, chunk_size, offsets)
    return o, final_state
