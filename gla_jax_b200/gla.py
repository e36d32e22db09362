"""The GLA operators with the reference's signatures (gla.py of zhixuan-lin/gla-jax), backed
by libgla_b200.so.

    chunk_gla(hidden_init, log_fgate, value, key, query, chunk_size, ...)   gla.py:657
    recurrent_gla(hidden_init, log_fgate, value, key, query, reverse, ...)  gla.py:405
    recurrent_gla_naive(hidden, log_fgate, value, key, query, reverse)      gla.py:26

All return ``(hidden_final, out)``.  Shapes are the reference's per-sequence shapes
``log_fgate, value, key, query : (T, H, D)``, ``hidden : (H, D, D)``; where the reference
adds a batch axis with ``jax.vmap`` (gla.py:1335), pass arrays with a leading batch axis
instead (``(B, T, H, D)`` and ``(B, H, D, D)``) — the kernels take the batch natively.

This adapter holds device memory in torch CUDA tensors and differentiates through autograd
nodes that mirror the reference's ``jax.custom_vjp`` pairs (gla.py:362/441 and gla.py:628/655);
the nodes and the host path to the library calls are native (csrc/gla_host.cc).  The JAX adapter (XLA FFI handlers plus
``jax.custom_vjp``) is ``jax_ffi.py`` / ``csrc/gla_xla_ffi.cc``; both call the same C ABI.
There is no CPU path: CPU tensors raise.
"""
from __future__ import annotations

from typing import Tuple

import torch

from . import _lib

_DT = {torch.float32: _lib.GLA_F32, torch.bfloat16: _lib.GLA_BF16}


def _ptr(t):
    return None if t is None else t.data_ptr()


_stream = _lib.stream_of


def _refused(what, hidden, log_fgate, value, key, query):
    """The native host path did not take these arguments: raise the error that says why (the reference's trace-time
    asserts, gla.py:118-127, 498-500)."""
    if not value.is_cuda:
        raise RuntimeError("gla_jax_b200 operators need CUDA tensors; there is no CPU fallback")
    if value.dim() not in (3, 4):
        raise ValueError(f"value must be (T,H,D) or (B,T,H,D), got {tuple(value.shape)}")
    batched = value.dim() == 4
    if not (log_fgate.shape == value.shape == key.shape == query.shape):
        raise ValueError("log_fgate, value, key, query must have the same shape "
                         f"({tuple(log_fgate.shape)}, {tuple(value.shape)}, {tuple(key.shape)}, {tuple(query.shape)})")
    want = (*value.shape[:-3], value.shape[-2], value.shape[-1], value.shape[-1])
    if tuple(hidden.shape) != want:
        raise ValueError(f"hidden must be {'(B,' if batched else '('}H,D,D) = {want}, got {tuple(hidden.shape)}")
    if value.dtype not in _DT:
        raise TypeError(f"unsupported dtype {value.dtype}: float32 and bfloat16 are implemented")
    if not (key.dtype == query.dtype == hidden.dtype == value.dtype):
        raise TypeError("value, key, query and hidden must share one dtype")
    _stream(value.device)
    raise ValueError(f"{what}: all arrays must be on {value.device}")


def _chunk_fwd_raw(hidden, g32, v, k, q, chunk, impl, need_grad):
    """gla_chunk_fwd on batched contiguous tensors -> (hidden_final, out, (saved,) or ())."""
    lib = _lib.load()
    B, T, H, D = v.shape
    dt = _DT[v.dtype]
    dev = v.device
    ws_n = lib.gla_chunk_fwd_workspace_bytes(B, T, H, D, chunk, dt, impl)
    if ws_n == 0:
        raise _lib.GlaError(f"chunk_gla: unsupported configuration T={T} H={H} D={D} chunk={chunk} dtype={v.dtype}")
    saved = None
    if need_grad:
        saved = torch.empty(lib.gla_chunk_saved_bytes(B, T, H, D, chunk, dt, impl), dtype=torch.uint8, device=dev)
    ws = torch.empty(ws_n, dtype=torch.uint8, device=dev)
    hf = torch.empty_like(hidden)
    out = torch.empty_like(v)
    st = lib.gla_chunk_fwd(_stream(dev), B, T, H, D, chunk, dt, impl, _ptr(hidden), _ptr(g32), _ptr(v), _ptr(k),
                           _ptr(q), _ptr(hf), _ptr(out), _ptr(saved), _ptr(ws), ws_n)
    _lib.check(st, "gla_chunk_fwd")
    return hf, out, ((saved,) if need_grad else ())


def _chunk_bwd_raw(g32, v, k, q, residuals, dhf, dout, chunk, impl):
    """gla_chunk_bwd -> (dhidden_init, dlog_fgate (float32), dvalue, dkey, dquery)."""
    lib = _lib.load()
    (saved,) = residuals
    B, T, H, D = v.shape
    dt = _DT[v.dtype]
    dev = v.device
    ws_n = lib.gla_chunk_bwd_workspace_bytes(B, T, H, D, chunk, dt, impl)
    ws = torch.empty(ws_n, dtype=torch.uint8, device=dev)
    dh = torch.empty(B, H, D, D, dtype=v.dtype, device=dev)
    dg = torch.empty_like(g32)
    dv, dk, dq = torch.empty_like(v), torch.empty_like(k), torch.empty_like(q)
    st = lib.gla_chunk_bwd(_stream(dev), B, T, H, D, chunk, dt, impl, _ptr(g32), _ptr(v), _ptr(k), _ptr(q),
                           _ptr(saved), _ptr(dhf), _ptr(dout), _ptr(dh), _ptr(dg), _ptr(dv), _ptr(dk), _ptr(dq),
                           _ptr(ws), ws_n)
    _lib.check(st, "gla_chunk_bwd")
    return dh, dg, dv, dk, dq


def chunk_gla(hidden_init, log_fgate, value, key, query, chunk_size: int,
              block_size_t: int = 64, block_size_d: int = 64, interpret: bool = False,
              num_warps: int = 4, num_stages: int = 2, impl: str = "auto") -> Tuple[torch.Tensor, torch.Tensor]:
    """Chunk-wise GLA with multi-scale secondary chunking (reference: gla.py:657-692).

    ``block_size_t``, ``block_size_d``, ``num_warps``, ``num_stages`` and ``interpret`` are
    the reference's Triton tuning knobs; they are accepted for caller compatibility and
    ignored (the CUDA kernels fix their own tiling).  ``impl`` selects the kernel family:
    ``"auto"`` (tensor cores when the shape has a kernel), ``"tcgen05"`` or ``"fp32"``.
    """
    del block_size_t, block_size_d, interpret, num_warps, num_stages
    chunk_size, impl = int(chunk_size), _lib.IMPL_BY_NAME[impl]
    r = _lib.native().chunk_gla(hidden_init, log_fgate, value, key, query, chunk_size, impl)
    if r is not None:
        return r
    T = value.shape[-3]
    if chunk_size <= 0 or chunk_size & (chunk_size - 1):
        raise ValueError(f"Chunk length must be power of 2, but got {chunk_size}")   # gla.py:500
    if T % chunk_size:
        raise ValueError(f"sequence length {T} is not a multiple of chunk_size {chunk_size}")  # gla.py:674
    return _refused("chunk_gla", hidden_init, log_fgate, value, key, query)


def recurrent_gla(hidden_init, log_fgate, value, key, query, reverse: bool = False,
                  max_block_size: int = 64, num_warps: int = 1, num_stages: int = 1,
                  interpret: bool = False) -> Tuple[torch.Tensor, torch.Tensor]:
    """Exact recurrence in float32 (reference: gla.py:405-439).  At head sizes 32, 64 and 128, from 48 tokens on (up to 192
    where the batch has fewer than 16 heads), chunks run side by side, with a float32 state per head and 64 tokens (32 where
    an array at head size 128 is float32) in memory during the call: D * D / 16 (D * D / 8) bytes per token and head in the
    forward, twice that in the backward.  Where that does not fit, and elsewhere, it walks the tokens and writes no states.
    ``max_block_size``, ``num_warps``, ``num_stages``, ``interpret`` are accepted and ignored."""
    del max_block_size, num_warps, num_stages, interpret
    r = _lib.native().recurrent_gla(hidden_init, log_fgate, value, key, query, bool(reverse), False)
    if r is not None:
        return r
    if value.shape[-2] != key.shape[-2]:
        raise ValueError("value and key must have the same number of heads")   # gla.py:417
    return _refused("recurrent_gla", hidden_init, log_fgate, value, key, query)


def recurrent_gla_naive(hidden, log_fgate, value, key, query, reverse: bool = False):
    """The definitional recurrence (reference: gla.py:26-47).  On this backend it runs the same
    on-chip recurrence kernel as ``recurrent_gla``; as in the reference ``out`` is float32
    and ``hidden_final`` keeps ``hidden``'s dtype (gla.py:43-46)."""
    r = _lib.native().recurrent_gla(hidden, log_fgate, value, key, query, bool(reverse), True)
    return r if r is not None else _refused("recurrent_gla_naive", hidden, log_fgate, value, key, query)


def chunk_gla_packed(hidden_init, log_fgate, value, key, query, cu_seqlens, chunk_size: int = 128):
    """``chunk_gla`` for variable-length sequences packed end to end on one time axis.

    ``value/key/query/log_fgate`` are (T, H, D) holding ``nseq`` sequences back to back; ``cu_seqlens`` holds the
    ``nseq + 1`` token offsets (0 first, T last); ``hidden_init`` is (nseq, H, D, D).  Returns
    ``(hidden_final (nseq, H, D, D), out (T, H, D))``, equal to calling ``chunk_gla`` on each sequence;
    differentiable.  The reference has one length per call and asserts T % chunk == 0 (gla.py:499-500, 674); this
    runs on the tensor-core kernels only (bf16, D = 128).

    Offsets given as a list or CPU tensor may be ANY rising sequence: every sequence starts a chunk of its own at its
    first token and the rows of its last chunk past its end are masked inside the kernels.  Offsets given as a CUDA
    int32 tensor are used as they are, without a host round trip, and must be multiples of 128 (the kernels clamp
    anything else and count it in ``gla_device_bad_offsets``)."""
    cu = cu_seqlens if torch.is_tensor(cu_seqlens) else torch.tensor(cu_seqlens, dtype=torch.int32)
    if cu.dtype != torch.int32:
        cu = cu.to(torch.int32)
    if cu.is_cuda and (cu.dim() != 1 or cu.device != value.device):
        cu = cu.to(value.device).reshape(-1)
    r = _lib.native().chunk_gla_packed(hidden_init, log_fgate, value, key, query, cu, int(chunk_size))
    if r is not None:
        return r
    if value.dim() != 3 or hidden_init.dim() != 4:
        raise ValueError("chunk_gla_packed: expected value (T, H, D) and hidden_init (nseq, H, D, D)")
    T, H, D = value.shape
    nseq = cu.numel() - 1
    if nseq < 1 or tuple(hidden_init.shape) != (nseq, H, D, D):
        raise ValueError("chunk_gla_packed: cu_seqlens must have nseq + 1 entries for hidden_init (nseq, H, D, D)")
    if key.shape != value.shape or query.shape != value.shape or log_fgate.shape != value.shape:
        raise ValueError("chunk_gla_packed: log_fgate, value, key, query must all be (T, H, D)")
    if not value.is_cuda:
        raise TypeError("chunk_gla_packed: CUDA tensors required (there is no CPU path)")
    if not cu.is_cuda and (int(cu[0]) != 0 or int(cu[-1]) != T or bool(((cu[1:] - cu[:-1]) <= 0).any())):
        raise ValueError("chunk_gla_packed: cu_seqlens must rise from 0 to T")
    _stream(value.device)
    if int(chunk_size) % 128 or int(chunk_size) <= 0 or int(chunk_size) & (int(chunk_size) - 1):
        raise _lib.GlaError(f"chunk_gla_packed: unsupported configuration T={T} H={H} D={D} chunk={chunk_size} dtype={value.dtype}")
    raise TypeError("chunk_gla_packed: bfloat16 arrays, all on one device, are required")


def decode_step(state, log_fgate, value, key, query, out_dtype=None):
    """One token of the recurrence (reference: the loop body of gla.py:26-47) for a batch of requests.

    ``state`` (B, H, D, D) float32 CUDA tensor is updated IN PLACE
    (``S <- exp(log_fgate)[..., None] * S + key[..., None] * value[..., None, :]``); returns
    ``out = query @ S`` of shape (B, H, D) in ``out_dtype`` (default: value's dtype).  ``log_fgate``,
    ``value``, ``key``, ``query`` are (B, H, D).  T calls equal one ``recurrent_gla`` over T tokens
    (``hidden_init`` -> ``hidden_final`` chaining, gla.py:720-723).  Not differentiable (serving path)."""
    out = _lib.native().decode_step(state, log_fgate, value, key, query, out_dtype)
    if out is not None:
        return out
    if state.dtype != torch.float32 or not state.is_contiguous() or state.dim() != 4:
        raise TypeError("decode_step: state must be a contiguous float32 (B, H, D, D) tensor")
    B, H, D, D2 = state.shape
    if D != D2 or tuple(value.shape) != (B, H, D) or key.shape != value.shape or query.shape != value.shape \
            or log_fgate.shape != value.shape:
        raise ValueError("decode_step: expected state (B, H, D, D) and log_fgate, value, key, query (B, H, D)")
    if key.dtype != value.dtype or query.dtype != value.dtype or value.dtype not in _DT or (out_dtype or value.dtype) not in _DT:
        raise TypeError("decode_step: value, key, query must share a dtype, float32 or bfloat16")
    _stream(value.device)
    raise RuntimeError("decode_step needs CUDA tensors on one device; there is no CPU fallback")


def auto_block_size(value_dim: int, key_dim: int, num_heads: int, max_block_size: int):
    """Reference helper (gla.py:390-403) kept for callers that import it: the Triton block
    sizes it would have chosen.  The CUDA kernels do not use them."""
    assert value_dim == key_dim, "Not supported yet"
    vb = min(max_block_size, value_dim)
    kb = min(max_block_size, key_dim)
    hb = None
    for c in sorted(c for c in range(1, num_heads + 1) if num_heads % c == 0):
        if c * vb <= max_block_size and c * kb <= max_block_size:
            hb = c
        else:
            break
    assert hb is not None
    return vb, kb, hb
