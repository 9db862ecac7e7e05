"""Tensor-level wrappers over the C ABI: they check dtypes and layouts, pick
the current CUDA stream, allocate outputs with torch and pass raw pointers.
The calls of a decoder layer do that in native code (csrc/b2_torch.cpp)."""
from __future__ import annotations

import ctypes as C

import torch

from . import _abi
from .runtime import get_runtime

_lib = _abi.lib
_native = _abi.native


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _bf16_rows(t: torch.Tensor, what: str) -> torch.Tensor:
    if t.dtype != torch.bfloat16 or not t.is_cuda:
        raise TypeError(f"{what}: expected a CUDA bf16 tensor, got {t.dtype} on {t.device}")
    if t.stride(-1) != 1:
        t = t.contiguous()
    return t


def _as2d(t: torch.Tensor) -> torch.Tensor:
    if t.dim() == 2:
        return t
    return t.reshape(-1, t.shape[-1])


def gemm(x: torch.Tensor, w: torch.Tensor, bias: torch.Tensor | None = None) -> torch.Tensor:
    """x[..., K] @ w[N, K]^T (+ bias)."""
    return _native.gemm(get_runtime().handle, x, w, bias)


def qkv_fused(x: torch.Tensor, w: torch.Tensor, bias, nq: int, nkv: int, head_dim: int, q_norm_w, k_norm_w, eps: float,
              positions: torch.Tensor, cos_sin: torch.Tensor, k_cache, v_cache, slot_mapping) -> torch.Tensor:
    """qkv projection + q/k head norm + RoPE + KV scatter; returns the [M, (nq + 2 nkv) head_dim] tensor with q and k
    already normalised and rotated."""
    return _native.qkv_fused(get_runtime().handle, x, w, bias, nq, nkv, head_dim, q_norm_w, k_norm_w, eps, positions, cos_sin,
                             k_cache, v_cache, slot_mapping)


def gemm_silu_mul(x: torch.Tensor, w_pairs: torch.Tensor) -> torch.Tensor:
    """silu(x @ gate^T) * (x @ up^T) where w_pairs interleaves gate and up rows (gate_0, up_0, gate_1, ...)."""
    return _native.gemm_silu_mul(get_runtime().handle, x, w_pairs)


def rowpar_form(M: int, N: int) -> int:
    """Which form of the fused row-parallel block serves M tokens of N features on this runtime
    (_abi.FORM_ONESHOT / FORM_OWNER: b2_rowpar_fused; FORM_TWOSHOT: b2_rowpar_fused_twoshot).  The library decides."""
    form = _lib.b2_rowpar_form(get_runtime().ctx, M, N)
    if form < 0:
        raise _abi.B2Error(f"b2_rowpar_form({M}, {N}): bad argument")
    return form


def rowpar_fused(x: torch.Tensor, w: torch.Tensor, bias: torch.Tensor | None, residual: torch.Tensor | None,
                 norm_w: torch.Tensor | None, eps: float):
    """Row-parallel GEMM + all-reduce (+ residual add + RMSNorm when norm_w is given).
    Returns y, or (normed, new_residual).

    For many tokens at tensor-parallel size >= 2 (rowpar_form(M, N) == FORM_TWOSHOT) the two-shot kernel runs:
    `normed` is then a view of a buffer owned by the runtime (valid until the next such call) and `new_residual`
    holds only the rows this rank owns (16-row blocks rank, rank + world, ...); the next fused call reads exactly
    those rows."""
    out = _native.rowpar_fused(get_runtime().handle, x, w, bias, residual, norm_w, eps)
    return _rowpar_twoshot(x, w, bias, residual, norm_w, eps) if out is None else out


def _rowpar_twoshot(x, w, bias, residual, norm_w, eps):
    rt = get_runtime()
    x2 = _as2d(_bf16_rows(x, "row-parallel input"))
    if x2.stride(0) % 8 != 0 or x2.data_ptr() % 16 != 0:
        x2 = x2.contiguous()
    M, Kr = x2.shape
    N = w.shape[0]
    res_out = None
    if norm_w is not None:
        residual = _bf16_rows(residual, "residual").contiguous()
        res_out = torch.empty_like(residual)
    ptr = C.c_void_p()
    _abi.check(_lib.b2_rowpar_fused_twoshot(rt.ctx, x2.data_ptr(), x2.stride(0), w.data_ptr(), w.stride(0),
                                            bias.data_ptr() if bias is not None else None, M, N, Kr,
                                            residual.data_ptr() if norm_w is not None else None, norm_w.data_ptr() if norm_w is not None else None,
                                            float(eps), C.byref(ptr), res_out.data_ptr() if res_out is not None else None, _stream()),
               "b2_rowpar_fused_twoshot")
    out = _library_view(ptr.value, (M, N), x.device)
    if norm_w is None:
        return out.clone().view(*x.shape[:-1], N)  # a plain forward hands out memory the caller may keep
    return out, res_out


def rmsnorm(x: torch.Tensor, w: torch.Tensor, eps: float) -> torch.Tensor:
    return _native.rmsnorm(x, w, eps)


def add_rmsnorm(x: torch.Tensor, residual: torch.Tensor, w: torch.Tensor, eps: float):
    return _native.add_rmsnorm(x, residual, w, eps)


def store_kvcache(key: torch.Tensor, value: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, slot_mapping: torch.Tensor) -> None:
    _native.store_kvcache(key, value, k_cache, v_cache, slot_mapping)


def silu_and_mul(x: torch.Tensor) -> torch.Tensor:
    return _native.silu_and_mul(x)


def qk_norm_rope_store(qkv: torch.Tensor, nq: int, nkv: int, head_dim: int, q_norm_w, k_norm_w, eps: float,
                       positions: torch.Tensor, cos_sin: torch.Tensor, k_cache, v_cache, slot_mapping) -> None:
    _native.qk_norm_rope_store(qkv, nq, nkv, head_dim, q_norm_w, k_norm_w, eps, positions, cos_sin, k_cache, v_cache, slot_mapping)


def rope(positions: torch.Tensor, q: torch.Tensor, k: torch.Tensor, cos_sin: torch.Tensor, head_dim: int) -> tuple[torch.Tensor, torch.Tensor]:
    """Rotated copies of q [tokens, heads, head_dim] and k (or flattened over the heads)."""
    return _native.rope(positions, q, k, cos_sin, head_dim)


def embed(ids: torch.Tensor, w: torch.Tensor, vocab_start: int, vocab_end: int, world: int) -> torch.Tensor:
    return _native.embed(get_runtime().handle if world > 1 else None, ids, w, vocab_start, vocab_end)


def paged_attention(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, context_lens: torch.Tensor, block_tables: torch.Tensor,
                    scale: float) -> torch.Tensor | None:
    """Decode attention: one query token per sequence, q [n, nq, head_dim], over the paged cache.  None when the
    kernel does not serve the call (head_dim other than 128, more than 2 query heads per KV head in a small batch, a layout it cannot address);
    operands that do not fit each other, or are not on one GPU, raise."""
    return _native.paged_attention(get_runtime().handle, q, k_cache, v_cache, context_lens, block_tables, scale)


def prefill_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, cu_seqlens_q: torch.Tensor, cu_seqlens_k: torch.Tensor, max_seqlen_q: int,
                      block_tables: torch.Tensor | None, scale: float) -> torch.Tensor | None:
    """Causal attention of q [tokens, nq, head_dim] over k, v [tokens, nkv, head_dim], or over the paged caches when
    block_tables is given.  None when the kernel does not serve the call (it takes head_dim 128, an even number of
    query heads per KV head, forward only); operands that do not fit each other, or are not on one GPU, raise."""
    return _native.prefill_attention(get_runtime().handle, q, k, v, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, block_tables, scale)


def decode_stack_served(rows: int, layers: int, hidden: int, nq: int, nkv: int, head_dim: int, inter: int, block_size: int) -> bool:
    """Whether decode_stack serves a step of this shape on this runtime (see b2_decode_stack_workspace)."""
    return _lib.b2_decode_stack_workspace(get_runtime().ctx, rows, layers, hidden, nq, nkv, head_dim, inter, block_size) > 0


def decode_stack(x: torch.Tensor, positions: torch.Tensor, layers: list[tuple], final_norm: torch.Tensor, nq: int, nkv: int, head_dim: int, inter: int,
                 eps: float, qk_eps: float, scale: float, cos_sin: torch.Tensor, context_lens: torch.Tensor, slot_mapping: torch.Tensor,
                 block_tables: torch.Tensor) -> torch.Tensor | None:
    """All decoder layers of a decode step in one launch: x [rows, hidden] the embedded tokens, layers a list of (qkv_w, o_w,
    gate_up_w with paired rows, down_w, in_norm, post_norm, q_norm, k_norm, k_cache, v_cache).  Returns the final norm's output.
    None when the kernel does not serve the call (a shape that decode_stack_served declines, no layers, a layout it cannot
    address); rows after the last one with a context come back as zeros."""
    return _native.decode_stack(get_runtime().handle, x, positions, layers, final_norm, nq, nkv, head_dim, inter, eps, qk_eps, scale, cos_sin,
                                context_lens, slot_mapping, block_tables)


class _DevicePtr:
    """Minimal __cuda_array_interface__ carrier so torch can view library-owned memory."""

    def __init__(self, ptr: int, shape: tuple[int, ...]):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<u2", "data": (ptr, False), "version": 3, "strides": None}


_LOGIT_VIEWS: dict = {}


def _library_view(ptr: int, shape: tuple[int, int], device) -> torch.Tensor:
    """bf16 tensor over memory the library owns; built once per (address, shape), outside any graph capture."""
    key = (ptr, *shape)
    view = _LOGIT_VIEWS.get(key)
    if view is None:
        view = torch.as_tensor(_DevicePtr(ptr, shape), device=device).view(torch.bfloat16)
        _LOGIT_VIEWS[key] = view
    return view


def lm_head(h: torch.Tensor, w: torch.Tensor, row_index: torch.Tensor | None):
    """Returns the gathered [B, vocab] logits on rank 0 (a view of the runtime's
    buffer, valid until the next call) and None elsewhere."""
    rt = get_runtime()
    h2 = _as2d(_bf16_rows(h, "lm_head input"))
    if h2.stride(0) % 8 != 0 or h2.data_ptr() % 16 != 0:
        h2 = h2.contiguous()
    B = h2.shape[0] if row_index is None else row_index.numel()
    if row_index is not None:
        assert row_index.dtype == torch.int32 and row_index.is_cuda
    Vr, H = w.shape
    out = C.c_void_p()
    _abi.check(_lib.b2_lm_head(rt.ctx, h2.data_ptr(), h2.stride(0), row_index.data_ptr() if row_index is not None else None,
                               w.data_ptr(), w.stride(0), B, Vr, H, C.byref(out), _stream()), "b2_lm_head")
    if rt.rank != 0:
        return None
    vocab = Vr * rt.world
    key = (out.value, B, vocab)
    view = _LOGIT_VIEWS.get(key)
    if view is None:  # built once per shape (outside any graph capture: the first call of a shape is a warm-up)
        view = torch.as_tensor(_DevicePtr(out.value, (B, vocab)), device=h.device).view(torch.bfloat16)
        _LOGIT_VIEWS[key] = view
    return view


def lm_head_sample(h: torch.Tensor, w: torch.Tensor, row_index: torch.Tensor | None, temperatures: torch.Tensor | None,
                   seed: int, out: torch.Tensor | None = None) -> torch.Tensor:
    """LM head and sampler in one pass over the vocabulary shard (no logits in memory).  Returns int64 token ids
    [B], valid on rank 0 only.  temperatures: fp32 [B] on the device, or None for greedy decoding."""
    rt = get_runtime()
    h2 = _as2d(_bf16_rows(h, "lm_head input"))
    if h2.stride(0) % 8 != 0 or h2.data_ptr() % 16 != 0:
        h2 = h2.contiguous()
    B = h2.shape[0] if row_index is None else row_index.numel()
    if row_index is not None:
        assert row_index.dtype == torch.int32 and row_index.is_cuda
    if temperatures is not None:
        assert temperatures.dtype == torch.float32 and temperatures.is_cuda and temperatures.is_contiguous() and temperatures.numel() >= B
    if out is None:
        out = torch.empty(B, dtype=torch.int64, device=h.device)
    assert out.dtype == torch.int64 and out.is_cuda and out.numel() >= B
    Vr, H = w.shape
    _abi.check(_lib.b2_lm_head_sample(rt.ctx, h2.data_ptr(), h2.stride(0), row_index.data_ptr() if row_index is not None else None,
                                      w.data_ptr(), w.stride(0), B, Vr, H, temperatures.data_ptr() if temperatures is not None else None,
                                      int(seed) & 0xFFFFFFFFFFFFFFFF, out.data_ptr(), _stream()), "b2_lm_head_sample")
    return out[:B]


def argmax(logits: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    assert logits.dim() == 2 and logits.dtype == torch.bfloat16 and logits.stride(1) == 1
    if out is None:
        out = torch.empty(logits.shape[0], dtype=torch.int64, device=logits.device)
    assert out.dtype == torch.int64 and out.numel() >= logits.shape[0]
    _abi.check(_lib.b2_argmax(logits.data_ptr(), logits.stride(0), logits.shape[0], logits.shape[1], out.data_ptr(), _stream()), "b2_argmax")
    return out


def broadcast_tokens(buf: torch.Tensor) -> torch.Tensor:
    """Rank 0's int64 token ids into `buf` on every rank (in place)."""
    assert buf.dtype == torch.int64 and buf.is_cuda and buf.is_contiguous()
    _abi.check(_lib.b2_broadcast_tokens(get_runtime().ctx, buf.data_ptr(), buf.numel(), _stream()), "b2_broadcast_tokens")
    return buf


def advance_decode(tokens, input_ids, positions, context_lens, slot_mapping, block_tables, block_size: int, num_slots: int) -> None:
    """Device-side equivalent of building the next decode step's inputs.  num_slots = slots of the KV cache
    (blocks * block_size): a row whose next position has no block, or whose slot would lie outside the cache, is
    frozen (slot -1, position and length unchanged) instead of being sent outside the cache."""
    n = tokens.numel()
    assert tokens.dtype == torch.int64 and positions.dtype == torch.int64 and block_tables.dtype == torch.int32
    assert block_tables.dim() == 2 and block_tables.stride(1) == 1 and block_tables.shape[0] >= n
    _abi.check(_lib.b2_advance_decode(tokens.data_ptr(), input_ids.data_ptr(), positions.data_ptr(), context_lens.data_ptr(),
                                      slot_mapping.data_ptr(), block_tables.data_ptr(), block_tables.stride(0), block_tables.shape[1],
                                      block_size, num_slots, n, _stream()), "b2_advance_decode")
