"""Paged-KV scatter on a hand-written CUDA kernel, and the attention call.

`store_kvcache` has the signature and preconditions of
nanovllm/layers/attention.py:33-40 (the Triton kernel at :10-30 is replaced by
b2_store_kvcache: 16-byte vector copies, several tokens per CTA, bit-exact).
`Attention` keeps the reference's interface (:43-75).  Decode attention runs on
b2_paged_attention_decode and prefill attention on b2_prefill_attention; the
shapes they do not serve stay a library call, as in the reference: flash-attn's
paged and varlen kernels.  So do batches of wide groups for which that library
is the better one (decode_is_cut, prefill_is_short).
"""
from __future__ import annotations

import functools

import torch
from torch import nn

from .. import ops
from ..utils.context import get_context

try:  # the attention library is outside this path; it is only called, never re-implemented
    from flash_attn import flash_attn_varlen_func, flash_attn_with_kvcache
except Exception:  # pragma: no cover
    flash_attn_varlen_func = flash_attn_with_kvcache = None


def store_kvcache(key: torch.Tensor, value: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, slot_mapping: torch.Tensor):
    ops.store_kvcache(key, value, k_cache, v_cache, slot_mapping)


def _sdpa_paged(q, k_cache, v_cache, context_lens, block_tables, scale, q_lens=None):
    """Plain-PyTorch attention over the paged cache: a slow stand-in for the
    library call, used for small shapes when flash-attn cannot run."""
    nh, hd = q.shape[-2], q.shape[-1]
    nkv = k_cache.shape[-2]
    bs = k_cache.shape[1]
    outs = []
    off = 0
    lens = context_lens.tolist()
    for i, n_ctx in enumerate(lens):
        tq = 1 if q_lens is None else q_lens[i]
        if n_ctx == 0:
            outs.append(torch.zeros(tq, nh, hd, dtype=q.dtype, device=q.device))
            off += tq
            continue
        nblk = (n_ctx + bs - 1) // bs
        blocks = block_tables[i, :nblk].long()
        k = k_cache[blocks].reshape(-1, nkv, hd)[:n_ctx]
        v = v_cache[blocks].reshape(-1, nkv, hd)[:n_ctx]
        qi = q[off:off + tq]
        mask = None
        if tq > 1:
            qpos = torch.arange(tq, device=q.device).unsqueeze(1) + (n_ctx - tq)
            mask = torch.arange(n_ctx, device=q.device).unsqueeze(0) <= qpos
        o = torch.nn.functional.scaled_dot_product_attention(qi.transpose(0, 1).unsqueeze(0), k.transpose(0, 1).unsqueeze(0),
                                                             v.transpose(0, 1).unsqueeze(0), attn_mask=mask, scale=scale, enable_gqa=True)
        outs.append(o.squeeze(0).transpose(0, 1))
        off += tq
    return torch.cat(outs)


@functools.lru_cache(maxsize=None)
def _sms(device: int) -> int:
    return torch.cuda.get_device_properties(device).multi_processor_count if device >= 0 else 0


def decode_is_cut(n_seqs: int, nq: int, nkv: int, block_size: int, sms: int) -> bool:
    """True for decode batches of three and more query heads per KV head that are the library's: below 0.8 of two (sequence, KV head) pairs
    per SM it cuts contexts into parts, each rounded for itself and walked beside the others, where the own kernel walks a context in one
    CTA.  Its results are nearer to float64 there (32 / 8 heads, error x 1e3: 20 contexts of 4000 tokens 2.220 and 2.271, of 100..3000 2.197
    and 2.205, 28 of 4000 2.213 and 2.260), and one long context does not hold up the batch (19 of 100 tokens and one of 4000 35 and 46 us, of 16000
    100 and 171), although batches of about equal contexts take longer (20 of 300 tokens 21.3 and 7.7 us, of 4000 83 and 60).  From that line on
    the results are the same and the own kernel was the faster one in all that was tried (30 contexts of 300 tokens 20 and 9 us, 29 of 100
    and one of 32000 552 and 359).  The library wants cache blocks of a multiple of 256 tokens."""
    return nq > 2 * nkv and 5 * n_seqs * nkv < 8 * sms and block_size % 256 == 0


def prefill_is_short(tokens: int, n_seqs: int, max_q: int, nq: int, nkv: int, block_size: int, sms: int) -> bool:
    """True for prefill batches over the cache of three and more query heads per KV head that are the library's.  One new token per sequence: it
    cuts the keys there (32 / 8 heads, 1 x 1 token over 768 cached 11 and 22 us, over 8000 23 and 166, 16 x 1 over 768 29 and 45).  Or few rows: the
    time is one CTA's walk over the keys, which is the library's shorter one by a fifth (16 tokens over 8000 139 and 171 us, 200 over 8000 143 and
    178, 4 x 64 over 512 0.88 of the own time) as long as its tiles of 64 rows of each head all run at once; past that the own kernel
    was 1.05 to 2.4 times as fast (300 tokens over 512 1.17, 4 x 100 over 512 1.15)."""
    tiles = min(n_seqs * -(-max_q // 64), tokens // 64 + n_seqs)  # at most so many
    return nq > 2 * nkv and block_size % 256 == 0 and (max_q <= 1 or nq * tiles <= sms)


class Attention(nn.Module):
    # "flash_attn" (own kernels, the reference's library call for what they do not serve) or "sdpa" (plain PyTorch, for tests on small
    # shapes when flash-attn cannot run)
    backend = "flash_attn"

    def __init__(self, num_heads, head_dim, scale, num_kv_heads):
        super().__init__()
        self.num_heads, self.head_dim, self.scale, self.num_kv_heads = num_heads, head_dim, scale, num_kv_heads
        self.k_cache = self.v_cache = torch.tensor([])

    def attend(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> torch.Tensor:
        """Attention over K/V that are already in the paged cache (decode, or
        prefill with a cached prefix) or passed in (plain prefill)."""
        ctx = get_context()
        k_cache, v_cache = self.k_cache, self.v_cache
        if Attention.backend == "sdpa":
            if ctx.is_prefill:
                cu_q, cu_k = ctx.cu_seqlens_q.tolist(), ctx.cu_seqlens_k.tolist()
                q_lens = [b - a for a, b in zip(cu_q[:-1], cu_q[1:])]
                k_lens = torch.tensor([b - a for a, b in zip(cu_k[:-1], cu_k[1:])])
                if ctx.block_tables is None:  # no cache bound (warm-up) or no prefix: attend over the passed K/V
                    outs = []
                    for i, (a, b) in enumerate(zip(cu_q[:-1], cu_q[1:])):
                        o = torch.nn.functional.scaled_dot_product_attention(
                            q[a:b].transpose(0, 1).unsqueeze(0), k[a:b].transpose(0, 1).unsqueeze(0), v[a:b].transpose(0, 1).unsqueeze(0),
                            is_causal=True, scale=self.scale, enable_gqa=True)
                        outs.append(o.squeeze(0).transpose(0, 1))
                    return torch.cat(outs)
                return _sdpa_paged(q, k_cache, v_cache, k_lens, ctx.block_tables, self.scale, q_lens)
            return _sdpa_paged(q, k_cache, v_cache, ctx.context_lens, ctx.block_tables, self.scale)
        n, nq, nkv = q.shape[0], self.num_heads, self.num_kv_heads
        sms, o = _sms(q.get_device()) if nq > 2 * nkv else 0, None  # (0: not a wide group, or tensors that the kernels refuse)
        if ctx.is_prefill:
            cached = ctx.block_tables is not None  # prefix cache / chunked prefill: read K/V from the cache
            if not (cached and sms and flash_attn_varlen_func is not None and
                    prefill_is_short(n, ctx.cu_seqlens_q.numel() - 1, ctx.max_seqlen_q, nq, nkv, k_cache.shape[1], sms)):
                o = ops.prefill_attention(q, k_cache if cached else k, v_cache if cached else v, ctx.cu_seqlens_q, ctx.cu_seqlens_k, ctx.max_seqlen_q,
                                          ctx.block_tables, self.scale)
        elif not (sms and flash_attn_with_kvcache is not None and decode_is_cut(n, nq, nkv, k_cache.shape[1], sms)):
            o = ops.paged_attention(q, k_cache, v_cache, ctx.context_lens, ctx.block_tables, self.scale)
        if o is not None:
            return o
        if flash_attn_varlen_func is None:
            raise RuntimeError("flash-attn is not importable; set Attention.backend = 'sdpa' for small test shapes")
        if ctx.is_prefill:
            if ctx.block_tables is not None:  # prefix cache / chunked prefill: read K/V from the cache
                k, v = k_cache, v_cache
            return flash_attn_varlen_func(q, k, v, max_seqlen_q=ctx.max_seqlen_q, cu_seqlens_q=ctx.cu_seqlens_q,
                                          max_seqlen_k=ctx.max_seqlen_k, cu_seqlens_k=ctx.cu_seqlens_k,
                                          softmax_scale=self.scale, causal=True, block_table=ctx.block_tables)
        return flash_attn_with_kvcache(q.unsqueeze(1), k_cache, v_cache, cache_seqlens=ctx.context_lens,
                                       block_table=ctx.block_tables, softmax_scale=self.scale, causal=True).squeeze(1)

    def forward(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> torch.Tensor:
        """Reference behaviour: scatter this step's K/V into the cache (when one is bound), then attend."""
        if self.k_cache.numel() and self.v_cache.numel():
            store_kvcache(k, v, self.k_cache, self.v_cache, get_context().slot_mapping)
        return self.attend(q, k, v)
