"""Run one kernel of the library a few times on one GPU, for profiling with
Nsight Compute (the cases are larger than the 126 MB L2 but hold well under a
few GB, so a `--set full` capture of 1-3 launches ends by itself).

    python tests/profile_case.py <case> [--launches 6]

cases:
  gemm_decode     column-parallel GEMM, M=64, N=24576, K=4096 (Qwen3-8B gate_up at TP=1), 4 weight copies
  silu_decode     the same GEMM with SiLU*mul in its epilogue (what the decoder layer launches)
  qkv_decode      qkv projection M=64, N=6144, K=4096 with q/k-norm + RoPE + KV scatter in its epilogue, 8 weight copies
  oproj_decode    fused row-parallel launch, M=64, N=4096, Kr=4096 (Qwen3-8B o_proj at TP=1), 8 weight copies
  gemm_prefill    GEMM M=4096, N=4096, K=4096
  gemm_mid        GEMM M=256, N=4096, K=1024 (Qwen3-0.6B qkv at a 256-sequence decode step), 40 weight copies
  qkv_prefill     qkv projection M=2048, N=4096, K=1024 with the head work in its epilogue (Qwen3-0.6B prefill), 24 weight copies
  silu_mid        gate/up + SiLU*mul, M=256, N=24576, K=4096, 2 weight copies
  attn_decode     decode attention, 64 contexts of 300..1371 tokens, 16 query / 8 KV heads, paged cache in shuffled blocks
  attn_decode_few the same with the first 24 of them
  attn_decode_wide the 64 contexts with 32 query heads
  attn_prefill    causal prefill attention, 8 sequences of 2048 tokens, 16 query / 8 KV heads
  attn_prefill_cached 8 sequences of 1024 tokens over 512 cached ones, 32 query / 8 KV heads, paged cache in shuffled blocks
  rowpar_decode   fused row-parallel launch, M=64, N=4096, Kr=12288 (Qwen3-8B down_proj at TP=1)
  rowpar_prefill  fused row-parallel launch, M=1024, N=5120, Kr=1024
  store_kvcache   paged-KV scatter, 16384 tokens x D=1024
  add_rmsnorm     residual add + RMSNorm, 16384 x 4096
  embed           embedding lookup, 16384 ids into a [151936, 4096] table (one rank)
  decode_stack    all 28 layers of a Qwen3-0.6B decode step in one launch, one sequence of 300 tokens (0.9 GB of weights)
  decode_stack_16 the same with 16 sequences of 300 tokens
  sampler         LM head fused with the sampler, 256 rows x 151936 x 1024 with temperatures
"""
from __future__ import annotations

import argparse
import os
import sys

import torch
import torch.distributed as dist

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("case")
    ap.add_argument("--launches", type=int, default=6)
    a = ap.parse_args()
    import __graft_entry__ as entry
    entry.load_package()
    from nanovllm_b200 import ops
    from nanovllm_b200.runtime import init_runtime, shutdown_runtime
    os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
    os.environ.setdefault("MASTER_PORT", "29579")
    torch.cuda.set_device(0)
    dist.init_process_group("gloo", rank=0, world_size=1)
    init_runtime(max_tokens=16384, hidden=5120, oneshot_tokens=1024, vocab=151936 if a.case == "sampler" else 0, max_seqs=256 if a.case == "sampler" else 0)
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(0)

    def rnd(*shape, scale=1.0):
        return (torch.randn(*shape, device=dev, generator=g) * scale).bfloat16()

    if a.case in ("gemm_decode", "gemm_prefill", "gemm_mid"):
        m, n, k, copies = {"gemm_decode": (64, 24576, 4096, 4), "gemm_prefill": (4096, 4096, 4096, 2), "gemm_mid": (256, 4096, 1024, 40)}[a.case]
        x, ws = rnd(m, k), [rnd(n, k, scale=0.02) for _ in range(copies)]
        call = lambda i: ops.gemm(x, ws[i % copies])
    elif a.case in ("silu_decode", "silu_mid"):
        m, i, k, copies = {"silu_decode": (64, 12288, 4096, 4), "silu_mid": (256, 12288, 4096, 2)}[a.case]
        x, ws = rnd(m, k), [rnd(2 * i, k, scale=0.02) for _ in range(copies)]
        call = lambda j: ops.gemm_silu_mul(x, ws[j % copies])
    elif a.case in ("qkv_decode", "qkv_prefill"):
        m, nq, nkv, k, copies = {"qkv_decode": (64, 32, 8, 4096, 8), "qkv_prefill": (2048, 16, 8, 1024, 24)}[a.case]
        x, ws = rnd(m, k), [rnd((nq + 2 * nkv) * 128, k, scale=0.02) for _ in range(copies)]
        qw, kw = rnd(128), rnd(128)
        pos = torch.randint(0, 2048, (m,), device=dev)
        t = torch.arange(2048, dtype=torch.float, device=dev)
        inv = 1.0 / (1e6 ** (torch.arange(0, 128, 2, dtype=torch.float, device=dev) / 128))
        fr = torch.outer(t, inv)
        cos_sin = torch.cat((fr.cos(), fr.sin()), dim=-1).contiguous()
        kc = torch.zeros(16, 256, nkv, 128, dtype=torch.bfloat16, device=dev)
        vc = torch.zeros_like(kc)
        slots = torch.randperm(16 * 256, device=dev)[:m].to(torch.int32)
        call = lambda j: ops.qkv_fused(x, ws[j % copies], None, nq, nkv, 128, qw, kw, 1e-6, pos, cos_sin, kc, vc, slots)
    elif a.case.startswith("attn_decode"):
        lens = [300 + 17 * i for i in range(24 if a.case == "attn_decode_few" else 64)]
        need = [-(-n // 256) for n in lens]
        order = torch.randperm(sum(need), device=dev, generator=g).to(torch.int32)
        tables = torch.zeros(len(lens), max(need), dtype=torch.int32, device=dev)
        for i, n in enumerate(need):
            tables[i, :n] = order[sum(need[:i]):sum(need[:i]) + n]
        kc, vc, q = rnd(sum(need), 256, 8, 128), rnd(sum(need), 256, 8, 128), rnd(len(lens), 32 if a.case == "attn_decode_wide" else 16, 128)
        context_lens = torch.tensor(lens, dtype=torch.int32, device=dev)
        call = lambda i: ops.paged_attention(q, kc, vc, context_lens, tables, 128 ** -0.5)
    elif a.case == "attn_prefill":
        q, k, v = rnd(16384, 16, 128), rnd(16384, 8, 128), rnd(16384, 8, 128)
        cu = torch.arange(0, 16385, 2048, dtype=torch.int32, device=dev)
        call = lambda i: ops.prefill_attention(q, k, v, cu, cu, 2048, None, 128 ** -0.5)
    elif a.case == "attn_prefill_cached":
        q, kc, vc = rnd(8192, 32, 128), rnd(48, 256, 8, 128), rnd(48, 256, 8, 128)
        cu, cu_k = (torch.arange(0, 8 * n + 1, n, dtype=torch.int32, device=dev) for n in (1024, 1536))
        tables = torch.randperm(48, device=dev, generator=g).to(torch.int32).view(8, 6)
        call = lambda i: ops.prefill_attention(q, kc, vc, cu, cu_k, 1024, tables, 128 ** -0.5)
    elif a.case in ("rowpar_decode", "rowpar_prefill", "oproj_decode"):
        m, n, k, copies = {"rowpar_decode": (64, 4096, 12288, 4), "rowpar_prefill": (1024, 5120, 1024, 8), "oproj_decode": (64, 4096, 4096, 8)}[a.case]
        x, ws, res, nw = rnd(m, k), [rnd(n, k, scale=0.02) for _ in range(copies)], rnd(m, n), rnd(n)
        call = lambda i: ops.rowpar_fused(x, ws[i % copies], None, res, nw, 1e-6)
    elif a.case == "store_kvcache":
        n, heads = 16384, 8
        key, value = rnd(n, heads, 128), rnd(n, heads, 128)
        kc = torch.zeros(2, 128, 256, heads, 128, dtype=torch.bfloat16, device=dev)
        vc = torch.zeros_like(kc)
        perm = torch.randperm(128, device=dev, generator=g)
        base = (perm[torch.arange(n, device=dev) // 256] * 256 + torch.arange(n, device=dev) % 256).to(torch.int32)
        call = lambda i: ops.store_kvcache(key, value, kc[i % 2], vc[i % 2], base)
    elif a.case == "add_rmsnorm":
        xs, rs, nw = [rnd(16384, 4096) for _ in range(2)], [rnd(16384, 4096) for _ in range(2)], rnd(4096)
        call = lambda i: ops.add_rmsnorm(xs[i % 2], rs[i % 2], nw, 1e-6)
    elif a.case == "embed":
        w = rnd(151936, 4096)
        ids = [torch.randint(0, 151936, (16384,), device=dev, generator=g) for _ in range(2)]
        call = lambda i: ops.embed(ids[i % 2], w, 0, 151936, 1)
    elif a.case in ("decode_stack", "decode_stack_16"):
        rows, context, nq, nkv, h, inter = 16 if a.case.endswith("16") else 1, 300, 16, 8, 1024, 3072
        blocks = -(-context // 256)

        def layer():
            kv = [rnd(rows * blocks, 256, nkv, 128) for _ in range(2)]
            return (rnd((nq + 2 * nkv) * 128, h, scale=0.02), rnd(h, nq * 128, scale=0.02), rnd(2 * inter, h, scale=0.02), rnd(h, inter, scale=0.02), rnd(h), rnd(h),
                    rnd(128), rnd(128), *kv)

        layers, x, norm = [layer() for _ in range(28)], rnd(rows, h), rnd(h)
        cos_sin = torch.randn(context, 128, device=dev, generator=g)
        ints = lambda values: torch.tensor(values, dtype=torch.int32, device=dev)
        tables, lens = ints([[i * blocks + j for j in range(blocks)] for i in range(rows)]), ints([context] * rows)
        slots, pos = ints([(i * blocks + blocks - 1) * 256 + (context - 1) % 256 for i in range(rows)]), torch.full((rows,), context - 1, device=dev)

        def call(i):
            assert ops.decode_stack(x, pos, layers, norm, nq, nkv, 128, inter, 1e-6, 1e-6, 128 ** -0.5, cos_sin, lens, slots, tables) is not None
    elif a.case == "sampler":
        x, w, temps = rnd(256, 1024), rnd(151936, 1024, scale=0.02), torch.full((256,), 0.6, device=dev)
        call = lambda i: ops.lm_head_sample(x, w, None, temps, 5)
    else:
        raise SystemExit(f"unknown case {a.case}")
    with torch.inference_mode():
        for i in range(a.launches):
            call(i)
    torch.cuda.synchronize()
    shutdown_runtime()
    dist.destroy_process_group()
    print("done", a.case)


if __name__ == "__main__":
    main()
