"""The many-token GEMM (CTA pairs over tiles of up to 256 tokens) where its dispatch branches: tile edges, split K in a cluster,
ranges of K blocks over the grid, whole rounds; and its epilogues."""
import pytest
import torch

from oracle import tp_path as O
from tests.gpu_util import assert_close_bf16, ensure_group, ulp_mismatch_fraction

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def rt(pkg):
    ensure_group()
    from nanovllm_b200.runtime import init_runtime, shutdown_runtime
    r = init_runtime(max_tokens=4096, hidden=5120)
    yield r
    shutdown_runtime()


# one token past the decode kernels; edges of 32-, 64- and 256-token tiles; features that end inside a CTA's half; few K blocks; a
# split over 2..4 pairs; ranges of K blocks (long K, tiles that do not fill the pairs); whole tiles, two CTAs per SM; whole rounds with
# a remainder
SHAPES = [(65, 256, 64), (96, 128, 128), (97, 1032, 520), (128, 1024, 2048), (160, 4096, 4096), (255, 136, 1024), (256, 4096, 4096), (257, 512, 1024),
          (391, 5120, 25600), (511, 6144, 4096), (512, 4096, 520), (777, 5120, 8192), (777, 6144, 4096), (1500, 24576, 512)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_against_fp32_and_repeatable(rt, m, n, k):
    from nanovllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x = torch.empty(m, k, device=DEV).normal_(generator=g).bfloat16()
    w = torch.empty(n, k, device=DEV).normal_(0, 0.02, generator=g).bfloat16()
    bias = torch.empty(n, device=DEV).normal_(generator=g).bfloat16()
    ys = [ops.gemm(x, w, bias) for _ in range(3)]  # the second launch finds the first one's workspace and counters
    torch.cuda.synchronize()
    rt.check_status()
    ref = x.double() @ w.double().t() + bias.double()
    for y in ys:
        assert_close_bf16(y, ref.float(), f"tile gemm {m}x{n}x{k}", abs_tol=2e-2 * max(1.0, (k / 4096) ** 0.5))
    if m >= 512:  # one unbroken sum over K
        assert torch.equal(ys[0], ys[2])


@pytest.mark.parametrize("m,bias", [(65, False), (150, True), (300, False), (1030, False)])
def test_qkv_epilogue_matches_the_head_kernel(rt, m, bias):
    """Head norm (or a projection bias instead), rotation and KV scatter in the epilogue against gemm + the head kernel."""
    from nanovllm_b200 import ops
    nq, nkv, hd, k = 16, 8, 128, 1024
    g = torch.Generator(device=DEV).manual_seed(m)
    x = torch.empty(m, k, device=DEV).normal_(generator=g).bfloat16()
    w = torch.empty((nq + 2 * nkv) * hd, k, device=DEV).normal_(0, 0.05, generator=g).bfloat16()
    b = torch.empty(w.shape[0], device=DEV).normal_(generator=g).bfloat16() if bias else None
    qw, kw = (None, None) if bias else ((torch.rand(hd, device=DEV, generator=g) + 0.5).bfloat16() for _ in range(2))
    pos = torch.randint(0, 2048, (m,), device=DEV, generator=g)
    table = O.rope_cache(hd, 2048, 1e6).to(DEV)
    slots = torch.randperm(m + 100, device=DEV, generator=g)[:m].to(torch.int32)
    slots[::7] = -1
    caches = [torch.zeros((m + 355) // 256, 256, nkv, hd, dtype=torch.bfloat16, device=DEV) for _ in range(4)]
    got = ops.qkv_fused(x, w, b, nq, nkv, hd, qw, kw, 1e-6, pos, table, caches[0], caches[1], slots)
    two = ops.gemm(x, w, b)
    ops.qk_norm_rope_store(two, nq, nkv, hd, qw, kw, 1e-6, pos, table, caches[2], caches[3], slots)
    torch.cuda.synchronize()
    rt.check_status()
    for a, c in ((got, two), (caches[0], caches[2]), (caches[1], caches[3])):
        assert ulp_mismatch_fraction(a, c, 1) < 1e-3


@pytest.mark.parametrize("m", [65, 200, 513, 2100])
def test_silu_epilogue(rt, m):
    from nanovllm_b200 import ops
    g = torch.Generator().manual_seed(m)
    x = torch.randn(m, 512, generator=g).bfloat16()
    w = (torch.randn(2 * 1544, 512, generator=g) * 0.1).bfloat16()
    got = ops.gemm_silu_mul(x.to(DEV), w.to(DEV))
    torch.cuda.synchronize()
    rt.check_status()
    ref = O.silu_and_mul(torch.cat([O.linear(x, w[0::2]), O.linear(x, w[1::2])], dim=-1))
    assert ulp_mismatch_fraction(got, ref, 2) < 2e-2


@pytest.mark.parametrize("m", [65, 300, 513])
def test_qkv_with_operands_off_the_16_byte_grid(rt, m):
    """Norm weights, rotary table and caches that no 16-byte vector can read: the heads are finished by the head kernel."""
    from nanovllm_b200 import ops
    nq, nkv, hd, k = 4, 2, 128, 512
    g = torch.Generator(device=DEV).manual_seed(m)
    x = torch.empty(m, k, device=DEV).normal_(generator=g).bfloat16()
    w = torch.empty((nq + 2 * nkv) * hd, k, device=DEV).normal_(0, 0.05, generator=g).bfloat16()
    pos = torch.randint(0, 512, (m,), device=DEV, generator=g)
    slots = torch.randperm(768, device=DEV, generator=g)[:m].to(torch.int32)
    tables = (O.rope_cache(hd, 512, 1e6).to(DEV), (torch.rand(2, hd, device=DEV, generator=g) + 0.5).bfloat16())
    outs = []
    for off in (0, 8):  # bytes

        def shifted(t):
            n = off // t.element_size()
            return torch.empty(t.numel() + 8, dtype=t.dtype, device=DEV)[n:n + t.numel()].view(t.shape).copy_(t)

        table, qw, kw = shifted(tables[0]), shifted(tables[1][0]), shifted(tables[1][1])
        kc, vc = (shifted(torch.zeros(3, 256, nkv, hd, dtype=torch.bfloat16, device=DEV)) for _ in range(2))
        outs.append((ops.qkv_fused(x, w, None, nq, nkv, hd, qw, kw, 1e-6, pos, table, kc, vc, slots), kc, vc))
    torch.cuda.synchronize()
    rt.check_status()
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("m", [513, 530, 565, 777, 1041])
def test_rows_are_the_same_whatever_the_width_of_the_tile(rt, m):
    """From 512 tokens on K is not cut, so a row's results are the same bits in a batch whose tiles are another number of columns wide
    (here 16 past a multiple of 32: 176, 144, 208; the whole batch 256 or 192), with each of the epilogues."""
    from nanovllm_b200 import ops
    nq, nkv, hd, k, full = 8, 4, 128, 512, 1536
    g = torch.Generator(device=DEV).manual_seed(m)
    x = torch.empty(full, k, device=DEV).normal_(generator=g).bfloat16()
    w = torch.empty((nq + 2 * nkv) * hd, k, device=DEV).normal_(0, 0.05, generator=g).bfloat16()
    qw, kw = ((torch.rand(hd, device=DEV, generator=g) + 0.5).bfloat16() for _ in range(2))
    pos = torch.randint(0, 2048, (full,), device=DEV, generator=g)
    table, slots = O.rope_cache(hd, 2048, 1e6).to(DEV), torch.arange(full, device=DEV, dtype=torch.int32)

    def run(n):
        kc, vc = (torch.zeros(full // 256, 256, nkv, hd, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        qkv = ops.qkv_fused(x[:n], w, None, nq, nkv, hd, qw, kw, 1e-6, pos[:n], table, kc, vc, slots[:n])
        return [ops.gemm(x[:n], w)[:m], ops.gemm_silu_mul(x[:n], w)[:m], qkv[:m]] + [c.view(full, -1)[:m] for c in (kc, vc)]

    part, whole = run(m), run(full)
    torch.cuda.synchronize()
    rt.check_status()
    for a, b in zip(part, whole):
        assert torch.equal(a, b)
