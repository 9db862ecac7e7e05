"""Decode attention over the paged cache against plain PyTorch attention in fp32."""
import pytest
import torch

from tests.gpu_util import assert_close_bf16, ensure_group

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def rt(pkg):
    ensure_group()
    from nanovllm_b200.runtime import init_runtime, shutdown_runtime
    r = init_runtime(max_tokens=1024, hidden=1024)
    yield r
    shutdown_runtime()


# tile edges (63, 64, 65; 16-row groups), block edges (255..257), padded rows (0), one context over many CTAs, a batch whose
# work ends inside a CTA's range, every group size
CASES = [((1,), 16, 8), ((63, 64, 65, 0, 15, 16, 17), 16, 8), ((255, 256, 257, 0), 16, 8), ((4096,), 2, 1), ((4000, 3), 8, 8), ((300,), 8, 8),
         (tuple(range(1, 620, 7)), 8, 4), ((700,) * 130, 2, 1)]


@pytest.mark.parametrize("lens,nq,nkv", CASES)
def test_paged_attention_against_fp32(rt, lens, nq, nkv):
    from nanovllm_b200 import ops
    g = torch.Generator().manual_seed(sum(lens) + nq)
    n, hd, bs, scale = len(lens), 128, 256, 128 ** -0.5
    need = [max(1, -(-x // bs)) for x in lens]
    free = torch.randperm(sum(need), generator=g).tolist()
    tables = torch.full((n, 16), -1, dtype=torch.int32)
    for i, k in enumerate(need):
        tables[i, :k] = torch.tensor([free.pop() for _ in range(k)], dtype=torch.int32)
    shape = (sum(need), bs, nkv, hd)
    kc, vc = torch.randn(shape, generator=g).bfloat16(), torch.randn(shape, generator=g).bfloat16()
    qkv = torch.randn(n, (nq + 2 * nkv) * hd, generator=g).bfloat16()
    ref = torch.zeros(n, nq, hd)
    for i, x in enumerate(lens):
        blocks = tables[i, :need[i]].long()
        k, v = (c[blocks].reshape(-1, nkv, hd)[:x].float().repeat_interleave(nq // nkv, 1) for c in (kc, vc))
        if x % bs:  # what lies past the context's end must not matter
            vc[blocks[-1], x % bs:] = float("nan")
        q = qkv[i, :nq * hd].float().view(nq, hd)
        p = torch.softmax(torch.einsum("hd,thd->ht", q, k) * scale, -1) if x else torch.zeros(nq, 0)
        ref[i] = torch.einsum("ht,thd->hd", p, v)
    q = qkv.to(DEV)[:, :nq * hd].view(n, nq, hd)
    args = (kc.to(DEV), vc.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), tables.to(DEV), scale)
    for _ in range(2):  # the second launch finds the first one's counters
        got = ops.paged_attention(q, *args)
    torch.cuda.synchronize()
    rt.check_status()
    assert_close_bf16(got, ref, f"paged attention {nq}/{nkv} heads")


def test_paged_attention_declines_other_shapes(rt):
    from nanovllm_b200 import ops
    kc = torch.zeros(1, 256, 1, 128, dtype=torch.bfloat16, device=DEV)
    lens, tables = torch.ones(1, dtype=torch.int32, device=DEV), torch.zeros(1, 1, dtype=torch.int32, device=DEV)
    assert ops.paged_attention(torch.zeros(1, 3, 128, dtype=torch.bfloat16, device=DEV), kc, kc, lens, tables, 1.0) is None
