"""Attention - decode over the paged cache, causal prefill over rows and over the cache - against plain PyTorch in fp32."""
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
# work ends inside a CTA's range, one and two query heads per KV head
CASES = [((1,), 16, 8), ((63, 64, 65, 0, 15, 16, 17), 16, 8), ((255, 256, 257, 0), 16, 8), ((4096,), 2, 1), ((4000, 3), 8, 8), ((300,), 8, 8),
         (tuple(range(1, 620, 7)), 8, 4), ((700,) * 130, 2, 1),
         # dealt whole or cut: the longest item just within and just past the limit, as many items as CTAs and one sequence more, equal counts
         ((576,), 16, 8), ((577,), 16, 8), (tuple(range(40, 706, 18)), 16, 8), (tuple(range(40, 724, 18)), 16, 8), ((3000,), 16, 8),
         # rows without a context at the end, between others, alone
         (tuple(range(40, 706, 18)) + (0,) * 11, 16, 8), ((0, 300, 0, 0, 900, 0), 16, 8), ((0, 0), 16, 8), ((700,) * 60 + (0,) * 4, 8, 8)]

# wide groups, where there are enough (sequence, KV head) pairs: edges of the 16-row groups, the tiles of 64 and the blocks of 128 tokens, of a
# cache block, rows without a context, three, four, seven and eight query heads per KV head, the fewest pairs that are served (one CTA per SM), two
WIDE = [((0, 1, 15, 16, 17, 63, 64, 65, 79, 80, 81, 127, 128, 129, 191, 192, 193, 255, 256, 257, 0, 383, 384, 385, 511, 512, 513, 700, 1200, 0), 32, 8),
        (tuple(range(1, 900, 29)), 64, 8), (tuple(range(40, 520, 6)), 9, 3), (tuple(range(3, 1000, 16)) + (0,) * 3, 28, 4), ((257,) * 128, 4, 1),
        (tuple(range(1, 700, 14)), 32, 8), (tuple(range(1, 480, 8)), 64, 8)]  # and three and four CTAs per SM


@pytest.mark.parametrize("lens,nq,nkv", CASES + WIDE)
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


# (new tokens, cached tokens) per sequence: edges of the 128-token tiles and the 64-token key blocks, a prefix, several blocks, one token
PREFILL = [([(1, 0)], False), ([(63, 0), (64, 0), (65, 0), (191, 0), (193, 0)], False), ([(64, 64), (63, 1), (65, 63)], True), ([(127, 0), (128, 0), (129, 0)], False), ([(117, 0)], False), ([(300, 0), (5, 0), (1000, 0)], False),
           ([(100, 512), (130, 256), (1, 255), (256, 1)], True), ([(900, 1100)], True)]


@pytest.mark.parametrize("nq,nkv", [(16, 8), (8, 2), (8, 1)])
@pytest.mark.parametrize("seqs,paged", PREFILL)
def test_prefill_attention_against_fp32(rt, seqs, paged, nq, nkv):
    from nanovllm_b200 import ops
    hd, bs, scale = 128, 256, 128 ** -0.5
    g = torch.Generator().manual_seed(sum(a + b for a, b in seqs))
    tokens = sum(a for a, _ in seqs)
    qkv = torch.randn(tokens, (nq + 2 * nkv) * hd, generator=g).bfloat16()
    need = [-(-(a + b) // bs) for a, b in seqs]
    free = torch.randperm(sum(need), generator=g).tolist()
    tables = torch.full((len(seqs), max(need) + 1), -1, dtype=torch.int32)
    kc, vc = (torch.full((sum(need), bs, nkv, hd), float("nan")).bfloat16() for _ in range(2))
    ref, at = torch.zeros(tokens, nq, hd), 0
    for i, (new, old) in enumerate(seqs):
        tables[i, :need[i]] = torch.tensor([free.pop() for _ in range(need[i])], dtype=torch.int32)
        rows = qkv[at:at + new]
        k, v = (rows[:, (nq + j * nkv) * hd:(nq + (j + 1) * nkv) * hd].view(new, nkv, hd) for j in (0, 1))
        if paged:
            k, v = (torch.cat((torch.randn(old, nkv, hd, generator=g).bfloat16(), x)) for x in (k, v))
            for p in range(old + new):
                blk = int(tables[i, p // bs])
                kc[blk, p % bs], vc[blk, p % bs] = k[p], v[p]
        q = rows[:, :nq * hd].float().view(new, nq, hd)
        kf, vf = (x.float().repeat_interleave(nq // nkv, 1) for x in (k, v))
        s = torch.einsum("qhd,khd->hqk", q, kf) * scale
        s.masked_fill_(torch.arange(old + new) > (torch.arange(new) + old).unsqueeze(1), float("-inf"))
        ref[at:at + new] = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), vf)
        at += new
    cu = torch.tensor([0] + [a for a, _ in seqs]).cumsum(0).to(torch.int32).to(DEV)
    cu_k = torch.tensor([0] + [a + b for a, b in seqs]).cumsum(0).to(torch.int32).to(DEV)
    x = qkv.to(DEV)
    q, k, v = (x[:, a * hd:b * hd].view(tokens, b - a, hd) for a, b in ((0, nq), (nq, nq + nkv), (nq + nkv, nq + 2 * nkv)))
    max_q = max(a for a, _ in seqs)
    if paged:
        got = ops.prefill_attention(q, kc.to(DEV), vc.to(DEV), cu, cu_k, max_q, tables.to(DEV), scale)
    else:
        got = ops.prefill_attention(q, k, v, cu, cu_k, max_q, None, scale)
    torch.cuda.synchronize()
    rt.check_status()
    assert_close_bf16(got, ref, f"prefill attention {seqs}")


def test_prefill_does_not_see_the_next_sequence(rt):
    """Rows past a sequence's last key are its neighbour's: their values, whatever they are, must not reach it."""
    from nanovllm_b200 import ops
    nq, nkv, hd = 4, 2, 128
    g = torch.Generator(device=DEV).manual_seed(5)
    lens = [100, 60, 129, 40]  # every one ends inside a block of 128 keys
    t = sum(lens)
    q, k, v = (torch.empty(t, h, hd, device=DEV).normal_(generator=g).bfloat16() for h in (nq, nkv, nkv))
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).to(DEV)
    clean = ops.prefill_attention(q, k, v, cu, cu, max(lens), None, hd ** -0.5)
    k[100:160], v[100:160] = float("nan"), float("inf")  # the second sequence
    q[289:], k[289:], v[289:] = float("inf"), float("-inf"), float("nan")  # and the fourth
    got = ops.prefill_attention(q, k, v, cu, cu, max(lens), None, hd ** -0.5)
    torch.cuda.synchronize()
    rt.check_status()
    for a, b in ((0, 100), (160, 289)):
        assert torch.equal(got[a:b], clean[a:b])


@pytest.mark.parametrize("std", [1.0, 4.0])
def test_prefill_rounds_probabilities_against_the_row_maximum(rt, std):
    """Probabilities are rounded to bf16 relative to their row's maximum, which is then exact: the error against float64 is that of
    plain PyTorch doing the same, whether the scores are flat or peaked.  Bound: the maximum of an earlier block is not the row's,
    which moves each rounding but not their size; over 1.5 million elements the two errors agree to a percent or two.  (A scale that
    lags behind the maximum by up to 2^8 shows 1.2 times the error at the second setting.)"""
    from nanovllm_b200 import ops
    nq, nkv, hd, t = 8, 4, 128, 1500
    g = torch.Generator(device=DEV).manual_seed(17)
    q, k, v = (torch.empty(t, h, hd, device=DEV).normal_(0, s, generator=g).bfloat16() for h, s in ((nq, std), (nkv, 1.0), (nkv, 1.0)))
    cu = torch.tensor([0, t], dtype=torch.int32, device=DEV)
    got = ops.prefill_attention(q, k, v, cu, cu, t, None, hd ** -0.5)
    kd, vd = (x.double().repeat_interleave(2, 1) for x in (k, v))
    scores = torch.einsum("qhd,khd->hqk", q.double(), kd) * hd ** -0.5
    scores.masked_fill_(torch.ones(t, t, dtype=torch.bool, device=DEV).triu(1), float("-inf"))
    exact = torch.einsum("hqk,khd->qhd", torch.softmax(scores, -1), vd)
    p = torch.exp(scores - scores.amax(-1, keepdim=True)).float()
    plain = (torch.einsum("hqk,khd->qhd", p.bfloat16().double(), vd) / p.double().sum(-1).t().unsqueeze(-1)).bfloat16()
    ours, bound = ((x.double() - exact).norm().item() for x in (got, plain))
    assert ours <= 1.05 * bound, f"error {ours / exact.norm().item():.3e} against {bound / exact.norm().item():.3e}"


@pytest.mark.parametrize("nq,nkv", [(2, 1), (8, 4), (32, 16)])
@pytest.mark.parametrize("slope", [0.0, 0.05, -0.05])
def test_prefill_rescales_as_maxima_grow(rt, nq, nkv, slope):
    """Scores that rise or fall along the keys, by 2^9 from one block of 128 keys to the next: with the rise every block's maximum
    outgrows all earlier ones and the sum so far is scaled away, with the fall the first block outweighs the rest.  Both query
    heads of a KV head, in several head layouts, get their own scale."""
    from nanovllm_b200 import ops
    hd, lens = 128, [700, 129, 64]
    t = sum(lens)
    g = torch.Generator().manual_seed(nq)
    q, k, v = (torch.randn(t, h, hd, generator=g).bfloat16().float() for h in (nq, nkv, nkv))
    if slope:  # dimension 0 carries the trend, half as steep for the second head of a pair
        q[..., 0] = torch.tensor([16.0, 8.0]).repeat(nq // 2)
        at = torch.cat([torch.arange(n) for n in lens])
        k[..., 0] = (at * slope * hd ** 0.5 / 16.0).unsqueeze(1)
    q, k, v = (x.bfloat16() for x in (q, k, v))
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    ref = torch.zeros(t, nq, hd)
    for a, b in zip(cu[:-1].tolist(), cu[1:].tolist()):
        kf, vf = (x[a:b].double().repeat_interleave(2, 1) for x in (k, v))
        s = torch.einsum("qhd,khd->hqk", q[a:b].double(), kf) * hd ** -0.5
        s.masked_fill_(torch.ones(b - a, b - a, dtype=torch.bool).triu(1), float("-inf"))
        ref[a:b] = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), vf).float()
    cu = cu.to(DEV)
    got = ops.prefill_attention(q.to(DEV), k.to(DEV), v.to(DEV), cu, cu, max(lens), None, hd ** -0.5)
    torch.cuda.synchronize()
    rt.check_status()
    assert_close_bf16(got, ref, f"prefill {nq}/{nkv} heads, slope {slope}")


def test_prefill_of_a_sequence_without_keys_is_zero(rt):
    from nanovllm_b200 import ops
    nq, nkv, hd = 4, 2, 128
    q = torch.randn(210, nq, hd, generator=torch.Generator().manual_seed(1)).bfloat16().to(DEV)
    cache = torch.randn(2, 1, 256, nkv, hd, generator=torch.Generator().manual_seed(2)).bfloat16().to(DEV)
    cu_q = torch.tensor([0, 5, 205, 210], dtype=torch.int32, device=DEV)
    cu_k = torch.tensor([0, 5, 5, 12], dtype=torch.int32, device=DEV)
    tables = torch.zeros(3, 1, dtype=torch.int32, device=DEV)
    torch.full((210, nq, hd), 7.0, dtype=torch.bfloat16, device=DEV)  # what the allocator hands out next is not zero already
    got = ops.prefill_attention(q, cache[0], cache[1], cu_q, cu_k, 200, tables, hd ** -0.5)
    torch.cuda.synchronize()
    rt.check_status()
    assert (got[5:205] == 0).all() and (got[:5] != 0).any() and (got[205:] != 0).any()


def paged_cache(total, nkv, g, bs=256):
    """Keys and values of sequences of so many tokens, in shuffled cache blocks: caches, block tables, and each sequence's own rows."""
    need = [max(1, -(-x // bs)) for x in total]
    ids = torch.randperm(sum(need), generator=g).split(need)
    tables = torch.zeros(len(total), max(16, max(need)), dtype=torch.int32)
    caches = [torch.randn(sum(need), bs, nkv, 128, generator=g).bfloat16() for _ in range(2)]
    for i, own in enumerate(ids):
        tables[i, :need[i]] = own
    return caches, tables, [[c[own].reshape(-1, nkv, 128)[:x] for c in caches] for own, x in zip(ids, total)]


def exact_attention(q, k, v, scale):
    """Causal attention of the last q.shape[0] positions in fp64: q [t, nq, hd], k, v [context, nkv, hd]."""
    k, v = (x.double().repeat_interleave(q.shape[1] // k.shape[1], 1) for x in (k, v))
    s = torch.einsum("qhd,khd->hqk", q.double(), k) * scale
    t, n = q.shape[0], k.shape[0]
    s.masked_fill_(torch.arange(n, device=q.device) > (torch.arange(t, device=q.device) + n - t).unsqueeze(1), float("-inf"))
    return torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v)


SCALES = [-128 ** -0.5, -0.5, 0.0, -0.0, 1e-39]


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("nq,nkv,n", [(16, 8, 20), (16, 8, 60), (32, 8, 31), (32, 8, 40), (64, 8, 60)])
def test_decode_takes_any_scale(rt, nq, nkv, n, scale):
    """Negative scales, zero and one that no normal number holds, on either kernel and each of the wide one's forms: contexts that end
    inside a block, where scores are masked."""
    from nanovllm_b200 import ops
    g = torch.Generator().manual_seed(n)
    lens = [(1 + 37 * i) % 300 for i in range(n)]
    caches, tables, rows = paged_cache(lens, nkv, g)
    q = torch.randn(n, nq, 128, generator=g).bfloat16()
    ref = torch.stack([exact_attention(q[i:i + 1], *rows[i], scale)[0].float() if lens[i] else torch.zeros(nq, 128) for i in range(n)])
    got = ops.paged_attention(q.to(DEV), *(c.to(DEV) for c in caches), torch.tensor(lens, dtype=torch.int32, device=DEV), tables.to(DEV), scale)
    torch.cuda.synchronize()
    rt.check_status()
    assert_close_bf16(got, ref, f"decode {nq}/{nkv} heads, scale {scale}")


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("nq,nkv", [(4, 2), (8, 2)])
@pytest.mark.parametrize("paged", [False, True])
def test_prefill_takes_any_scale(rt, paged, nq, nkv, scale):
    from nanovllm_b200 import ops
    g = torch.Generator().manual_seed(nq)
    new, old = [150, 64, 1, 200], [100, 0, 300, 56] if paged else [0] * 4
    total = [a + b for a, b in zip(new, old)]
    caches, tables, rows = paged_cache(total, nkv, g)
    q = torch.randn(sum(new), nq, 128, generator=g).bfloat16()
    ref = torch.cat([exact_attention(x, *kv, scale).float() for x, kv in zip(q.split(new), rows)])
    cu, cu_k = (torch.tensor([0] + x).cumsum(0).to(torch.int32).to(DEV) for x in (new, total))
    k, v = caches if paged else (torch.cat([kv[j] for kv in rows]) for j in (0, 1))
    got = ops.prefill_attention(q.to(DEV), k.to(DEV), v.to(DEV), cu, cu_k, max(new), tables.to(DEV) if paged else None, scale)
    torch.cuda.synchronize()
    rt.check_status()
    assert_close_bf16(got, ref, f"prefill {nq}/{nkv} heads, scale {scale}")


@pytest.mark.parametrize("n", [55, 56, 130])
@pytest.mark.parametrize("std", [1.0, 3.0])
def test_decode_of_narrow_groups_rounds_against_each_warps_own_maximum(rt, n, std):
    """With one or two query heads per KV head a probability is rounded to bf16 against the maximum that its warp (16 tokens of every 64) has
    seen, in a batch of any size: the error against float64 is that of plain PyTorch doing the same.  Bound: where a context is cut into
    parts the maxima are those of fewer tokens, which only makes more of the largest probabilities exact; over a million elements the
    two errors agree to half a percent.  (One maximum for all tokens of a block shows 1.05 times the error.)"""
    from nanovllm_b200 import ops
    nq, nkv, hd, t, bs = 16, 8, 128, 640, 256
    g = torch.Generator(device=DEV).manual_seed(n)
    kc, vc = (torch.empty(3 * n, bs, nkv, hd, device=DEV).normal_(generator=g).bfloat16() for _ in range(2))
    q = torch.empty(n, nq, hd, device=DEV).normal_(0, std, generator=g).bfloat16()
    tables = torch.randperm(3 * n, device=DEV, generator=g).to(torch.int32).view(n, 3)
    got = ops.paged_attention(q, kc, vc, torch.full((n,), t, dtype=torch.int32, device=DEV), tables, hd ** -0.5)
    ours = bound = 0.0
    for i in range(n):
        k, v = (c[tables[i].long()].view(-1, nkv, hd)[:t].double().repeat_interleave(2, 1) for c in (kc, vc))
        s = torch.einsum("hd,thd->ht", q[i].double(), k) * hd ** -0.5
        exact = torch.einsum("ht,thd->hd", torch.softmax(s, -1), v)
        by_warp = s.view(nq, t // 64, 4, 16)
        seen = by_warp.amax(-1).cummax(1).values.unsqueeze(-1)
        p, far = torch.exp(by_warp - seen), torch.exp(seen - s.amax(-1).view(nq, 1, 1, 1))
        p, rounded = ((x.double() * far).view(nq, t) for x in (p, p.float().bfloat16()))
        plain = (torch.einsum("ht,thd->hd", rounded, v) / p.sum(-1, keepdim=True)).bfloat16()
        ours += (got[i].double() - exact).pow(2).sum().item()
        bound += (plain.double() - exact).pow(2).sum().item()
    rt.check_status()
    assert ours ** 0.5 <= 1.02 * bound ** 0.5, f"{ours ** 0.5 / bound ** 0.5:.4f} times the error"


LIBRARY_DECODE = [((257,) * 30, 32, 8), (tuple(range(1, 1200, 18)), 32, 8), (tuple(range(70, 700, 6)), 64, 8), ((1056,) * 80, 9, 3)]


@pytest.mark.parametrize("lens,nq,nkv", LIBRARY_DECODE)
def test_wide_decode_is_the_librarys_result(rt, lens, nq, nkv):
    """Where the library does not cut contexts (0.8 of two pairs per SM and more) every probability has the same fp32 value and is rounded
    against the same maximum, and a product's sums are the same chain.  Bound: only the sum of probabilities is added up in another order; if its
    last bit differs, by 2^-23, one in 2^15 results falls on the other side of a tie between two bf16 numbers, 2^-8 apart."""
    flash = pytest.importorskip("flash_attn")
    from nanovllm_b200 import ops
    g = torch.Generator().manual_seed(len(lens))
    caches, tables, _ = paged_cache(lens, nkv, g)
    q = torch.randn(len(lens), nq, 128, generator=g).bfloat16().to(DEV)
    kc, vc, tables = (x.to(DEV) for x in (*caches, tables))
    lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    got = ops.paged_attention(q, kc, vc, lens, tables, 128 ** -0.5)
    ref = flash.flash_attn_with_kvcache(q.unsqueeze(1), kc, vc, cache_seqlens=lens, block_table=tables, softmax_scale=128 ** -0.5, causal=True).squeeze(1)
    rt.check_status()
    assert (got != ref).sum().item() <= max(4, got.numel() * 2 ** -15)
    assert_close_bf16(got, ref.float(), "wide decode and the library")


@pytest.mark.parametrize("nq,nkv,new,old", [(16, 8, (117, 64, 300), None), (32, 8, (500, 129, 1), None), (64, 8, (700,), None), (4, 2, (1500,), None),
                                            (32, 8, (100, 300, 65), (512, 77, 0)), (64, 8, (900,), (700,)), (8, 1, (257, 128), (256, 3000))])
def test_prefill_is_the_librarys_result(rt, nq, nkv, new, old):
    """Bit for bit: over rows for any group, over a block table for groups of four and more (two heads per KV head take one maximum per 64 keys there,
    the library one per 128)."""
    flash = pytest.importorskip("flash_attn")
    from nanovllm_b200 import ops
    g = torch.Generator().manual_seed(sum(new))
    total = [a + b for a, b in zip(new, old or [0] * len(new))]
    caches, tables, rows = paged_cache(total, nkv, g)
    q = torch.randn(sum(new), nq, 128, generator=g).bfloat16().to(DEV)
    k, v = (x.to(DEV) for x in (caches if old else (torch.cat([kv[j] for kv in rows]) for j in (0, 1))))
    cu, cu_k = (torch.tensor([0, *x]).cumsum(0).to(torch.int32).to(DEV) for x in (new, total))
    tables = tables.to(DEV) if old else None
    got = ops.prefill_attention(q, k, v, cu, cu_k, max(new), tables, 128 ** -0.5)
    ref = flash.flash_attn_varlen_func(q, k, v, max_seqlen_q=max(new), cu_seqlens_q=cu, max_seqlen_k=max(total), cu_seqlens_k=cu_k, softmax_scale=128 ** -0.5,
                                       causal=True, block_table=tables)
    rt.check_status()
    assert torch.equal(got, ref)


def trend(q, rows, slope):
    """Dimension 0 carries scores that rise or fall along the keys, half as steep for every other query head (the scale is 128 ** -0.5)."""
    q[..., 0] = torch.tensor([16.0, 8.0]).repeat(-(-q.shape[1] // 2))[:q.shape[1]].bfloat16()
    for k, _ in rows:
        k[..., 0] = (torch.arange(len(k)) * slope * 128 ** 0.5 / 16.0).unsqueeze(1).bfloat16()


def put_back(caches, tables, rows, bs=256):
    """The sequences' own rows into the cache again."""
    for i, kv in enumerate(rows):
        for cache, x in zip(caches, kv):
            for p in range(0, len(x), bs):
                cache[tables[i, p // bs], :len(x[p:p + bs])] = x[p:p + bs]


# every form: narrow groups with whole items and with even ranges, on both sides of 444 pairs; wide ones with two CTAs per SM and more
RAGGED = [0, 1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 191, 193, 255, 256, 257, 0, 511, 513, 640]


@pytest.mark.parametrize("slope", [0.05, -0.05])
@pytest.mark.parametrize("nq,nkv,n,far", [(16, 8, 20, 0), (16, 8, 55, 3000), (16, 8, 56, 3000), (16, 8, 64, 0), (8, 8, 60, 1500), (32, 8, 31, 0), (32, 8, 31, 2000), (64, 8, 60, 0)])
def test_decode_rescales_as_maxima_grow(rt, nq, nkv, n, far, slope):
    """Scores that rise or fall along the context by 2^9 in 128 tokens: whichever end a walk starts from, one of the two has every block's
    maximum outgrow all earlier ones.  Ragged lengths, rows without a context, one far longer than the rest."""
    from nanovllm_b200 import ops
    g = torch.Generator().manual_seed(n)
    lens = [RAGGED[i % len(RAGGED)] for i in range(n)]
    if far:
        lens[n // 2] = far
    caches, tables, rows = paged_cache(lens, nkv, g)
    q = torch.randn(n, nq, 128, generator=g).bfloat16()
    trend(q, rows, slope)
    put_back(caches, tables, rows)
    ref = torch.stack([exact_attention(q[i:i + 1], *rows[i], 128 ** -0.5)[0].float() if lens[i] else torch.zeros(nq, 128) for i in range(n)])
    got = ops.paged_attention(q.to(DEV), *(c.to(DEV) for c in caches), torch.tensor(lens, dtype=torch.int32, device=DEV), tables.to(DEV), 128 ** -0.5)
    torch.cuda.synchronize()
    rt.check_status()
    assert_close_bf16(got, ref, f"decode {nq}/{nkv} heads, slope {slope}")


@pytest.mark.parametrize("slope", [0.05, -0.05])
@pytest.mark.parametrize("nq,nkv", [(4, 2), (8, 2), (8, 1)])
def test_prefill_over_the_cache_rescales_as_maxima_grow(rt, nq, nkv, slope):
    from nanovllm_b200 import ops
    g = torch.Generator().manual_seed(nq + nkv)
    new, old = [300, 65, 128, 1], [200, 0, 64, 700]
    total = [a + b for a, b in zip(new, old)]
    caches, tables, rows = paged_cache(total, nkv, g)
    q = torch.randn(sum(new), nq, 128, generator=g).bfloat16()
    trend(q, rows, slope)
    put_back(caches, tables, rows)
    ref = torch.cat([exact_attention(x, *kv, 128 ** -0.5).float() for x, kv in zip(q.split(new), rows)])
    cu, cu_k = (torch.tensor([0] + x).cumsum(0).to(torch.int32).to(DEV) for x in (new, total))
    got = ops.prefill_attention(q.to(DEV), *(c.to(DEV) for c in caches), cu, cu_k, max(new), tables.to(DEV), 128 ** -0.5)
    torch.cuda.synchronize()
    rt.check_status()
    assert_close_bf16(got, ref, f"prefill over the cache {nq}/{nkv} heads, slope {slope}")


@pytest.mark.parametrize("nq,nkv,n", [(16, 8, 20), (16, 8, 60), (32, 8, 31), (32, 8, 60)])
def test_decode_keeps_nan_in_its_sequence(rt, nq, nkv, n):
    """A key that is NaN, or a value that is infinite, shows in its sequence's results, and in no other's."""
    from nanovllm_b200 import ops
    g = torch.Generator().manual_seed(n)
    lens = [200 + 13 * i for i in range(n)]
    caches, tables, rows = paged_cache(lens, nkv, g)
    q = torch.randn(n, nq, 128, generator=g).bfloat16().to(DEV)

    def run():
        return ops.paged_attention(q, *(c.to(DEV) for c in caches), torch.tensor(lens, dtype=torch.int32, device=DEV), tables.to(DEV), 128 ** -0.5).cpu()

    clean = run()
    rows[3][0][70], rows[7][1][5, :, 9] = float("nan"), float("inf")
    put_back(caches, tables, rows)
    got = run()
    rt.check_status()
    others = [i for i in range(n) if i not in (3, 7)]
    assert torch.equal(got[others], clean[others])
    assert got[3].isnan().all() and (got[7, :, 9] == float("inf")).all()
    rest = [d for d in range(128) if d != 9]
    assert torch.equal(got[7][:, rest], clean[7][:, rest])


@pytest.mark.parametrize("nq,nkv,paged", [(4, 2, False), (4, 2, True), (8, 2, False), (8, 2, True)])
def test_prefill_keeps_nan_from_earlier_rows(rt, nq, nkv, paged):
    """A key that is NaN shows in every row that sees it and in none before it, also where they share a block of keys."""
    from nanovllm_b200 import ops
    g = torch.Generator().manual_seed(3)
    lens = [300, 140]
    caches, tables, rows = paged_cache(lens, nkv, g)
    q = torch.randn(sum(lens), nq, 128, generator=g).bfloat16().to(DEV)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).to(DEV)

    def run():
        k, v = caches if paged else (torch.cat([kv[j] for kv in rows]) for j in (0, 1))
        return ops.prefill_attention(q, k.to(DEV), v.to(DEV), cu, cu, 300, tables.to(DEV) if paged else None, 128 ** -0.5).cpu()

    clean = run()
    rows[0][0][170] = float("nan")
    put_back(caches, tables, rows)
    got = run()
    rt.check_status()
    assert torch.equal(got[:170], clean[:170]) and torch.equal(got[300:], clean[300:])
    assert got[170:300].isnan().all()
