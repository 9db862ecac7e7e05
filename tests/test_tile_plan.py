"""The planner of the many-token GEMM, read through b2_plan_tile_gemm (host arithmetic, no GPU): every K block of every tile is
computed once, by the pairs that the combine step expects, in the memory that the launch asks for."""
import ctypes as C

import pytest
from hypothesis import given, settings, strategies as st

SMS = 148
# clusters of 2 S CTAs resident at once: two CTAs per SM, then one
RESIDENT = [0, 148, 66, 44, 32, 0, 74, 33, 22, 16]
TMEM_COLUMNS = 512


def plan_of(abi, m, n, k, sms=SMS, resident=RESIDENT):
    p = abi.TilePlan()
    rc = abi.lib.b2_plan_tile_gemm(m, n, k, sms, (C.c_int * 10)(*resident) if resident else None, C.byref(p))
    return rc, p


def segments(abi, p, pair):
    buf = (C.c_int * (3 * 4096))()
    count = abi.lib.b2_plan_tile_segments(C.byref(p), pair, buf, 4096)
    assert 0 <= count <= 4096
    return [tuple(buf[3 * i:3 * i + 3]) for i in range(count)]


def check(abi, p, m, n, k, sms=SMS, resident=RESIDENT):
    tiles = p.tiles_f * p.tiles_t
    assert p.bn % 32 == 0 and 32 <= p.bn <= 256
    assert p.tiles_f * 256 >= n > (p.tiles_f - 1) * 256 and p.tiles_t * p.bn >= m > (p.tiles_t - 1) * p.bn
    assert p.kblocks * 64 >= k > (p.kblocks - 1) * 64 and p.grid % 2 == 0 and 1 <= p.group <= p.tiles_t
    # shared memory: the ring, the staging buffers, barriers; two accumulators fit tensor memory
    stage = 128 * 64 * 2 + p.bn * 64
    assert p.stages >= 1 and p.stages <= 12 and p.stages * stage <= p.bar_off and p.bar_off + 256 + 1024 <= p.smem <= 227 * 1024
    assert p.out_off + (8 if p.multi else 4) * 4096 <= p.bar_off
    if p.multi:
        assert p.out_off >= p.stages * stage and p.grid <= sms and p.split == 1
        assert 2 * max(32, 1 << (p.bn - 1).bit_length()) <= TMEM_COLUMNS
    else:
        assert p.grid == 2 * tiles * p.split and 1 <= p.split <= 4
        if p.split > 1:  # the exchange buffers lie where the ring was; all clusters wait for nobody but must be resident to pay
            most = (p.bn // 8 + p.split - 1) // p.split
            assert (p.split - 1) * most * 4096 <= p.out_off
            assert resident[(5 if p.smem > 113 * 1024 else 0) + p.split] >= tiles
    if m >= 512:  # one unbroken sum over K
        assert p.split == 1 and p.ranged == 0
    blocks = [0] * tiles
    holders, first_of = {}, {}
    for pair in range(p.grid // 2):
        for tile, k0, k1 in segments(abi, p, pair):
            assert 0 <= tile < tiles and 0 <= k0 < k1 <= p.kblocks
            assert k0 == (0 if tile not in holders else holders[tile][-1][1]), "ranges of a tile follow each other, pair by pair"
            holders.setdefault(tile, []).append((pair, k1))
            blocks[tile] += k1 - k0
            if k0 == 0 and k1 < p.kblocks and p.multi:
                assert pair not in first_of, "two split tiles in one workspace slot"
                first_of[pair] = tile
    assert blocks == [p.kblocks] * tiles
    if p.multi:
        first, last = C.c_int(), C.c_int()
        for tile, parts in holders.items():
            if len(parts) > 1:
                assert abi.lib.b2_plan_tile_holders(C.byref(p), tile, C.byref(first), C.byref(last)) == 0
                assert [x for x, _ in parts] == list(range(first.value, last.value + 1))
    return holders


# whole tiles in rounds, K ranges, split over 2..4 pairs, two CTAs per SM, one token past the decode sizes, ragged features
SHAPES = [(65, 256, 64), (97, 1032, 520), (160, 4096, 4096), (256, 24576, 4096), (391, 5120, 25600), (391, 51200, 5120), (511, 6144, 4096), (512, 4096, 12288),
          (777, 6144, 4096), (1500, 24576, 512), (8000, 4096, 1024), (16384, 51200, 5120), (300, 8, 8), (100, 151936, 4096)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_every_block_once(pkg, m, n, k):
    from nanovllm_b200 import _abi
    rc, p = plan_of(_abi, m, n, k)
    assert rc == 0
    check(_abi, p, m, n, k)


def test_each_way_to_run_is_chosen_somewhere(pkg):
    from nanovllm_b200 import _abi
    plans = {s: plan_of(_abi, *s)[1] for s in [(391, 5120, 25600), (160, 4096, 4096), (777, 6144, 4096), (4096, 24576, 4096), (65, 256, 64)]}
    assert plans[391, 5120, 25600].multi and plans[391, 5120, 25600].ranged > 0           # ranges of K blocks over the grid
    assert plans[160, 4096, 4096].split > 1                                               # K split over a cluster
    assert not plans[777, 6144, 4096].multi and SMS < plans[777, 6144, 4096].grid <= 2 * SMS  # whole tiles, two CTAs per SM
    assert plans[4096, 24576, 4096].multi and plans[4096, 24576, 4096].ranged == 0        # whole rounds
    assert (plans[65, 256, 64].split, plans[65, 256, 64].multi) == (1, 0)                 # one K block


def test_bad_arguments(pkg):
    from nanovllm_b200 import _abi
    for bad in [(0, 64, 64), (64, 0, 64), (64, 64, 0)]:
        assert plan_of(_abi, *bad)[0] == _abi.ERR_ARG
    assert plan_of(_abi, 100, 64, 64, sms=1)[0] == _abi.ERR_ARG
    assert _abi.lib.b2_plan_tile_gemm(100, 64, 64, SMS, None, None) == _abi.ERR_ARG
    rc, p = plan_of(_abi, 100, 64, 64, resident=None)
    assert rc == 0 and p.split == 1 and _abi.lib.b2_plan_tile_segments(C.byref(p), p.grid // 2, None, 0) < 0


@settings(max_examples=150, deadline=None)
@given(m=st.integers(65, 3000), n8=st.integers(1, 2000), k8=st.integers(1, 1000), sms=st.sampled_from([148, 132, 7, 2]))
def test_plan_property(m, n8, k8, sms):
    import __graft_entry__
    __graft_entry__.load_package()
    from nanovllm_b200 import _abi
    resident = [0] + [sms // s for s in (1, 2, 3, 4)] + [0] + [sms // (2 * s) for s in (1, 2, 3, 4)]
    rc, p = plan_of(_abi, m, n8 * 8, k8 * 8, sms=sms, resident=resident)
    assert rc == 0
    check(_abi, p, m, n8 * 8, k8 * 8, sms=sms, resident=resident)


def check_width(p, m):
    """The columns that are launched: the fewest in steps of 16 that as many whole tiles cover the tokens with, the plan's own where K is cut."""
    assert 16 <= p.width <= p.bn and p.tiles_t * p.width >= m > (p.tiles_t - 1) * p.width  # (no tile without tokens)
    if p.split == 1 and p.ranged == 0:
        assert p.width % 16 == 0 and p.tiles_t * (p.width - 16) < m
    else:
        assert p.width == p.bn
    # the last 32 columns are read whole: inside what is allocated, in powers of two, for one accumulator
    assert -(-p.width // 32) * 32 <= max(32, 1 << (p.width - 1).bit_length())


@pytest.mark.parametrize("m,n,k", SHAPES + [(m, 4096, 4096) for m in (513, 530, 565, 593, 777, 1041)])
def test_launched_width(pkg, m, n, k):
    from nanovllm_b200 import _abi
    rc, p = plan_of(_abi, m, n, k)
    assert rc == 0
    check_width(p, m)


@settings(max_examples=150, deadline=None)
@given(m=st.integers(65, 16384), n8=st.integers(1, 7000), k8=st.integers(1, 3200))
def test_launched_width_property(m, n8, k8):
    import __graft_entry__
    __graft_entry__.load_package()
    from nanovllm_b200 import _abi
    rc, p = plan_of(_abi, m, n8 * 8, k8 * 8)
    assert rc == 0
    check_width(p, m)
