"""Which calls of Attention.attend go to the own kernels and which to the library: the rule's lines, on fakes of both."""
from types import SimpleNamespace

import pytest
import torch

SMS = 148


@pytest.fixture
def route(pkg, monkeypatch):
    """attend() on fakes: (own kernel serves, library present, call) -> who answered."""
    from nanovllm_b200.layers import attention as A

    def attend(nq, nkv, context, cache, q_rows, own=True, library=True, on_gpu=True):
        said = []

        def answer(name, result):
            return lambda q, *a, **k: said.append(name) or (q if result else None)

        if on_gpu:
            monkeypatch.setattr(A, "_sms", lambda _: SMS)
        monkeypatch.setattr(A, "ops", SimpleNamespace(paged_attention=answer("own", own), prefill_attention=answer("own", own)))
        for f in ("flash_attn_varlen_func", "flash_attn_with_kvcache"):
            monkeypatch.setattr(A, f, answer("library", True) if library else None)
        monkeypatch.setattr(A, "get_context", lambda: context)
        layer = A.Attention(nq, 128, 1.0, nkv)
        layer.k_cache = layer.v_cache = cache
        x = torch.empty(q_rows, nq, 128, device="meta")
        kv = torch.empty(q_rows, nkv, 128, device="meta")
        assert layer.attend(x, kv, kv) is not None
        return said[-1]

    return attend


def meta_cache(nkv, block=256):
    return torch.empty(4, block, nkv, 128, device="meta")


# wide groups: 236 pairs are the last that the library cuts on 148 SMs; it does not take blocks of 128 tokens
@pytest.mark.parametrize("n,nq,nkv,block,who", [(16, 32, 8, 256, "library"), (29, 64, 8, 256, "library"), (30, 32, 8, 256, "own"), (236, 4, 1, 256, "library"),
                                                (237, 4, 1, 256, "own"), (64, 32, 8, 256, "own"), (16, 16, 8, 256, "own"), (1, 8, 8, 256, "own"), (16, 32, 8, 128, "own")])
def test_decode(route, n, nq, nkv, block, who):
    context = SimpleNamespace(is_prefill=False, context_lens=None, block_tables=None)
    assert route(nq, nkv, context, meta_cache(nkv, block), n) == who
    assert route(nq, nkv, context, meta_cache(nkv, block), n, library=False) == "own"
    assert route(nq, nkv, context, meta_cache(nkv, block), n, own=False) == "library"


# wide groups over the cache: one row per sequence; up to 148 tiles of 64 rows and a head; not without a cache, not for narrow groups
@pytest.mark.parametrize("rows,nq,nkv,cached,block,who", [
    ([1], 32, 8, True, 256, "library"), ([1] * 40, 32, 8, True, 256, "library"), ([16], 32, 8, True, 256, "library"), ([256], 32, 8, True, 256, "library"),
    ([257], 32, 8, True, 256, "own"), ([100] * 2, 32, 8, True, 256, "library"), ([100] * 4, 32, 8, True, 256, "own"), ([1024], 32, 8, True, 256, "own"),
    ([250, 1], 24, 8, True, 256, "library"), ([250, 1, 1], 32, 8, True, 256, "own"), ([1], 32, 8, False, 256, "own"), ([16], 32, 8, False, 256, "own"),
    ([1], 16, 8, True, 256, "own"), ([16], 16, 8, True, 256, "own"), ([16], 32, 8, True, 128, "own")])
def test_prefill(route, rows, nq, nkv, cached, block, who):
    cu = torch.tensor([0] + rows).cumsum(0).to(torch.int32)
    context = SimpleNamespace(is_prefill=True, cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=max(rows), max_seqlen_k=max(rows),
                              block_tables=torch.zeros(len(rows), 4, dtype=torch.int32) if cached else None)
    assert route(nq, nkv, context, meta_cache(nkv, block), sum(rows)) == who
    assert route(nq, nkv, context, meta_cache(nkv, block), sum(rows), library=False) == "own"


def test_tensors_off_the_gpu_are_left_to_the_own_checks(route):
    """They are refused there, as ever: no device is asked for its SMs."""
    cu = torch.tensor([0, 1], dtype=torch.int32)
    for context in (SimpleNamespace(is_prefill=False, context_lens=None, block_tables=None),
                    SimpleNamespace(is_prefill=True, cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=1, max_seqlen_k=1, block_tables=torch.zeros(1, 4))):
        assert route(32, 8, context, meta_cache(8), 1, on_gpu=False) == "own"
