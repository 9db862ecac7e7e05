"""Which calls of Attention.attend go to the own kernels and which to the library: the rule's lines, on fakes of both."""
from types import SimpleNamespace

import pytest
import torch

SMS = 148


@pytest.fixture
def route(pkg, monkeypatch):
    """attend() on fakes: (own kernel serves, library present, call) -> who answered."""
    from nanovllm_b200.layers import attention as A

    def attend(nq, nkv, context, cache, q_rows, own=True, library=True):
        said = []

        def answer(name, result):
            return lambda q, *a, **k: said.append(name) or (q if result else None)

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
