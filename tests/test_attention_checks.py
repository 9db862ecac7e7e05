"""The attention calls read lengths, block tables, keys and values through raw pointers: a call whose operands do not fit each
other is refused on the host.  Shapes and types need no GPU; one operand on the wrong device does."""
import pytest
import torch

DEV = "cuda:0"


def paged_args(dev="cpu"):
    n, nq, nkv, hd = 3, 4, 2, 128
    cache = [torch.zeros(4, 256, nkv, hd, dtype=torch.bfloat16, device=dev) for _ in range(2)]
    return dict(q=torch.zeros(n, nq, hd, dtype=torch.bfloat16, device=dev), k_cache=cache[0], v_cache=cache[1],
                context_lens=torch.ones(n, dtype=torch.int32, device=dev), block_tables=torch.zeros(n, 2, dtype=torch.int32, device=dev))


def prefill_args(dev="cpu", paged=False):
    n, nq, nkv, hd = 5, 4, 2, 128
    kv = [torch.zeros(*((4, 256) if paged else (n,)), nkv, hd, dtype=torch.bfloat16, device=dev) for _ in range(2)]
    cu = torch.tensor([0, 2, 5], dtype=torch.int32, device=dev)
    return dict(q=torch.zeros(n, nq, hd, dtype=torch.bfloat16, device=dev), k=kv[0], v=kv[1], cu_q=cu, cu_k=cu.clone(), max_q=3,
                block_tables=torch.zeros(2, 2, dtype=torch.int32, device=dev) if paged else None)


def call(kind, args, handle=None):
    from nanovllm_b200 import _abi
    return (_abi.native.paged_attention if kind == "paged" else _abi.native.prefill_attention)(handle, *args.values(), 1.0)


def make(kind, dev="cpu"):
    return paged_args(dev) if kind == "paged" else prefill_args(dev, paged=kind == "prefix")


BAD = [("paged", "k_cache", lambda t: t[..., :64].contiguous(), ValueError), ("paged", "v_cache", lambda t: t[:2].contiguous(), ValueError),
       ("paged", "v_cache", lambda t: t.half(), TypeError), ("paged", "k_cache", lambda t: t.half(), TypeError),
       ("paged", "context_lens", lambda t: t[:2], ValueError), ("paged", "context_lens", lambda t: t.repeat(2)[::2], AssertionError),
       ("paged", "context_lens", lambda t: t.long(), AssertionError), ("paged", "context_lens", lambda t: t.view(-1, 1), ValueError),
       ("paged", "block_tables", lambda t: t[:2], ValueError), ("paged", "block_tables", lambda t: t.long(), AssertionError),
       ("prefill", "v", lambda t: t.half(), TypeError), ("prefill", "v", lambda t: t[:4], ValueError), ("prefill", "cu_k", lambda t: t[:2], ValueError),
       ("prefill", "cu_q", lambda t: t.long(), AssertionError), ("prefill", "cu_k", lambda t: t.repeat(2)[::2], AssertionError),
       ("prefill", "cu_q", lambda t: t[:0], ValueError), ("prefill", "max_q", lambda _: 0, ValueError),
       ("prefix", "block_tables", lambda t: t[:1], ValueError), ("prefix", "v", lambda t: t[:3], ValueError), ("prefix", "block_tables", lambda t: t.long(), AssertionError)]


@pytest.mark.parametrize("kind,name,spoil,error", BAD)
def test_operands_that_do_not_fit_are_refused(pkg, kind, name, spoil, error):
    args = make(kind)
    args[name] = spoil(args[name])
    with pytest.raises(error):
        call(kind, args)


@pytest.mark.parametrize("kind", ["paged", "prefill", "prefix"])
def test_host_tensors_are_refused(pkg, kind):
    with pytest.raises(TypeError, match="GPU"):
        call(kind, make(kind))


# layouts the kernels cannot address go to the general path (None), they are no error
OTHER = [("paged", "q", lambda t: torch.zeros(t.numel() + 1, dtype=t.dtype)[1:].view(t.shape)), ("paged", "q", lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)),
         ("paged", "block_tables", lambda t: t[:1].expand(3, 2)), ("paged", "k_cache", lambda t: t.transpose(0, 1).contiguous().transpose(0, 1)),
         ("paged", "k_cache", lambda t: t[0]), ("prefill", "v", lambda t: torch.zeros(t.shape[0], 3, 128, dtype=t.dtype)[:, :2]),
         ("prefill", "q", lambda t: t.half()), ("prefix", "block_tables", lambda t: t[:1].expand(2, 2)), ("prefill", "q", lambda t: t.requires_grad_())]


@pytest.mark.parametrize("kind,name,other", OTHER)
def test_layouts_of_the_general_path_are_declined(pkg, kind, name, other):
    args = make(kind)
    args[name] = other(args[name])
    assert call(kind, args) is None


@pytest.mark.parametrize("n_seqs,each,nq,served", [(75, 4, 8, False), (74, 4, 8, True), (75, 95, 8, False), (75, 96, 8, True), (75, 4, 4, True), (300, 1, 2, False), (8, 1, 8, True)])
def test_many_short_prompts_of_wide_groups_are_declined(pkg, n_seqs, each, nq, served):
    """Four heads per KV head and more, over 296 tiles of which most rows would be empty; odd groups are never served."""
    nkv = 2
    kv = [torch.zeros(n_seqs * each, nkv, 128, dtype=torch.bfloat16) for _ in range(2)]
    cu = torch.arange(0, n_seqs * each + 1, each, dtype=torch.int32)
    args = dict(q=torch.zeros(n_seqs * each, nq, 128, dtype=torch.bfloat16), k=kv[0], v=kv[1], cu_q=cu, cu_k=cu.clone(), max_q=each, block_tables=None)
    if served:
        with pytest.raises(TypeError, match="GPU"):  # (host tensors)
            call("prefill", args)
    else:
        assert call("prefill", args) is None


@pytest.mark.gpu
@pytest.mark.parametrize("kind,name", [("paged", x) for x in ("k_cache", "v_cache", "context_lens", "block_tables")] +
                         [("prefix", x) for x in ("k", "v", "cu_q", "cu_k", "block_tables")])
def test_one_operand_on_the_host_is_refused(pkg, kind, name):
    args = make(kind, DEV)
    args[name] = args[name].cpu()
    with pytest.raises(TypeError, match=DEV):
        call(kind, args)
