"""All decoder layers of a decode step in one launch (b2_decode_stack) against float64 and against the layers called one by one.

What is compared is rounded to bf16 at about ten points of a layer in either form: 90 independent errors of 2^-9 / sqrt(3) over nine layers
are 2^-6.5.  The launch must be no further off than the layers (a tenth more is run-to-run luck of the roundings), and both within
2^-6.  With nine layers each of the three buffers that hand a phase's results to the next is used three times: a word left over
from three layers before would pass for a result."""
import pytest
import torch

from tests.gpu_util import ensure_group

pytestmark = pytest.mark.gpu
LAYERS, VOCAB = 9, 512


@pytest.fixture(params=[(16, 8, 3072), (8, 8, 1024), (16, 16, 2048), (24, 12, 3072)], ids=lambda s: f"{s[0]}q{s[1]}kv{s[2]}")
def shape(request):
    return request.param


def _runner(nq, nkv, inter, block_size=256, blocks=64):
    ensure_group()
    from nanovllm_b200.engine.model_runner import ModelConfig, ModelRunner
    config = ModelConfig(hidden_size=1024, num_attention_heads=nq, num_key_value_heads=nkv, head_dim=128, intermediate_size=inter, num_hidden_layers=LAYERS,
                         vocab_size=VOCAB, max_position_embeddings=4096)
    return ModelRunner(config, max_num_seqs=32, max_model_len=2048, max_num_batched_tokens=256, kvcache_block_size=block_size, num_kvcache_blocks=blocks,
                       enforce_eager=True, oneshot_tokens=64)


def _weights(runner):
    g = torch.Generator(device="cuda").manual_seed(3)
    for name, p in runner.model.named_parameters():
        if "norm" in name:
            p.data.uniform_(0.5, 1.5, generator=g)
        elif "embed" in name:
            p.data.normal_(0, 1, generator=g)


def _exact(runner, ids, pos, lens, tables, slots, qk_norms=True):
    """The same step in float64, on copies of the caches."""
    c = runner.config
    d, hd, nq, nkv = torch.float64, c.head_dim, c.num_attention_heads, c.num_key_value_heads

    def norm(x, m):
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + m.eps) * m.weight.to(d)

    model = runner.model.model
    h = model.embed_tokens.weight.to(d)[ids]
    n = len(lens)
    cs = model.layers[0].self_attn.rotary_emb.cos_sin_cache.reshape(-1, hd).to(d)[pos]
    cos, sin = cs[:, None, :hd // 2], cs[:, None, hd // 2:]

    def rope(x):
        a, b = x[..., :hd // 2], x[..., hd // 2:]
        return torch.cat((a * cos - b * sin, b * cos + a * sin), -1)

    new = []
    for layer in model.layers:
        at, mlp = layer.self_attn, layer.mlp
        qkv = (norm(h, layer.input_layernorm) @ at.qkv_proj.weight.to(d).t()).view(n, nq + 2 * nkv, hd)
        q, k, v = qkv.split([nq, nkv, nkv], 1)
        q, k = (rope(norm(q, at.q_norm)), rope(norm(k, at.k_norm))) if qk_norms else (rope(q), rope(k))
        kc, vc = at.attn.k_cache.to(d).view(-1, nkv, hd), at.attn.v_cache.to(d).view(-1, nkv, hd)
        for i, s in enumerate(slots):
            if s >= 0:
                kc[s], vc[s] = k[i], v[i]
        new.append((k, v))
        o = torch.zeros(n, nq, hd, dtype=d, device="cuda")
        for i, length in enumerate(lens):
            if length == 0:
                continue
            t = torch.arange(length, device="cuda")
            rows = torch.tensor(tables[i], device="cuda")[t // runner.block_size] * runner.block_size + t % runner.block_size
            kk, vv = kc[rows].repeat_interleave(nq // nkv, 1), vc[rows].repeat_interleave(nq // nkv, 1)
            p = torch.softmax(torch.einsum("hd,thd->ht", q[i], kk) * at.scaling, -1)
            o[i] = torch.einsum("ht,thd->hd", p, vv)
        h = h + o.view(n, -1) @ at.o_proj.weight.to(d).t()
        gu = norm(h, layer.post_attention_layernorm) @ mlp.gate_up_proj.weight.to(d).t()
        h = h + (torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2]) @ mlp.down_proj.weight.to(d).t()
    return norm(h, model.norm), new


def _compare(runner, monkeypatch, lens, tables, slots, qk_norms=True):
    from nanovllm_b200 import ops
    from nanovllm_b200.layers.attention import Attention
    from nanovllm_b200.models import qwen3
    from nanovllm_b200.utils.context import get_context, reset_context, set_context
    model = runner.model.model
    n = len(lens)
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    for plane in runner.kv_cache:
        plane.normal_(generator=g)
    runner.kv_cache[1][:, -1] = float("nan")  # a block nobody may read (it is in no table)
    cache = runner.kv_cache.clone()
    ids = torch.randint(0, VOCAB, (n,), generator=g, device="cuda")
    pos = torch.tensor([max(0, x - 1) for x in lens], device="cuda")
    width = max(len(t) for t in tables)
    rows = torch.tensor([t + [-1] * (width - len(t)) for t in tables], dtype=torch.int32, device="cuda")
    exact, _ = _exact(runner, ids, pos, lens, tables, slots, qk_norms)

    def stack_without_qk_norms():  # (no model has neither these norms nor a bias: the call itself)
        at, ctx = model.layers[0].self_attn, get_context()
        return ops.decode_stack(model.embed_tokens(ids), pos, [(*w[:6], None, None, *w[8:]) for w in model._stock_layers()], model.norm.weight, at.num_heads,
                                at.num_kv_heads, at.head_dim, runner.config.intermediate_size, model.norm.eps, at.rms_norm_eps, at.attn.scale,
                                at.rotary_emb.cos_sin_cache, ctx.context_lens, ctx.slot_mapping, ctx.block_tables)

    def run(forward):
        set_context(False, slot_mapping=torch.tensor(slots, dtype=torch.int32, device="cuda"), context_lens=torch.tensor(lens, dtype=torch.int32, device="cuda"),
                    block_tables=rows)
        runner.kv_cache.copy_(cache)
        out = forward()
        reset_context()
        return out, runner.kv_cache.clone()

    calls = []
    stack = ops.decode_stack
    monkeypatch.setattr(ops, "decode_stack", lambda *a: calls.append(stack(*a)) or calls[-1])
    with torch.inference_mode():
        launch = (lambda: runner.model(ids, pos)) if qk_norms else stack_without_qk_norms
        got, kv = run(launch)
        again, kv_again = run(launch)
        assert len(calls) == 2 and calls[0] is not None
        monkeypatch.setattr(qwen3, "_is_stock", lambda layer: False)
        if runner.block_size % 64 != 0:
            monkeypatch.setattr(Attention, "backend", "sdpa")  # (the only attention of the layers that takes such blocks)
        for layer in model.layers:
            monkeypatch.setattr(layer.self_attn, "qkv_bias", not qk_norms)  # (the layers leave the norms out of what would have a bias)
        layers, kv_layers = run(lambda: runner.model(ids, pos))
    runner.runtime.check_status()
    live = max((i + 1 for i, x in enumerate(lens) if x > 0), default=0)
    assert not got[live:].any()
    if live == 0:
        return

    def off(x):
        return ((x.double() - exact)[:live].norm() / exact[:live].norm()).item()

    assert off(got) <= 1.1 * off(layers) and off(got) < 2 ** -6, f"relative error {off(got):.2e}, the layers' {off(layers):.2e}"
    assert torch.equal(got, again) and torch.equal(kv.view(torch.int16), kv_again.view(torch.int16))
    # the cache: new rows within the roundings of one layer and more, everything else as it was
    flat = [x.view(2 * LAYERS, -1, x.shape[-2] * x.shape[-1]) for x in (kv, kv_layers, cache)]
    written = sorted({s for s in slots[:live] if s >= 0})
    other = torch.ones(flat[0].shape[1], dtype=torch.bool, device="cuda")
    other[written] = False
    assert torch.equal(flat[0][:, other].view(torch.int16), flat[2][:, other].view(torch.int16))
    if written:
        a, b = flat[0][:, written].float(), flat[1][:, written].float()
        assert (a - b).norm() <= 2 ** -6 * b.norm()
        assert torch.equal(a[0], b[0]) or (a[0] - b[0]).abs().max() <= 2 ** -6 * b[0].abs().max()


def _batch(lens, block_size, blocks, seed=1):
    """Tables from a shuffled free list, slots of the last tokens."""
    order = torch.randperm(blocks - 1, generator=torch.Generator().manual_seed(seed)).tolist()
    tables, slots = [], []
    for n in lens:
        need = max(1, -(-n // block_size))
        t, order = order[:need], order[need:]
        tables.append(t)
        slots.append(t[(n - 1) // block_size] * block_size + (n - 1) % block_size if n else -1)
    return tables, slots


# one row; few groups and many; edges of a group, of a block and of the 8 tokens multiplied at a time; gaps and padding
LENS = {"one": [1], "short": [17, 16, 15], "long_one": [2000], "edges": [255, 256, 257, 1, 33, 512, 513], "eight": [300] * 8, "nine": [40 * i + 1 for i in range(9)],
        "sixteen": [64 * i + 5 for i in range(16)], "uneven": [1900] + [3] * 10, "gaps": [0, 31, 0, 700, 0, 0], "padding": [0, 0, 0]}


@pytest.mark.parametrize("lens", list(LENS.values()), ids=list(LENS))
def test_batches(pkg, monkeypatch, lens):
    runner = _runner(16, 8, 3072)
    try:
        _weights(runner)
        _compare(runner, monkeypatch, lens, *_batch(lens, 256, 64))
    finally:
        runner.exit()


def test_shapes(pkg, monkeypatch, shape):
    runner = _runner(*shape)
    try:
        _weights(runner)
        lens = [1, 200, 77, 1030, 16, 512, 5, 300, 31, 90]
        _compare(runner, monkeypatch, lens, *_batch(lens, 256, 64))
    finally:
        runner.exit()


@pytest.mark.parametrize("block_size", [16, 32, 64])
def test_small_blocks(pkg, monkeypatch, block_size):
    runner = _runner(16, 8, 3072, block_size=block_size, blocks=200)
    try:
        _weights(runner)
        lens = [1, 64, 65, 500, 128, 63]
        _compare(runner, monkeypatch, lens, *_batch(lens, block_size, 200))
    finally:
        runner.exit()


def test_without_head_norms(pkg, monkeypatch):
    runner = _runner(16, 8, 3072)
    try:
        _weights(runner)
        lens = [1, 200, 77, 1030, 16, 512, 5, 300, 31, 90]
        tables, slots = _batch(lens, 256, 64)
        _compare(runner, monkeypatch, lens, tables, slots, qk_norms=False)
        monkeypatch.undo()
        slots[1] = -1  # (all new rows stored ahead)
        _compare(runner, monkeypatch, lens, tables, slots, qk_norms=False)
    finally:
        runner.exit()


@pytest.mark.parametrize("kind", ["several_new_tokens", "frozen_row", "slot_elsewhere"])
def test_rows_that_read_each_other(pkg, monkeypatch, kind):
    """Batches whose new rows cannot be handed from the projection to one reader: two new tokens of one sequence, a row that stores
    nothing and reads what its cache holds, a row that stores where its table does not say."""
    runner = _runner(16, 8, 3072)
    try:
        _weights(runner)
        lens = [100, 300, 301, 40]
        tables, slots = _batch(lens, 256, 64)
        if kind == "several_new_tokens":
            tables[1] = tables[2]
            slots[1] = tables[2][299 // 256] * 256 + 299 % 256
        elif kind == "frozen_row":
            slots[3] = -1
        else:
            slots[0] = 62 * 256 + 7  # a block of no table
            assert all(62 not in t for t in tables)
        _compare(runner, monkeypatch, lens, tables, slots)
    finally:
        runner.exit()


def test_left_to_the_layers(pkg, monkeypatch):
    """More rows than are served, hooks on a layer, and another attention backend go through the layers."""
    from nanovllm_b200 import ops
    from nanovllm_b200.layers.attention import Attention
    from nanovllm_b200.utils.context import reset_context, set_context
    runner = _runner(16, 8, 3072)
    try:
        _weights(runner)
        outs = []
        stack = ops.decode_stack
        monkeypatch.setattr(ops, "decode_stack", lambda *a: outs.append(stack(*a)) or outs[-1])

        def run(lens):
            tables, slots = _batch(lens, 256, 64)
            outs.clear()
            set_context(False, slot_mapping=torch.tensor(slots, dtype=torch.int32, device="cuda"), context_lens=torch.tensor(lens, dtype=torch.int32, device="cuda"),
                        block_tables=torch.tensor(tables, dtype=torch.int32, device="cuda"))
            with torch.inference_mode():
                out = runner.model(torch.arange(len(lens), device="cuda"), torch.tensor(lens, device="cuda") - 1)
            reset_context()
            assert torch.isfinite(out.float()).all()
            return [o is not None for o in outs]

        assert run([5] * 16) == [True]
        assert run([5] * 17) == [False]
        seen = []
        handle = runner.model.model.layers[1].register_forward_hook(lambda *a: seen.append(1))
        assert run([5] * 3) == [] and seen == [1]
        handle.remove()
        monkeypatch.setattr(Attention, "backend", "sdpa")
        assert run([5] * 3) == []
        monkeypatch.undo()
    finally:
        runner.exit()


def test_captured_step_serves_later_batches(pkg):
    """One captured launch, replayed for batches of other lengths and with padded rows, gives what an eager call gives."""
    from nanovllm_b200.utils.context import reset_context, set_context
    runner = _runner(16, 8, 3072)
    try:
        _weights(runner)
        g = torch.Generator(device="cuda").manual_seed(9)
        for plane in runner.kv_cache:
            plane.normal_(generator=g)
        cache = runner.kv_cache.clone()
        n, width = 8, 8
        ids, pos = torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(n, dtype=torch.int64, device="cuda")
        lens, slots = torch.zeros(n, dtype=torch.int32, device="cuda"), torch.full((n,), -1, dtype=torch.int32, device="cuda")
        tables = torch.zeros(n, width, dtype=torch.int32, device="cuda")
        with torch.inference_mode():
            set_context(False, slot_mapping=slots, context_lens=lens, block_tables=tables)
            runner.model(ids, pos)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                out = runner.model(ids, pos)
            for batch in ([300] * 8, [1, 2000, 17], [5, 0, 700, 33, 256]):
                t, s = _batch(batch, 256, 64)
                m = len(batch)
                lens.zero_(), slots.fill_(-1)
                lens[:m], slots[:m] = torch.tensor(batch, dtype=torch.int32), torch.tensor(s, dtype=torch.int32)
                pos[:m] = torch.tensor(batch).sub(1).clamp_min(0)
                ids.copy_(torch.randint(0, VOCAB, (n,), generator=g, device="cuda"))
                for i, x in enumerate(t):
                    tables[i, :len(x)] = torch.tensor(x, dtype=torch.int32)
                for _ in range(2):  # a replay after a replay
                    runner.kv_cache.copy_(cache)
                    graph.replay()
                    kv = runner.kv_cache.clone()
                runner.kv_cache.copy_(cache)
                eager = runner.model(ids, pos)
                assert torch.equal(out, eager) and torch.equal(kv, runner.kv_cache)
        reset_context()
        runner.runtime.check_status()
        del graph
    finally:
        runner.exit()


@pytest.mark.parametrize("kind", ["inf", "nan"])
def test_scores_that_are_no_numbers(pkg, monkeypatch, kind):
    """A context that many CTAs share, with an infinite key in the last of its parts, or with one part (here of 14 groups of 16 tokens)
    whose keys are all NaN: the row comes out as NaN, as layer by layer, and the row beside it is untouched."""
    from nanovllm_b200.models import qwen3
    from nanovllm_b200.utils.context import reset_context, set_context
    runner = _runner(16, 8, 3072)
    try:
        _weights(runner)
        lens = [2000, 1900]
        tables, slots = _batch(lens, 256, 64)
        for plane in runner.kv_cache:
            plane.normal_(generator=torch.Generator(device="cuda").manual_seed(5))
        keys = runner.kv_cache[0, 0].view(-1, 8, 128)
        for token in [1900] if kind == "inf" else range(5 * 14 * 16, 6 * 14 * 16):
            keys[tables[0][token // 256] * 256 + token % 256, 0, :1 if kind == "inf" else 128] = float(kind)

        def run():
            set_context(False, slot_mapping=torch.tensor(slots, dtype=torch.int32, device="cuda"), context_lens=torch.tensor(lens, dtype=torch.int32, device="cuda"),
                        block_tables=torch.tensor(tables, dtype=torch.int32, device="cuda"))
            with torch.inference_mode():
                out = runner.model(torch.tensor([1, 2], device="cuda"), torch.tensor(lens, device="cuda") - 1)
            reset_context()
            return out.float()

        got = run()
        monkeypatch.setattr(qwen3, "_is_stock", lambda layer: False)
        layers = run()
        runner.runtime.check_status()
        assert layers[0].isnan().all() and got[0].isnan().all()
        assert (got[1] - layers[1]).norm() <= 2 ** -6 * layers[1].norm()
    finally:
        runner.exit()


def test_rotary_table_off_16_bytes(pkg, monkeypatch):
    """The layers read the rotary factors one by one for so few rows; the launch takes four at a time and leaves such a table to them."""
    from nanovllm_b200.models import qwen3
    from nanovllm_b200.utils.context import reset_context, set_context
    runner = _runner(16, 8, 3072)
    rotary = runner.model.model.layers[0].self_attn.rotary_emb
    table = rotary.cos_sin_cache
    try:
        _weights(runner)
        lens = [5, 40]
        tables, slots = _batch(lens, 256, 64)

        def run():
            set_context(False, slot_mapping=torch.tensor(slots, dtype=torch.int32, device="cuda"), context_lens=torch.tensor(lens, dtype=torch.int32, device="cuda"),
                        block_tables=torch.tensor(tables, dtype=torch.int32, device="cuda"))
            runner.kv_cache.zero_()
            with torch.inference_mode():
                out = runner.model(torch.tensor([1, 2], device="cuda"), torch.tensor(lens, device="cuda") - 1)
            reset_context()
            return out

        with torch.no_grad():
            rotary.cos_sin_cache = torch.empty(table.numel() + 1, device="cuda")[1:].view(table.shape).copy_(table)
        got = run()
        rotary.cos_sin_cache = table
        monkeypatch.setattr(qwen3, "_is_stock", lambda layer: False)
        assert torch.equal(got, run())
    finally:
        rotary.cos_sin_cache = table
        runner.exit()


def test_slot_mapping_longer_than_the_batch(pkg, monkeypatch):
    """The layers read as many slots as there are rows (a buffer kept for the largest batch will do), and so does the launch; fewer are refused."""
    from nanovllm_b200.models import qwen3
    from nanovllm_b200.utils.context import reset_context, set_context
    runner = _runner(16, 8, 3072)
    try:
        _weights(runner)
        lens = [5, 40]
        tables, slots = _batch(lens, 256, 64)

        def run(slots):
            set_context(False, slot_mapping=torch.tensor(slots, dtype=torch.int32, device="cuda"), context_lens=torch.tensor(lens, dtype=torch.int32, device="cuda"),
                        block_tables=torch.tensor(tables, dtype=torch.int32, device="cuda"))
            runner.kv_cache.zero_()
            try:
                with torch.inference_mode():
                    return runner.model(torch.tensor([1, 2], device="cuda"), torch.tensor(lens, device="cuda") - 1), runner.kv_cache.clone()
            finally:
                reset_context()

        for a, b in zip(run(slots), run(slots + [3, 4, 5])):
            assert torch.equal(a, b)
        with pytest.raises(ValueError):
            run(slots[:1])
        monkeypatch.setattr(qwen3, "_is_stock", lambda layer: False)
        run(slots + [3, 4, 5])
    finally:
        runner.exit()
