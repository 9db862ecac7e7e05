"""Timed cases of the tensor-parallel layer path, through the calls a serving program makes.

Three kinds of work:

  step     one ModelRunner.step() of a whole Qwen3 model on one GPU: "decode" (one new token for each of `seqs`
           sequences, CUDA graphs, paged KV cache) or "prefill" (the prompts of `seqs` sequences, with or without
           `cached` leading tokens of each in the cache already).  Greedy or with a temperature.
  layer    one decoder layer as models/qwen3.py wires it - qkv_fused, o_proj.forward_fused, the MLP's activation,
           down_proj.forward_fused - called eagerly, as prefill and enforce_eager run it.  The attention product
           between the first two is a library call: its result is one of the inputs.
  drop_in  the same layer as the original model code wires it, on the drop-in classes: separate norms, projections,
           rotary embedding, store_kvcache and activation.

The models are the configurations of engine/model_runner.py: Qwen3-0.6B, Qwen3-8B and Qwen3-32B shapes in bf16.
"""
import math
import random

import numpy as np
import torch
import torch.distributed as dist

import __graft_entry__

__graft_entry__.load_package()

from nanovllm_b200 import init_runtime, ops, shutdown_runtime  # noqa: E402
from nanovllm_b200.engine.model_runner import QWEN3_0_6B, QWEN3_8B, QWEN3_32B, ModelConfig, ModelRunner, Seq  # noqa: E402
from nanovllm_b200.layers.attention import store_kvcache  # noqa: E402
from nanovllm_b200.layers.layernorm import RMSNorm  # noqa: E402
from nanovllm_b200.layers.linear import MergedColumnParallelLinear  # noqa: E402
from nanovllm_b200.models.qwen3 import Qwen3DecoderLayer  # noqa: E402

MODELS = {"0.6b": QWEN3_0_6B, "8b": QWEN3_8B, "32b": QWEN3_32B}
BLOCK = 256          # tokens of a KV block
MAX_MODEL_LEN = 4096
MAX_TOKENS = 16384   # of one prefill step
EMBED_STD = 0.25


# ---- the cases -------------------------------------------------------------------------------------------------
def listed():
    def step(name, phase, model, seqs, longest, shortest, temperature=0.0, cached=0):
        return dict(name=name, kind="step", phase=phase, model=model, seqs=seqs, longest=longest, shortest=shortest,
                    temperature=temperature, cached=cached)

    def layer(name, kind, model, tokens, bias=False):
        return dict(name=name, kind=kind, model=model, tokens=tokens, bias=bias)

    return [
        # one user chatting with a small model: launches and latency
        step("decode_one", "decode", "0.6b", 1, 300, 300),
        # a lightly loaded server, contexts of all lengths, sampling
        step("decode_few", "decode", "0.6b", 37, 700, 40, temperature=0.6),
        # the throughput workload: 256 sequences, 100..1024 tokens, temperature 0.6
        step("decode_many", "decode", "0.6b", 256, 1024, 100, temperature=0.6),
        # the headline workload: Qwen3-8B, batch 64, greedy, just past 1024-token prompts
        step("decode_8b", "decode", "8b", 64, 1056, 1056),
        # a single short prompt: time to first token
        step("prompt_short", "prefill", "0.6b", 1, 117, 117),
        # a batch of prompts that share a cached system prompt
        step("prompts_cached", "prefill", "0.6b", 16, 900, 100, temperature=0.6, cached=512),
        # four 1024-token prompts of the headline workload
        step("prompts_8b", "prefill", "8b", 4, 1024, 1024),
        # one layer, called eagerly, from a few tokens to a long prefill chunk
        layer("layer_5", "layer", "8b", 5),
        layer("layer_150", "layer", "32b", 150),
        layer("layer_777", "layer", "8b", 777, bias=True),
        layer("layer_8192", "layer", "32b", 8192),
        # the original model code on the drop-in classes
        layer("drop_in_391", "drop_in", "8b", 391),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["decode", "decode", "prefill", "layer", "layer", "drop_in"])
    if kind in ("layer", "drop_in"):
        # a layer sees anything from one decode row to half of the largest prefill step
        return dict(kind=kind, model=rng.choice(["0.6b", "8b", "32b"]), tokens=_log_uniform(rng, 1, 8192), bias=rng.random() < 0.25)
    temperature = rng.choice([0.0, 0.6, 1.0])
    if kind == "decode":
        model = rng.choice(["0.6b", "0.6b", "8b"])
        seqs = _log_uniform(rng, 1, 512 if model == "0.6b" else 96)
        # the KV cache of one batch stays within what the listed cases hold
        longest = _log_uniform(rng, 32, min(3000, (140_000 if model == "0.6b" else 70_000) // seqs))
        return dict(kind="step", phase="decode", model=model, seqs=seqs, longest=longest, shortest=max(1, longest // rng.randint(1, 10)),
                    temperature=temperature, cached=0)
    model = rng.choice(["0.6b", "0.6b", "8b"])
    tokens = _log_uniform(rng, 16, 8192 if model == "0.6b" else 4096)
    seqs = rng.randint(max(1, -(-tokens // 2048)), max(1, min(32, tokens // 16)))
    longest = tokens // seqs
    return dict(kind="step", phase="prefill", model=model, seqs=seqs, longest=longest, shortest=max(1, longest // rng.randint(1, 4)),
                temperature=temperature, cached=rng.choice([0, 0, 256, 768]))


def _lengths(case):
    """Token counts of the sequences: evenly spread from shortest to longest."""
    n, lo, hi = case["seqs"], case["shortest"], case["longest"]
    return [hi - (hi - lo) * i // max(1, n - 1) for i in range(n)]


def _blocks(tokens):
    return -(-tokens // BLOCK)


def _layer_params(m):
    q, kv = m["num_attention_heads"] * m["head_dim"], m["num_key_value_heads"] * m["head_dim"]
    return m["hidden_size"] * (q + 2 * kv) + q * m["hidden_size"] + 3 * m["hidden_size"] * m["intermediate_size"]


def work(case):
    m = MODELS[case["model"]]
    h, q, kv = m["hidden_size"], m["num_attention_heads"] * m["head_dim"], m["num_key_value_heads"] * m["head_dim"]
    if case["kind"] == "step":
        lens, layers, n = _lengths(case), m["num_hidden_layers"], case["seqs"]
        head = m["vocab_size"] * h
        cached = case["cached"]
        if case["phase"] == "decode":
            rows, pairs, kv_read, kv_new = n, sum(lens), sum(lens) - n, n
        else:
            rows, pairs = sum(lens), sum(k * cached + k * (k + 1) // 2 for k in lens)
            kv_read, kv_new = cached * n, rows
        return {"bytes": 2 * (layers * _layer_params(m) + head) + 2 * layers * 2 * kv * (kv_read + kv_new) + 2 * rows * h,
                "flops": 2 * rows * layers * _layer_params(m) + 2 * n * head + 4 * pairs * q * layers}
    t = case["tokens"]
    # in: normed rows, residual, the attention's result; out: qkv, the cache rows, normed rows and residual
    return {"bytes": 2 * _layer_params(m) + 2 * t * (2 * h + q + (q + 2 * kv) + 2 * kv + 2 * h), "flops": 2 * t * _layer_params(m)}


def tolerance(case):
    # bf16 activations: an element carries a few roundings of 2^-9 from one layer, and those of every earlier layer in a
    # whole model.  Token ids: one in a hundred may fall on another side of a tie.
    if case["kind"] == "step":
        return {"rel": 2e-2, "differ": 0.01}
    return {"rel": 1e-2}


# ---- what a program has set up before the call -------------------------------------------------------------------
class _Session:
    """The process's runtime: there is one at a time, created for one model's runner or for layers alone."""
    key = None
    runner = None
    free_regions: list = []


def _open(key, make):
    if _Session.key == key:
        return _Session.runner
    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    if _Session.runner is not None:
        _Session.runner.exit()
    elif _Session.key is not None:
        shutdown_runtime()
    _Session.key = _Session.runner = None
    torch.cuda.empty_cache()
    _Session.runner = make()
    _Session.key = key
    return _Session.runner


REGIONS = 4  # batches whose KV blocks the cache has room for at once


class _Batch:
    """One batch of sequences with its own region of the runner's KV blocks, which it gives back."""

    def __init__(self, runner, case, seed):
        m = MODELS[case["model"]]
        rng = random.Random(seed)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        decode = case["phase"] == "decode"
        lens = _lengths(case)
        rng.shuffle(lens)
        total = [n + case["cached"] for n in lens]
        need = sum(_blocks(n) for n in total)
        self.region = _Session.free_regions.pop()
        self.runner, self.decode = runner, decode
        first = self.region * need
        ids = list(range(first, first + need))
        rng.shuffle(ids)  # the free list of a server that has been running for a while
        words = np.random.RandomState(seed & 0x7FFFFFFF)
        self.seqs = []
        for n in total:
            table, ids = ids[:_blocks(n)], ids[_blocks(n):]
            self.seqs.append(Seq(words.randint(0, m["vocab_size"], n).tolist(), table, 0 if decode else case["cached"]))
        self.temperatures = [case["temperature"]] * len(lens) if case["temperature"] > 0 else None
        self.kv = runner.kv_cache[:, :, first:first + need]
        if decode or case["cached"]:
            for plane in self.kv:  # normalised keys, values of the size the model produces
                for layer in plane:
                    layer.normal_(generator=gen)
        else:
            self.kv.zero_()
        self.rows = None
        if decode:
            slots = [s.block_table[(len(s) - 1) // BLOCK] * BLOCK + (len(s) - 1) % BLOCK for s in self.seqs]
            self.rows = torch.tensor(slots, device="cuda")
            self.flat = runner.kv_cache.view(2 * m["num_hidden_layers"], -1, m["num_key_value_heads"] * m["head_dim"])

    def __del__(self):
        if hasattr(self, "region"):
            _Session.free_regions.append(self.region)


def _make_runner(case):
    m = MODELS[case["model"]]
    need = sum(_blocks(n + case["cached"]) for n in _lengths(case))
    runner = ModelRunner(ModelConfig(**m), max_model_len=MAX_MODEL_LEN, max_num_batched_tokens=MAX_TOKENS, kvcache_block_size=BLOCK,
                         num_kvcache_blocks=REGIONS * need)
    # Random weights with a trained model's two traits that matter here: the residual stream does not explode over the
    # layers, and every row has one clear next token (here: the successor of its last token, or the token itself where
    # the embeddings are tied), so that a last-bit difference of a logit does not change the text.
    model = runner.model
    shrink = 1 / math.sqrt(2 * m["num_hidden_layers"])
    for layer in model.model.layers:
        layer.self_attn.o_proj.weight.data.mul_(shrink)
        layer.mlp.down_proj.weight.data.mul_(shrink)
    embed = model.model.embed_tokens.weight.data
    embed.normal_(0, EMBED_STD, generator=torch.Generator(device="cuda").manual_seed(1))
    if not m["tie_word_embeddings"]:
        model.lm_head.weight.data.copy_(torch.roll(embed, 1, 0))
    _Session.free_regions = list(range(REGIONS))
    return runner


class _Layer:
    """One decoder layer's weights, its cache, and the tokens that come in."""

    def __init__(self, case, seed):
        m, t = MODELS[case["model"]], case["tokens"]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        self.nq, self.nkv, self.hd = m["num_attention_heads"], m["num_key_value_heads"], m["head_dim"]
        config = ModelConfig(**dict(m, attention_bias=case["bias"]))
        prev = torch.get_default_dtype()
        torch.set_default_dtype(torch.bfloat16)
        try:
            with torch.device("cuda"):
                self.layer = Qwen3DecoderLayer(config)
                self.next_norm = RMSNorm(config.hidden_size, config.rms_norm_eps)
                if case["kind"] == "drop_in":  # gate and up stacked, as the original model code keeps them
                    self.layer.mlp.gate_up_proj = MergedColumnParallelLinear(config.hidden_size, [config.intermediate_size] * 2)
        finally:
            torch.set_default_dtype(prev)
        for name, p in list(self.layer.named_parameters()) + list(self.next_norm.named_parameters()):
            if p.dim() == 1 and "bias" not in name:
                p.data.uniform_(0.5, 1.5, generator=gen)
            else:
                p.data.normal_(0, 0.02, generator=gen)

        def rows(width, std=1.0):
            return torch.empty(t, width, dtype=torch.bfloat16, device="cuda").normal_(0, std, generator=gen)

        self.hidden, self.residual = rows(config.hidden_size), rows(config.hidden_size)
        self.attn = rows(self.nq * self.hd, 0.3)
        blocks = _blocks(t)
        self.k_cache = torch.zeros(blocks, BLOCK, self.nkv, self.hd, dtype=torch.bfloat16, device="cuda")
        self.v_cache = torch.zeros_like(self.k_cache)
        order = torch.randperm(blocks, generator=gen, device="cuda")
        at = torch.arange(t, device="cuda")
        self.slots = (order[at // BLOCK] * BLOCK + at % BLOCK).to(torch.int32)
        self.positions = torch.randint(0, MAX_MODEL_LEN, (1,), generator=gen, device="cuda") + at  # a chunk of some prompt


def prepare(case, seed):
    if case["kind"] == "step":
        key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
        return _Batch(_open(key, lambda: _make_runner(case)), case, seed)

    def layers_only():
        init_runtime(max_tokens=MAX_TOKENS, hidden=QWEN3_32B["hidden_size"])

    _open("layers", layers_only)
    state = _Layer(case, seed)
    state.run = _drop_in if case["kind"] == "drop_in" else _fused
    return state


# ---- one pass ----------------------------------------------------------------------------------------------------
def _step(b):
    tokens = np.array(b.runner.step(b.seqs, not b.decode, b.temperatures))
    if b.decode:  # the rows this step has added to the cache, and what the LM head saw
        return {"tokens": tokens, "kv": b.flat.index_select(1, b.rows), "hidden": b.runner.graph_vars["outputs"][:len(b.seqs)]}
    return {"tokens": tokens, "kv": b.kv}


def _fused(s):
    layer = s.layer
    attn, mlp = layer.self_attn, layer.mlp
    norms = (None, None) if attn.qkv_bias else (attn.q_norm.weight, attn.k_norm.weight)
    qkv = ops.qkv_fused(s.hidden, attn.qkv_proj.weight, attn.qkv_proj.bias, s.nq, s.nkv, s.hd, *norms, attn.rms_norm_eps,
                        s.positions, attn.rotary_emb.cos_sin_cache, s.k_cache, s.v_cache, s.slots)
    normed, residual = attn.o_proj.forward_fused(s.attn, s.residual, layer.post_attention_layernorm)
    normed, residual = mlp.down_proj.forward_fused(mlp.activation(normed), residual, s.next_norm)
    return {"qkv": qkv, "k_cache": s.k_cache, "v_cache": s.v_cache, "normed": normed, "residual": residual}


def _drop_in(s):
    layer = s.layer
    attn, mlp = layer.self_attn, layer.mlp
    x, residual = layer.input_layernorm(s.hidden, s.residual)
    q, k, v = attn.qkv_proj(x).split([attn.q_size, attn.kv_size, attn.kv_size], dim=-1)
    q, k, v = q.view(-1, s.nq, s.hd), k.view(-1, s.nkv, s.hd), v.view(-1, s.nkv, s.hd)
    if not attn.qkv_bias:
        q, k = attn.q_norm(q), attn.k_norm(k)
    q, k = attn.rotary_emb(s.positions, q, k)
    store_kvcache(k, v, s.k_cache, s.v_cache, s.slots)
    x, residual = layer.post_attention_layernorm(attn.o_proj(s.attn), residual)
    y = mlp.down_proj(mlp.act_fn(mlp.gate_up_proj(x)))
    return {"q": q, "k_cache": s.k_cache, "v_cache": s.v_cache, "out": y, "residual": residual}


def run(state):
    if isinstance(state, _Batch):
        return _step(state)
    return state.run(state)
