"""The part of the model runner that hosts the tensor-parallel layer path.

It covers what nanovllm/engine/model_runner.py does around the model on each
rank: runtime set-up between device selection and model construction (:26-31),
KV-cache allocation and binding (:103-121), batch -> tensors for prefill and
decode (:123-188), CUDA-graph capture and replay for decode (:195-212,
:222-257) and teardown order (:50-59).  The scheduler, block manager,
tokenizer and the shared-memory RPC between ranks stay outside: callers hand
in token lists and block tables (every rank must be given the same batch).
"""
from __future__ import annotations

from dataclasses import dataclass, field

import numpy as np
import torch
import torch.distributed as dist

from ..layers.sampler import Sampler
from ..models.qwen3 import Qwen3ForCausalLM
from ..runtime import get_runtime, init_runtime, shutdown_runtime
from ..utils.context import reset_context, set_context

_TORCH_DTYPE = {np.dtype(np.int64): torch.int64, np.dtype(np.int32): torch.int32, np.dtype(np.float32): torch.float32}

FUSED_SAMPLER_MAX_ROWS = 256  # b2_lm_head_sample takes one token tile of the feature-lane layout


@dataclass
class ModelConfig:
    """The fields of a HF Qwen3 config the model reads (nanovllm/models/qwen3.py:127-143,167-171,199-203)."""
    hidden_size: int
    num_attention_heads: int
    num_key_value_heads: int
    head_dim: int
    intermediate_size: int
    num_hidden_layers: int
    vocab_size: int
    rms_norm_eps: float = 1e-6
    rope_theta: float = 1e6
    max_position_embeddings: int = 40960
    tie_word_embeddings: bool = False
    attention_bias: bool = False
    hidden_act: str = "silu"
    rope_scaling: dict | None = None


QWEN3_0_6B = dict(hidden_size=1024, num_attention_heads=16, num_key_value_heads=8, head_dim=128, intermediate_size=3072,
                  num_hidden_layers=28, vocab_size=151936, tie_word_embeddings=True)
QWEN3_8B = dict(hidden_size=4096, num_attention_heads=32, num_key_value_heads=8, head_dim=128, intermediate_size=12288,
                num_hidden_layers=36, vocab_size=151936, tie_word_embeddings=False)
QWEN3_32B = dict(hidden_size=5120, num_attention_heads=64, num_key_value_heads=8, head_dim=128, intermediate_size=25600,
                 num_hidden_layers=64, vocab_size=151936, tie_word_embeddings=False)


@dataclass
class Seq:
    """Minimal per-request state: the token ids so far, the KV blocks they
    occupy and how many leading tokens are already in the cache."""
    token_ids: list[int]
    block_table: list[int] = field(default_factory=list)
    num_cached_tokens: int = 0

    def __len__(self):
        return len(self.token_ids)


def random_init_(model: torch.nn.Module, seed: int, tp_rank: int) -> None:
    """Seeded N(0, 0.02) weights generated on the device (norm weights stay 1).
    Each rank draws its own shard: enough for throughput runs, where only the
    shapes matter; parity tests load shards of one full model instead."""
    g = torch.Generator(device="cuda").manual_seed(seed * 1000 + tp_rank)
    for name, p in model.named_parameters():
        if "norm" in name:
            p.data.fill_(1.0)
        else:
            p.data.copy_(torch.empty(p.shape, dtype=torch.float32, device=p.device).normal_(0, 0.02, generator=g))


_ROW_INPUT_BYTES = 28


def _row_inputs(buf: torch.Tensor) -> dict[str, torch.Tensor]:
    """The per-row inputs of a decode step as views of one byte buffer of _ROW_INPUT_BYTES per row."""
    n, out, at = buf.numel() // _ROW_INPUT_BYTES, {}, 0
    for name, dtype in (("input_ids", torch.int64), ("positions", torch.int64), ("slot_mapping", torch.int32),
                        ("context_lens", torch.int32), ("temperatures", torch.float32)):
        size = n * dtype.itemsize
        out[name] = buf[at:at + size].view(dtype)
        at += size
    return out


class ModelRunner:

    def __init__(self, config: ModelConfig, *, max_num_seqs: int = 512, max_model_len: int = 4096, max_num_batched_tokens: int = 16384,
                 kvcache_block_size: int = 256, num_kvcache_blocks: int | None = None, gpu_memory_utilization: float = 0.9,
                 enforce_eager: bool = False, oneshot_tokens: int = 1024, timeout_ms: int = 5000, seed: int = 0,
                 full_weights: dict | None = None, fused_sampler: bool | None = None, sample_seed: int = 0):
        assert dist.is_initialized(), "create the process group first (world size 1 included), as the reference does"
        self.config = config
        self.rank, self.world = dist.get_rank(), dist.get_world_size()
        self.block_size = kvcache_block_size
        self.max_num_seqs, self.max_model_len, self.max_num_batched_tokens = max_num_seqs, max_model_len, max_num_batched_tokens
        self.enforce_eager = enforce_eager
        # LM head and sampler in one pass (no [B, vocab] logits, no gather): the default at every world size
        if fused_sampler is None:
            fused_sampler = True
        self.fused_sampler = fused_sampler
        self.sample_seed = sample_seed
        self.device = torch.device("cuda", torch.cuda.current_device())
        # symmetric buffers exist before the layers are built, so graph capture sees fixed addresses
        self.runtime = init_runtime(max_tokens=max_num_batched_tokens, hidden=config.hidden_size, oneshot_tokens=oneshot_tokens,
                                    vocab=config.vocab_size, max_seqs=max_num_seqs, timeout_ms=timeout_ms)
        prev_dtype = torch.get_default_dtype()
        torch.set_default_dtype(torch.bfloat16)
        try:
            with self.device:  # (torch.set_default_device would leave a Python hook on every later torch call of the process)
                self.model = Qwen3ForCausalLM(config)
                if full_weights is not None:
                    self.model.load_full_weights(full_weights)
                else:
                    random_init_(self.model, seed, self.rank)
                self.sampler = Sampler()
                self._allocate_kv_cache(num_kvcache_blocks, gpu_memory_utilization)
                self.graphs: dict[int, torch.cuda.CUDAGraph] = {}
                if not enforce_eager:
                    self._capture_graphs()
        finally:
            torch.set_default_dtype(prev_dtype)

    # ---- teardown (reference :50-59) --------------------------------------
    def exit(self):
        self.graphs = {}
        self.graph_pool = None
        torch.cuda.synchronize()
        shutdown_runtime()

    # ---- KV cache (reference :103-121) -------------------------------------
    def _allocate_kv_cache(self, num_blocks: int | None, utilization: float):
        c = self.config
        self.num_kv_heads = c.num_key_value_heads // self.world
        block_bytes = 2 * c.num_hidden_layers * self.block_size * self.num_kv_heads * c.head_dim * 2
        if num_blocks is None:
            free, total = torch.cuda.mem_get_info()
            budget = int(total * utilization) - (total - free)
            # activations of the largest prefill step: a few [tokens, widest layer output] bf16 tensors
            widest = max(2 * c.intermediate_size // self.world, c.hidden_size, (c.num_attention_heads + 2 * c.num_key_value_heads) * c.head_dim // self.world)
            budget -= 6 * self.max_num_batched_tokens * widest * 2
            num_blocks = budget // block_bytes
        assert num_blocks > 0, "no memory left for the KV cache"
        self.num_kvcache_blocks = int(num_blocks)
        self.kv_cache = torch.zeros(2, c.num_hidden_layers, self.num_kvcache_blocks, self.block_size, self.num_kv_heads, c.head_dim,
                                    dtype=torch.bfloat16, device=self.device)
        for i, layer in enumerate(self.model.model.layers):
            layer.self_attn.attn.k_cache = self.kv_cache[0, i]
            layer.self_attn.attn.v_cache = self.kv_cache[1, i]

    # ---- batch -> tensors -----------------------------------------------------
    def _h2d(self, values, dtype):
        return torch.tensor(values, dtype=dtype, pin_memory=True).to(self.device, non_blocking=True)

    def _to_device(self, *arrays: np.ndarray) -> list[torch.Tensor]:
        """The arrays on the device, sent as one pinned buffer in one copy (a copy costs the host and the stream a few
        microseconds however small it is).  torch's pinned pool keeps the buffer until the copy has run."""
        offsets, size = [], 0
        for a in arrays:
            offsets.append(size)
            size += (a.nbytes + 15) & ~15
        host = torch.empty(max(size, 16), dtype=torch.uint8, pin_memory=True)
        raw = host.numpy()
        for a, off in zip(arrays, offsets):
            raw[off:off + a.nbytes] = a.reshape(-1).view(np.uint8)
        dev = host.to(self.device, non_blocking=True)
        return [dev[off:off + a.nbytes].view(_TORCH_DTYPE[a.dtype]).view(a.shape) for a, off in zip(arrays, offsets)]

    def _block_tables(self, seqs: list[Seq]) -> np.ndarray:
        width = max(len(s.block_table) for s in seqs)
        tables = np.full((len(seqs), width), -1, dtype=np.int32)
        for row, s in zip(tables, seqs):
            row[:len(s.block_table)] = s.block_table
        return tables

    def prepare_prefill(self, seqs: list[Seq], num_new: list[int] | None = None):
        """Tokens [num_cached, num_cached + new) of each sequence are computed;
        their K/V go to the slots their block table assigns (reference :129-170)."""
        bs = self.block_size
        starts = [s.num_cached_tokens for s in seqs]
        ends = [len(s) if num_new is None else a + num_new[i] for i, (s, a) in enumerate(zip(seqs, starts))]
        news = [b - a for a, b in zip(starts, ends)]
        total = sum(news)
        ids, pos = np.empty(total, dtype=np.int64), np.empty(total, dtype=np.int64)
        slots = np.empty(total, dtype=np.int32)
        used, at = 0, 0  # tokens with a slot, tokens so far
        for s, a, b, n in zip(seqs, starts, ends, news):
            ids[at:at + n] = s.token_ids[a:b]
            pos[at:at + n] = p = np.arange(a, b)
            if s.block_table:
                slots[used:used + n] = np.asarray(s.block_table, dtype=np.int32)[p // bs] * bs + p % bs
                used += n
            at += n
        cu_q, cu_k = np.zeros(len(seqs) + 1, dtype=np.int32), np.zeros(len(seqs) + 1, dtype=np.int32)
        np.cumsum(news, out=cu_q[1:])
        np.cumsum(ends, out=cu_k[1:])
        arrays = [ids, pos, cu_q, cu_k, cu_q[1:] - 1, slots[:used]]
        if cu_k[-1] > cu_q[-1]:
            arrays.append(self._block_tables(seqs))
        ids_t, pos_t, cu_q_t, cu_k_t, last_t, slots_t, *tables_t = self._to_device(*arrays)
        set_context(True, cu_q_t, cu_k_t, max(news), max(ends), slots_t if used else None, None, tables_t[0] if tables_t else None,
                    last_token_index=last_t)
        return ids_t, pos_t

    def prepare_decode(self, seqs: list[Seq]):
        """One new token per sequence: the last one of its list (reference :172-188)."""
        bs = self.block_size
        lens = [len(s) for s in seqs]
        ids_t, pos_t, slots_t, lens_t, tables_t = self._to_device(
            np.array([s.token_ids[-1] for s in seqs], dtype=np.int64), np.array([n - 1 for n in lens], dtype=np.int64),
            np.array([s.block_table[(n - 1) // bs] * bs + (n - 1) % bs for s, n in zip(seqs, lens)], dtype=np.int32),
            np.array(lens, dtype=np.int32), self._block_tables(seqs))
        set_context(False, slot_mapping=slots_t, context_lens=lens_t, block_tables=tables_t)
        return ids_t, pos_t

    # ---- forward ---------------------------------------------------------------
    @torch.inference_mode()
    def run_model(self, input_ids: torch.Tensor, positions: torch.Tensor, is_prefill: bool):
        return self.model.compute_logits(self.run_hidden(input_ids, positions, is_prefill))

    def run_hidden(self, input_ids: torch.Tensor, positions: torch.Tensor, is_prefill: bool):
        """The model forward up to the final norm (eager for prefill, a graph replay for decode)."""
        from ..utils.context import get_context
        n = input_ids.size(0)
        if is_prefill or self.enforce_eager or n > self.graph_bs[-1]:
            return self.model(input_ids, positions)
        ctx = get_context()
        bs = next(b for b in self.graph_bs if b >= n)
        gv = self.graph_vars
        gv["input_ids"][:n] = input_ids
        gv["positions"][:n] = positions
        gv["slot_mapping"].fill_(-1)  # padded rows store nothing
        gv["slot_mapping"][:n] = ctx.slot_mapping
        gv["context_lens"].zero_()
        gv["context_lens"][:n] = ctx.context_lens
        gv["block_tables"][:n, :ctx.block_tables.size(1)] = ctx.block_tables
        self._bt_rows = {}  # the graph's table no longer matches what _decode_graph_step last staged
        self.graphs[bs].replay()
        return gv["outputs"][:n]

    def _decode_staging(self):
        """Pinned host mirrors of the graphs' input buffers, allocated once: a decode step fills them with
        numpy and issues one asynchronous copy for all the per-row inputs straight into the graph's inputs (no per-step
        pinned allocations, no device-to-device staging copies)."""
        if getattr(self, "_stage", None) is None:
            gv = self.graph_vars
            self._stage = torch.zeros(gv["rows"].shape, dtype=torch.uint8, pin_memory=True)
            self._stage_tables = torch.zeros(gv["block_tables"].shape, dtype=torch.int32, pin_memory=True)
            self._stage_np = {k: v.numpy() for k, v in _row_inputs(self._stage).items()}
            self._stage_np["block_tables"] = self._stage_tables.numpy()
            self._bt_rows = {}  # row of the staged block table -> the blocks last copied into the graph's table for it
        return self._stage_np

    @torch.inference_mode()
    def _decode_graph_step(self, seqs: list[Seq], temperatures: list[float] | None):
        """prepare_decode + the graph replay of run_model in one go, for batches a captured graph covers.  Returns the
        hidden rows and the temperatures on the device (None for greedy decoding)."""
        n = len(seqs)
        bs = next(b for b in self.graph_bs if b >= n)
        np_ = self._decode_staging()
        blk = self.block_size
        lens = [len(s) for s in seqs]
        np_["input_ids"][:n] = [s.token_ids[-1] for s in seqs]
        np_["positions"][:n] = [l - 1 for l in lens]
        np_["context_lens"][:n] = lens
        np_["context_lens"][n:bs] = 0          # padded rows attend to nothing ...
        np_["slot_mapping"][:n] = [s.block_table[(l - 1) // blk] * blk + (l - 1) % blk for s, l in zip(seqs, lens)]
        np_["slot_mapping"][n:bs] = -1         # ... and store nothing
        if temperatures is not None:
            np_["temperatures"][:n] = temperatures
        # block tables change only when a sequence takes a new block (every 256 tokens) or the batch changes: rows are
        # rewritten, and the table copied, only then
        bt = np_["block_tables"]
        rows = self._bt_rows
        width, dirty = 0, False
        for i, s in enumerate(seqs):
            t = s.block_table
            width = max(width, len(t))
            if rows.get(i) != t:
                bt[i, :len(t)] = t
                rows[i] = list(t)
                dirty = True
        gv = self.graph_vars
        gv["rows"].copy_(self._stage, non_blocking=True)
        if dirty:
            gv["block_tables"][:n, :width].copy_(self._stage_tables[:n, :width], non_blocking=True)
        self.graphs[bs].replay()
        set_context(False)  # the LM head only needs to know this is not a prefill step
        return gv["outputs"][:n], gv["temperatures"][:n] if temperatures is not None else None

    @torch.inference_mode()
    def step(self, seqs: list[Seq], is_prefill: bool, temperatures: list[float] | None = None, num_new: list[int] | None = None):
        """One forward pass + sampling on rank 0; the chosen token ids are
        returned on every rank.  temperatures=None means greedy (argmax)."""
        if not is_prefill and not self.enforce_eager and len(seqs) <= self.graph_bs[-1]:
            hidden, temps = self._decode_graph_step(seqs, temperatures)
        else:
            ids, pos = self.prepare_prefill(seqs, num_new) if is_prefill else self.prepare_decode(seqs)
            hidden = self.run_hidden(ids, pos, is_prefill)
            temps = None if temperatures is None else self._h2d(temperatures, torch.float32)
        if getattr(self, "_picked", None) is None or self._picked.numel() < len(seqs):
            self._picked = torch.zeros(max(len(seqs), self.max_num_seqs), dtype=torch.int64, device=self.device)
        picked = self._picked[:len(seqs)]  # one buffer for every step: rank 0's sampler fills it, the broadcast hands it to the others
        if self.fused_sampler and (len(seqs) <= FUSED_SAMPLER_MAX_ROWS or self.world == 1):
            # (several ranks exchange once per call, so they take one call or the unfused path)
            for i in range(0, len(seqs), FUSED_SAMPLER_MAX_ROWS):
                rows = slice(i, i + FUSED_SAMPLER_MAX_ROWS)
                self.model.sample_tokens(hidden, None if temps is None else temps[rows], self.sample_seed, out=picked[rows], rows=rows)
        else:
            logits = self.model.compute_logits(hidden)
            if self.rank == 0:
                picked = Sampler.greedy(logits) if temps is None else self.sampler(logits, temps)
        if self.world > 1:
            from .. import ops
            ops.broadcast_tokens(picked)  # rank 0's choice reaches every rank on the device
        tokens = picked.tolist()  # the step's synchronisation point
        reset_context()
        self.runtime.check_status()
        return tokens

    # ---- CUDA graphs (reference :222-257) -----------------------------------------
    @torch.inference_mode()
    def _capture_graphs(self):
        c = self.config
        max_bs = min(self.max_num_seqs, 512)
        max_blocks = (self.max_model_len + self.block_size - 1) // self.block_size
        dev = self.device
        rows = torch.zeros(max_bs * _ROW_INPUT_BYTES, dtype=torch.uint8, device=dev)
        gv = dict(
            rows=rows,  # the per-row inputs below, side by side: one copy fills them all
            **_row_inputs(rows),
            block_tables=torch.zeros(max_bs, max_blocks, dtype=torch.int32, device=dev),
            outputs=torch.zeros(max_bs, c.hidden_size, dtype=torch.bfloat16, device=dev),
        )
        gv["slot_mapping"].fill_(-1)
        self.graph_bs = [b for b in (1, 2, 4, 8) if b <= max_bs] + list(range(16, max_bs + 1, 16))
        self.graph_pool = None
        for bs in reversed(self.graph_bs):
            graph = torch.cuda.CUDAGraph()
            set_context(False, slot_mapping=gv["slot_mapping"][:bs], context_lens=gv["context_lens"][:bs], block_tables=gv["block_tables"][:bs])
            gv["outputs"][:bs] = self.model(gv["input_ids"][:bs], gv["positions"][:bs])  # warm-up (also runs the collectives once)
            with torch.cuda.graph(graph, self.graph_pool):
                gv["outputs"][:bs] = self.model(gv["input_ids"][:bs], gv["positions"][:bs])
            if self.graph_pool is None:
                self.graph_pool = graph.pool()
            self.graphs[bs] = graph
            torch.cuda.synchronize()
            reset_context()
        self.graph_vars = gv


class ResidentDecoder:
    """Decode steps that never leave the device: one CUDA graph holds the model
    forward, the LM head with its gather, the greedy pick on rank 0, the token
    broadcast to the other ranks and the computation of the next step's inputs
    (what nanovllm/engine/model_runner.py:172-188 and :195-212 do with a host
    round trip every step).  `load(seqs)` puts a batch on the device;
    `replay()` advances every sequence by one token."""

    @torch.inference_mode()
    def __init__(self, runner: ModelRunner, batch: int):
        from .. import ops
        assert not runner.enforce_eager and batch in runner.graphs, "batch must be one of the captured decode batch sizes"
        self.r, self.bs, self.ops = runner, batch, ops
        self.tokens = torch.zeros(batch, dtype=torch.int64, device=runner.device)
        gv = runner.graph_vars
        gv["slot_mapping"].fill_(-1)
        gv["context_lens"].zero_()
        before = ops._abi.launch_count()
        self._body()  # warm-up: also creates the logits view outside the capture
        self.kernels_per_step = ops._abi.launch_count() - before
        gv["slot_mapping"].fill_(-1)
        gv["context_lens"].zero_()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph, runner.graph_pool):
            self._body()
        torch.cuda.synchronize()
        self.replays_left = 0  # nothing loaded yet

    @torch.inference_mode()
    def _body(self):
        r, bs, gv = self.r, self.bs, self.r.graph_vars
        set_context(False, slot_mapping=gv["slot_mapping"][:bs], context_lens=gv["context_lens"][:bs], block_tables=gv["block_tables"][:bs])
        hidden = r.model(gv["input_ids"][:bs], gv["positions"][:bs])
        if r.fused_sampler and bs <= FUSED_SAMPLER_MAX_ROWS:
            r.model.sample_tokens(hidden, None, r.sample_seed, out=self.tokens)  # greedy: rank 0 gets the picks
        else:
            logits = r.model.compute_logits(hidden)
            if r.rank == 0:
                self.ops.argmax(logits, self.tokens)
        if r.world > 1:
            self.ops.broadcast_tokens(self.tokens)
        self.ops.advance_decode(self.tokens, gv["input_ids"], gv["positions"], gv["context_lens"], gv["slot_mapping"],
                                gv["block_tables"][:bs], r.block_size, r.num_kvcache_blocks * r.block_size)
        reset_context()

    @torch.inference_mode()
    def load(self, seqs: list[Seq]) -> None:
        """The batch's state as prepare_decode would build it for the next step."""
        r, gv, n = self.r, self.r.graph_vars, len(seqs)
        assert n == self.bs
        bs = r.block_size
        width = max(len(s.block_table) for s in seqs)
        assert width <= gv["block_tables"].shape[1], "a block table is longer than max_model_len allows"
        assert all(len(s) <= len(s.block_table) * bs for s in seqs), "a sequence is longer than its block table"
        gv["input_ids"][:n] = r._h2d([s.token_ids[-1] for s in seqs], torch.int64)
        gv["positions"][:n] = r._h2d([len(s) - 1 for s in seqs], torch.int64)
        gv["context_lens"][:n] = r._h2d([len(s) for s in seqs], torch.int32)
        gv["slot_mapping"][:n] = r._h2d([s.block_table[(len(s) - 1) // bs] * bs + (len(s) - 1) % bs for s in seqs], torch.int32)
        r._bt_rows = {}  # the graph's table is rewritten here: _decode_graph_step must stage its rows again
        gv["block_tables"][:n].fill_(-1)  # columns past a sequence's own blocks: no room (the advance kernel freezes such a row)
        gv["block_tables"][:n, :width] = r._h2d([s.block_table + [-1] * (width - len(s.block_table)) for s in seqs], torch.int32)
        # replays until the first sequence has filled its last block: each replay stores the K/V of one more position
        self.replays_left = min(len(s.block_table) * bs - len(s) for s in seqs) + 1

    def replay(self) -> None:
        if self.replays_left <= 0:
            raise RuntimeError("ResidentDecoder.replay: a sequence has filled the blocks it was loaded with; load() a batch with more blocks")
        self.replays_left -= 1
        self.graph.replay()


def sequential_block_tables(lengths: list[int], block_size: int, first_block: int = 0, permutation: list[int] | None = None) -> list[list[int]]:
    """Block tables for sequences of the given (maximum) lengths, taking blocks
    in order from `first_block`, or from `permutation` (a shuffled free list)."""
    tables, nxt = [], first_block
    for n in lengths:
        need = (n + block_size - 1) // block_size
        ids = list(range(nxt, nxt + need))
        if permutation is not None:
            ids = [permutation[i] for i in ids]
        tables.append(ids)
        nxt += need
    return tables
