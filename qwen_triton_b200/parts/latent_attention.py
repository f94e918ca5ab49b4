"""Softmax attention through a latent: per token the cache holds one normed latent vector and one rotated key part that
all heads share, and every head expands its keys and values from the latent with matrices of its own.

From the mixer's input h: the query latent c_q = rms(W_dq h) w_q and q = W_uq c_q, laid out head by head as
[``head_dim`` plain | ``rot_dim`` rotated] (without ``q_rank`` there is no query latent: q = W_q h, rows of the first projection);
W_dkv h = [``kv_rank`` | ``rot_dim``] rows, of which the first, RMS-normed with a
weight, are the latent c and the last, rotated by the position encoding, the key part k_r shared by the heads.  Head h has
k_h = W_uk_h c and v_h = W_uv_h c; its score is (q_plain_h . k_h + q_rot_h . k_r) * ``scale``, causal, over all earlier keys or
the last ``window`` of them, plain softmax; the concatenated heads are multiplied by sigmoid(W_g h) (``gate`` true: one number
per element; "head": one per head; false: none) and projected by W_o.  Only c and k_r are cached, under a window in a ring.

What runs: since q_plain_h . (W_uk_h c) = (W_uk_h^T q_plain_h) . c, every head's query becomes
[W_uk_h^T q_plain_h | q_rot_h] (a product per head, ``kernels.head_product``) and the attention kernels run all heads
against the one cached row [c | k_r] per token, with the row's first ``kv_rank`` elements as values; the head's output is
W_uv_h (sum_j p_j c_j), a second product per head, in whose epilogue the gate is applied.  Keys and values are never
expanded per token, in prompts or in one-token steps.

A layer with ``own_kv`` false has no W_dkv: it reads the cache rows of the schedule position named by ``LayerCall.cache_of``
(which must have the same ``kv_rank``, ``rot_dim`` and rotation) under its own W_uk, W_uv, queries and everything else.

A rotation of neighbouring pairs (2i, 2i + 1) becomes one of (i, i + dims / 2) when the weights are loaded: the rotated rows of the
query's and of the shared key part's matrices are put in that order, which changes no score.

Norms, rotation (float cos/sin table), scores, softmax and the gate are float; the query latent, the queries, the cache
rows and the heads' outputs are rounded to the activation type between the products (in a prompt that forms keys and values per head, queries,
keys and values to halves with a power of two per query and per 64 tokens, which keep more bits over the same range).

Parameters: ``hidden_size``, ``num_heads``, ``head_dim``, ``rot_dim``, ``v_head_dim``, ``q_rank``, ``kv_rank``, ``scale``, ``eps``,
``position`` (a position part over ``rot_dim``; either pairing), ``window``, ``own_kv``, ``gate``, ``float_out``, and the tensor-name pieces ``dq``, ``uq``
(or ``q``), ``dkv``, ``uk``, ``uv``, ``g``, ``o``, ``weight_suffix``, ``norm_suffix``.
"""
from __future__ import annotations

import torch

from ..ops import kernels
from ..weights.tensors import TensorSpec
from .attention import _MAX_SPLIT_PAIRS, _MIN_KEYS_PER_SPLIT
from .base import DeferredProduct, KVRequest, Runtime, part_class, register_mixer, to_device
from .linear import Linear


_EXPAND_TOKENS = 64      # longest portion from which a prompt may form keys and values per head
_MANY_TOKENS = 256       # steps of more tokens form the queries and the cache rows in products of their own (without a query latent)


def own_keys_pay(heads: int, d: int, rot: int, dv: int, rank: int, window: int | None, longest: int, n_seqs: int, tokens: int) -> bool:
    """Whether keys and values of every head's own take less time than the latent rows in a step of prompts, the longest of ``longest`` tokens (64
    and more; the others are taken as equal).  Over latent rows a query and key cost 2 rank + rot multiplications and a head and token rank (d + dv)
    in products per head; over its own keys a third of the former, at the price of three more kernels, a product over every run of 64
    rows, and blocks for every sequence and head.  Microseconds over rows / over its own, all products of the layer in: 16 heads of 128 + 64
    over rows of 512 + 64: 2,048 tokens 519 / 166, 400 122 / 98, 64 59 / 59, 32 x 64 214 / 167, 8 x 64 91 / 93, 64 beside 31 x 3 63 / 99, beside 31 x 17
    107 / 122; 128 such heads: 1,000 tokens 1,261 / 435, 64 beside 31 x 3 162 / 485; 8 heads of 64 + 32 over 256 + 32: 2,048 tokens 174 / 94, 64 32 / 41; 16
    heads of 128 + 64 over 64 + 64: 2,048 tokens 227 / 143, 400 76 / 89, 32 x 64 115 / 142.  The factors are fitted to 210 such pairs, of which ten
    take the slower form by more than 3 % (by 18 % at most)."""
    if longest < _EXPAND_TOKENS:
        return False
    rest = (tokens - longest) / (n_seqs - 1) if n_seqs > 1 else 0.0
    pairs = longest * min(longest, 2 * (window or longest)) + (tokens - longest) * min(rest, 2 * (window or longest))
    key = 128 if d + rot <= 128 else 192
    saved = 3.0e-9 * heads * pairs * (2 * rank + rot) + 2.2e-8 * heads * tokens * rank * (d + dv) + 3.0e-5 * longest * (2 * rank + rot) + 0.01 * longest + 4.7e-4 * heads * tokens
    spent = 9.6 + 4.5e-9 * heads * 64 * (tokens // 64 + n_seqs) * (key + dv) * (rank + rot) + 0.032 * heads * n_seqs
    return saved > spent


@register_mixer("latent_attention")
class LatentAttention:
    graph_safe = True

    def __init__(self, params, prefix: str, runtime: Runtime) -> None:
        self.prefix, self.runtime, self.params = prefix, runtime, params
        self.hidden = int(params["hidden_size"])
        self.heads, self.d, self.rot, self.dv = (int(params[k]) for k in ("num_heads", "head_dim", "rot_dim", "v_head_dim"))
        self.q_rank, self.rank = int(params.get("q_rank") or 0), int(params["kv_rank"])      # q_rank 0: no query latent
        self.row = self.rank + self.rot                        # one cached row, and one head's query as the kernels see it
        if self.row > 640 or self.rank > 512:
            raise ValueError(f"{prefix}: a latent of {self.rank} + {self.rot} elements is beyond what the attention kernels take (512 + 128)")
        self.scale = float(params["scale"])
        self.eps = float(params.get("eps", 1e-6))
        self.own_kv = bool(params.get("own_kv", True))
        self.gated = bool(params.get("gate", True))
        self.head_gate = params.get("gate") == "head"
        self.window = int(params["window"]) if params.get("window") else None
        position_spec = params["position"]
        self.position = part_class("position", position_spec)(position_spec.params, runtime)
        self.interleaved = bool(getattr(self.position, "interleaved", False))
        self.cos_sin = None
        self.at_kv = self.q_rank or self.heads * (self.d + self.rot)
        self.at_gate = self.at_kv + (self.row if self.own_kv else 0)
        used = self.at_gate + (self.heads * (1 if self.head_gate else self.dv) if self.gated else 0)
        self.proj_rows = -(-used // 8) * 8
        self.proj = Linear("latent.proj" + ("" if self.own_kv else ".reader"), self.proj_rows, self.hidden, runtime, float_out=True, role="qkv")
        self.takes_scaled_rows = self.proj.fused_capable
        # Many tokens without a query latent: the queries are most of the first product's columns, and what reads them rounds them to
        # the activation type anyway, so they are a product of their own that hands them on in it (over the same weight rows).
        self.many = None
        if not self.q_rank and runtime.dtype == torch.bfloat16 and self.hidden % 8 == 0 and runtime.max_step_tokens > _MANY_TOKENS and self.proj_rows > self.at_kv:
            self.many = (Linear("latent.queries", self.at_kv, self.hidden, runtime),
                         Linear("latent.rows", self.proj_rows - self.at_kv, self.hidden, runtime, float_out=True))
            # whole over K, or it would hand on float planes after all
            self.many[0].split_plans = [(rows, splits) for rows, splits in self.many[0].split_plans if rows <= _MANY_TOKENS]
        self.uq = Linear("latent.uq", self.heads * (self.d + self.rot), self.q_rank, runtime) if self.q_rank else None
        float_out = bool(params.get("float_out", False))
        self.o = Linear("latent.o" + (".float" if float_out else ""), self.hidden, self.heads * self.dv, runtime, float_out=float_out, role="attn_out")
        ws = runtime.workspace
        tokens = runtime.max_step_tokens
        if self.q_rank:
            ws.declare("latent.cq", tokens * self.q_rank, runtime.dtype)
        ws.declare("latent.heads", tokens * self.heads * self.dv, runtime.dtype)
        ws.declare("attn.part_acc", _MAX_SPLIT_PAIRS * self.heads * self.rank, torch.float32)
        ws.declare("attn.part_ml", _MAX_SPLIT_PAIRS * self.heads * 2, torch.float32)
        # Prompts from position 0 on form every head's keys and values from the cached rows in one product and run over those (forward)
        turning = getattr(self.position, "rotary_dim", 0)
        self.key = 128 if self.d + self.rot <= 128 else 192                     # a head's query and key there, filled up with zeros
        self.expands = (runtime.dtype == torch.bfloat16 and runtime.page_tokens == 64 and self.d + self.rot <= 192 and self.dv in (64, 128) and self.scale > 0
                        and self.d % 8 == 0 and self.rot % 8 == 0 and turning % 16 == 0 and self.row % 8 == 0 and self.at_kv % 8 == 0)
        self.most_runs = tokens // 64 + min(64, tokens // 32)      # of sequences of 32 tokens and more on average: fewer do not pay
        # queries and results of the form over latent rows; a step takes one form, so the other's queries, keys and values lie there too
        ws.declare("latent.q", tokens * self.heads * (max(self.row, self.key) if self.expands else self.row), runtime.dtype)
        ws.declare("latent.ctx", max(tokens * self.heads * self.rank, 64 * self.most_runs * self.heads * (self.key + self.dv) if self.expands else 0), runtime.dtype)
        if self.expands:
            ws.declare("latent.rows", 64 * self.most_runs * self.row, runtime.dtype)
            ws.declare("latent.run_scale", 4 * self.most_runs, torch.float32)
            ws.declare("latent.query_scale", tokens * self.heads, torch.float32)
        self.q_norm = self.kv_norm = self.uk_t = self.uv = self.expand = None
        self.key_norm = self.value_norm = 0.0                  # the largest sum of magnitudes over a row of W_uk, of W_uv (and 1 %)

    # ------------------------------------------------------------------ weights
    @staticmethod
    def _names(params, prefix: str) -> dict[str, str]:
        w, nw = str(params.get("weight_suffix", ".weight")), str(params.get("norm_suffix", ".norm"))
        n = {key: f"{prefix}.{params.get(key, key)}{w}" for key in ("dq", "uq", "q", "dkv", "uk", "uv", "g", "o")}
        n["dq_norm"], n["dkv_norm"] = f"{prefix}.{params.get('dq', 'dq')}{nw}", f"{prefix}.{params.get('dkv', 'dkv')}{nw}"
        return n

    @classmethod
    def expected_tensors(cls, params, prefix: str) -> dict[str, TensorSpec]:
        hidden, heads, d, rot, dv = (int(params[k]) for k in ("hidden_size", "num_heads", "head_dim", "rot_dim", "v_head_dim"))
        q_rank, rank = int(params.get("q_rank") or 0), int(params["kv_rank"])
        n = cls._names(params, prefix)
        std = float(params.get("init_std", 0.02))
        if q_rank:
            out = {n["dq"]: TensorSpec((q_rank, hidden), init_std=std), n["dq_norm"]: TensorSpec((q_rank,), role="vector", init_std=0.1, init_mean=1.0),
                   n["uq"]: TensorSpec((heads * (d + rot), q_rank), init_std=std)}
        else:
            out = {n["q"]: TensorSpec((heads * (d + rot), hidden), init_std=std)}
        out |= {n["uk"]: TensorSpec((heads * d, rank), init_std=std),
               n["uv"]: TensorSpec((heads * dv, rank), init_std=std), n["o"]: TensorSpec((hidden, heads * dv), init_std=std)}
        if params.get("gate", True):
            out[n["g"]] = TensorSpec((heads * (1 if params.get("gate") == "head" else dv), hidden), init_std=std)
        if params.get("own_kv", True):
            out[n["dkv"]] = TensorSpec((rank + rot, hidden), init_std=std)
            out[n["dkv_norm"]] = TensorSpec((rank,), role="vector", init_std=0.1, init_mean=1.0)
        return out

    def _halves_order(self, weight: torch.Tensor, groups: int, plain: int) -> torch.Tensor:
        """Rows stored as ``groups`` of [plain | rotated], the rotated ones of neighbouring pairs put in the order of a rotation of
        halves: the even ones of the turning elements first, then the odd ones."""
        if not self.interleaved:
            return weight
        turning = self.position.rotary_dim
        place = torch.arange(plain + self.rot)
        place[plain:plain + turning] = plain + torch.cat((torch.arange(0, turning, 2), torch.arange(1, turning, 2)))
        return weight.view(groups, plain + self.rot, weight.shape[1])[:, place.to(weight.device)].reshape(weight.shape)

    def load(self, source) -> None:
        n = self._names(self.params, self.prefix)
        dtype, device = self.runtime.dtype, self.runtime.device
        rows = [source(n["dq"]).to(dtype) if self.q_rank else self._halves_order(source(n["q"]), self.heads, self.d).to(dtype)]
        if self.own_kv:
            rows.append(self._halves_order(source(n["dkv"]), 1, self.rank).to(dtype))
        if self.gated:
            rows.append(source(n["g"]).to(dtype))
        used = sum(r.shape[0] for r in rows)
        if self.proj_rows > used:
            rows.append(torch.zeros(self.proj_rows - used, self.hidden, dtype=dtype, device=rows[0].device))
        self.proj.set_weight(torch.cat(rows, dim=0))
        if self.many is not None:
            self.many[0].weight, self.many[1].weight = self.proj.weight[:self.at_kv], self.proj.weight[self.at_kv:]
        if self.q_rank:
            self.uq.set_weight(self._halves_order(source(n["uq"]), self.heads, self.d))
            self.q_norm = to_device(source(n["dq_norm"]), torch.float32, device)
        self.o.set_weight(source(n["o"]))
        if self.own_kv:
            self.kv_norm = to_device(source(n["dkv_norm"]), torch.float32, device)
        # W_uk per head, transposed: [heads, kv_rank, head_dim], the matrix of the product that carries a head's plain
        # query part into the latent's space; W_uv is stored as that product's matrix already: [heads, v_head_dim, kv_rank]
        self.uk_t = to_device(source(n["uk"]).view(self.heads, self.d, self.rank).transpose(1, 2), dtype, device)
        self.uv = to_device(source(n["uv"]).view(self.heads, self.dv, self.rank), dtype, device)
        if self.expands:
            # [heads * key | heads * dv, row]: W_uk of a head on the latent, ones that hand its shared rotated part on, zero rows; then W_uv
            expand = torch.zeros(self.heads * (self.key + self.dv), self.row, dtype=dtype, device=device)
            keys = expand[:self.heads * self.key].view(self.heads, self.key, self.row)
            keys[:, :self.d, :self.rank] = self.uk_t.transpose(1, 2)
            keys[:, self.d:self.d + self.rot, self.rank:] = torch.eye(self.rot, dtype=dtype, device=device)
            expand[self.heads * self.key:].view(self.heads, self.dv, self.row)[:, :, :self.rank] = self.uv
            self.expand = expand
            self.key_norm, self.value_norm = (1.01 * float(w.float().abs().sum(dim=dim).max()) for w, dim in ((self.uk_t, 1), (self.uv, 2)))
        tables = self.runtime.options.setdefault("position_tables", {})
        key = self.position.key() + (self.runtime.max_positions,)
        if key not in tables:
            tables[key] = self.position.table(self.runtime.max_positions)
        self.cos_sin = tables[key]

    # ------------------------------------------------------------------ what it keeps per sequence
    def cache_request(self):
        return KVRequest(1, self.row, self.window, shared_values=True)

    def _splits(self, ctx, page_tokens: int) -> int:
        """Partial results per (sequence, head) of a one-token step.  The tensor-core kernel runs one block per SM, each
        with up to 64 heads of a sequence and a range of its pages; with at most 16 (32) heads a block cuts the keys of
        every page into 4 (2) parts, each a partial result of its own.  The generic kernel runs four heads a block,
        several blocks per SM."""
        keys = min(ctx.max_context, self.window) if self.window else ctx.max_context
        if kernels.attention_latent_shape(self.runtime.dtype, self.row, self.rank, page_tokens) and self.scale > 0:
            parts = 4 if self.heads <= 16 else 2 if self.heads <= 32 else 1
            if parts * ctx.n_seqs > _MAX_SPLIT_PAIRS:
                parts = 1
            blocks = ctx.n_seqs * -(-self.heads // 64)
            most = max(1, min(keys // _MIN_KEYS_PER_SPLIT, _MAX_SPLIT_PAIRS // (ctx.n_seqs * parts), 32))
            return parts * max(1, min(most, self.runtime.sm_count // max(blocks, 1)))
        blocks = ctx.n_seqs * -(-self.heads // 4)
        most = max(1, min(keys // _MIN_KEYS_PER_SPLIT, _MAX_SPLIT_PAIRS // ctx.n_seqs, 32))
        return max(1, min(most, (2 * self.runtime.sm_count) // max(blocks, 1)))

    # ------------------------------------------------------------------ run
    def _expands_for(self, ctx, tokens: int) -> bool:
        """Whether a step forms keys and values per head: where all its sequences start at position 0, the scratch holds their runs and it
        pays."""
        return (self.expands and getattr(ctx, "from_start", False) and not ctx.is_decode and tokens // 64 + ctx.n_seqs <= self.most_runs
                and own_keys_pay(self.heads, self.d, self.rot, self.dv, self.rank, self.window, ctx.max_q_len, ctx.n_seqs, tokens))

    def _over_own_keys(self, q_full, gate, gate_offset: int, ctx, cache, table):
        """[T, heads, dv]: attention over every head's own keys and values, made from the cached rows."""
        ws, tokens = self.runtime.workspace, q_full.rows
        count = kernels.rows_of_runs(tokens, ctx.n_seqs)
        rows = ws.view("latent.rows", count, self.row)
        run_scale = ws.view("latent.run_scale", count // 64, 4)
        kernels.latent_rows(cache.k, rows, run_scale, self.rank, self.key_norm, self.value_norm, table, ctx.seq_start, ctx.n_seqs, ctx.max_q_len, cache.page_tokens, cache.ring_tokens)
        keys_values = ws.view("latent.ctx", count, self.heads * (self.key + self.dv), dtype=torch.float16)
        kernels.keys_and_values(rows, self.expand, keys_values, self.heads * self.key, run_scale)
        q, q_scale = ws.view("latent.q", tokens, self.heads, self.key, dtype=torch.float16), ws.view("latent.query_scale", tokens, self.heads)
        kernels.latent_queries(q_full, self.cos_sin, ctx.token_pos, q, q_scale, self.d, self.rot)
        out = ws.view("latent.heads", tokens, self.heads, self.dv)
        kernels.attention_prefill_rows(q, q_scale, keys_values, run_scale, out, ctx.seq_start, ctx.n_seqs, ctx.max_q_len, self.window, self.scale,
                                       gate=gate, gate_offset=gate_offset, gate_per_head=self.head_gate)
        return out

    def forward(self, x, ctx, cache):
        tokens = x.shape[0]
        ws = self.runtime.workspace
        write = cache.writable and self.own_kv
        if cache.k is None or cache.k.shape[-1] != self.row:
            raise ValueError(f"{self.prefix}: the cache rows it reads are not {self.rank} + {self.rot} elements long")
        table = ctx.block_table(cache.group)
        own_queries = self.many is not None and tokens > _MANY_TOKENS
        skipped = self.at_kv if own_queries else 0                              # columns that ``proj`` then lacks
        proj = self.many[1](x) if own_queries else self.proj.finished(x)
        cq = ws.view("latent.cq", tokens, self.q_rank) if self.q_rank else None
        if cq is not None or write:
            kernels.latent_prepare(proj, self.q_norm, self.kv_norm, self.eps, self.cos_sin, cq, cache.k if write else None, ctx.token_seq,
                                   ctx.token_pos, table if write else None, self.rank, self.rot, cache.page_tokens, cache.ring_tokens, write_kv=write,
                                   at_kv=self.at_kv - skipped)
        # [*, T, heads * (d + rot)], or with the first projection's other columns behind
        q_full = self.uq(cq) if cq is not None else self.many[0](x) if own_queries else proj
        if self._expands_for(ctx, tokens):
            heads = self._over_own_keys(q_full, proj if self.gated else None, self.at_gate - skipped, ctx, cache, table).view(tokens, self.heads * self.dv)
            return DeferredProduct(self.o, heads) if self.o.fusable(tokens) else self.o(heads)
        q = ws.view("latent.q", tokens, self.heads, self.row)
        kernels.head_product(q_full, self.uk_t, q, x_row=q_full.cols, x_head=self.d + self.rot)
        kernels.latent_query_rot(q_full, self.cos_sin, ctx.token_pos, q, self.heads, self.d, self.rot, self.rank)
        out = ws.view("latent.ctx", tokens, self.heads, self.rank)
        if ctx.is_decode:
            kernels.attention_decode(q, cache.k, cache.k, out, table, ctx.seq_len, 1, cache.page_tokens, cache.ring_tokens, self.window, self.scale,
                                     self._splits(ctx, cache.page_tokens), ws.view("attn.part_acc", _MAX_SPLIT_PAIRS * self.heads * self.rank),
                                     ws.view("attn.part_ml", _MAX_SPLIT_PAIRS * self.heads * 2), v_dim=self.rank)
        else:
            kernels.attention_prefill(q, cache.k, cache.k, out, table, ctx.seq_start, ctx.seq_past, ctx.max_q_len, 1, cache.page_tokens,
                                      cache.ring_tokens, self.window, self.scale, v_dim=self.rank)
        heads = ws.view("latent.heads", tokens, self.heads, self.dv)
        kernels.head_product(out, self.uv, heads, x_row=self.heads * self.rank, x_head=self.rank,
                             gate=proj if self.gated else None, gate_offset=self.at_gate - skipped, gate_per_head=self.head_gate)
        heads = heads.view(tokens, self.heads * self.dv)
        # few tokens: the product is left to the block, whose next norm launches it with the residual addition in its epilogue
        return DeferredProduct(self.o, heads) if self.o.fusable(tokens) else self.o(heads)
