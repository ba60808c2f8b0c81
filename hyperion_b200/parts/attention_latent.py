"""Attention whose keys and values are made from one small latent per token.

A token leaves one record in the cache: its latent c (``kv_rank`` entries, RMS-normed with a weight per entry) and one rotated
key part (``rot_dim`` entries) that all heads share.  Per head h, key = [K_h c | rotated part], value = V_h c, and queries come
through a latent of their own: c_q = norm(D_q x), q = U_q c_q, laid out head by head as [``head_dim`` unrotated | ``rot_dim`` rotated].

    score_h(i, j) = (q_h,plain(i) . K_h c_j + q_h,rot(i) . k_rot(j)) * scale,  causal softmax (optionally with a sink per head:
    one more term exp(sink_h) in the denominator), out_h = sum_j p_ij V_h c_j, then the output projection.

Nothing per head is ever cached or rebuilt from the cache.  Since q . (K_h c) = (K_h^T q) . c, the query is carried into the
latent's space once per token and head (a batched product with K_h), attention then runs as if there were ONE key/value head
whose keys are the cached records and whose values are the records' first ``kv_rank`` entries, and the result is carried out of
the latent's space by a batched product with V_h.  Norms, angles, scores and softmax are float.

Per step: one product for both down-projections (kept in float); one kernel that norms the latents, rotates the shared key part
and writes the record to its page (``csrc/heads_prepare.cu``); the queries' up-projection; the batched product with K_h; one
kernel that puts the query of every head together (rotating its rotated part); attention; the batched product with V_h; the
output projection.  In bfloat16, with records of a multiple of 16 entries and latents of a multiple of 8, attention runs on the
tensor cores (``csrc/attention_latent.cu``: blocks of 16, 32 or 64 (token, head) pairs over key tiles of 64 records, the keys split over
several blocks when a step brings few tokens).  Everything else, and float32, runs in ``csrc/attention_generic.cu``.

A step of nothing but prompts from position 0 on, long enough, takes the other way round (``_attend_expanded``): every key and value a query sees is a token of the step, so
the keys and values of all heads are made from the latents by one product, and attention runs over ordinary heads of ``head_dim`` + ``rot_dim`` entries: some third
of the operations per pair of a query and a key (1,531 tokens of 16 heads: 40 us a layer in csrc/attention_tcgen05.cu beside 225).  The records go to the cache all the same.
Keys and values per head are then rounded to bfloat16 where the other way rounds the carried query and the weighted latents, so in bfloat16 a prompt's last bits depend on which way its step
took: on whether it came from position 0 in one piece, and on what else was in the step.  The distance from 64 bits is the other way's to a few per cent (36 prompts of 400 to 1,531
tokens, 3 to 16 heads: 0.97 to 1.06 of it, 1.01 on average).  Float32 always goes through the latent.

Parameters: ``hidden_size``, ``heads``, ``head_dim``, ``rot_dim``, ``value_dim``, ``kv_rank``, ``q_rank``, ``scale``, ``position`` (a PartSpec
of kind ``rope_interleaved``, or None), ``sink`` (bool), ``eps``.  Tensors: dq, dq.norm, uq, dkv, dkv.norm, uk, uv, sink, o.
"""
from __future__ import annotations

from typing import Mapping

import numpy as np
import torch

from .. import ops
from ..ops import attention as fast_attention
from .attention_sloped import LARGEST_HEAD
from .base import POSITIONS, BuildContext, Mixer, PagedTokens, WeightSpec, make, register_mixer
from .spec import PartSpec


def _common_dtype(tensors) -> torch.dtype:
    return torch.float32 if any(t.dtype == torch.float32 for t in tensors) else tensors[0].dtype


EXPANDED_TOKENS = 300  # of a step, per prompt.  What the other way saves grows with the square of a prompt, what it adds (one product more, its keys and values written out) with
# the step's tokens.  A step of 8 layers, 4 of them over latents of 16 heads, expanded and through the latent, in us: one prompt of 200 tokens 872 and 844, two of 256 1,074 and
# 1,060, five of 300 1,342 and 1,421, three of 400 1,355 and 1,475, one of 1,024 1,622 and 1,906, one of 1,531 2,238 and 2,919; four of 128 999 and 927.
# More heads meet earlier: a step of one layer, the host's planning among it, expanded over latent with 16, 32 and 64 heads: 512 tokens 1.04, 0.97, 0.83; four prompts of 300 1.02, 0.92, 0.78.
EXPANDED_BYTES = 480 << 20  # of what a layer of such a step makes beside its queries: pages, the product that fills them, the dense latents (16 heads of 128 + 64: 21.6 KB a token, where the
# queries carried into the latent and what comes back of it are 66 KB).  Longer prompts keep to the latent.
EXPANDED_PAGE = 64


class LatentAttention(Mixer):
    def __init__(self, spec: PartSpec, build: BuildContext):
        super().__init__(spec, build)
        p = spec.params
        self.hidden, self.heads = int(p["hidden_size"]), int(p["heads"])
        self.head_dim, self.rot_dim, self.value_dim = int(p["head_dim"]), int(p["rot_dim"]), int(p["value_dim"])
        self.kv_rank, self.q_rank = int(p["kv_rank"]), int(p["q_rank"])
        self.scale, self.eps = float(p["scale"]), float(p["eps"])
        self.has_sink = bool(p.get("sink", False))
        self.position = make(POSITIONS, p["position"], build) if p.get("position") is not None else None
        if self.position is not None and not hasattr(self.position, "inv_freq"):
            raise ValueError("this attention rotates adjacent pairs: its position encoding must offer frequencies ('rope_interleaved')")
        self.rot_dims = self.position.dims if self.position is not None else 0
        if self.rot_dims > self.rot_dim:
            raise ValueError(f"a rotation of {self.rot_dims} dimensions in a part of {self.rot_dim}")
        self.record = self.kv_rank + self.rot_dim
        if self.record > LARGEST_HEAD:
            raise ValueError(f"a record of {self.record} entries per token is above the kernel's limit of {LARGEST_HEAD}")
        self.q_head = self.head_dim + self.rot_dim
        self.fast = self.dtype == torch.bfloat16 and fast_attention.latent_supported(self.record, self.kv_rank)
        # heads that the tcgen05 attention takes
        self.expands_fresh_prompts = (self.fast and self.q_head == fast_attention.WIDE_KEYS and self.value_dim == 128 and self.kv_rank % 8 == 0
                                      and not any(n % 8 for n in (self.head_dim, self.rot_dim, self.rot_dims)))

    def weights(self) -> dict[str, WeightSpec]:
        wanted = {"dq": WeightSpec((self.q_rank, self.hidden)), "dq.norm": WeightSpec((self.q_rank,), init="one_plus_normal"),
                  "uq": WeightSpec((self.heads * self.q_head, self.q_rank)), "dkv": WeightSpec((self.record, self.hidden)),
                  "dkv.norm": WeightSpec((self.kv_rank,), init="one_plus_normal"), "uk": WeightSpec((self.heads * self.head_dim, self.kv_rank)),
                  "uv": WeightSpec((self.heads * self.value_dim, self.kv_rank)), "o": WeightSpec((self.hidden, self.heads * self.value_dim))}
        if self.has_sink:
            wanted["sink"] = WeightSpec((self.heads,))
        return wanted

    def load(self, tensors: Mapping[str, torch.Tensor]) -> None:
        down = [tensors["dq"], tensors["dkv"]]
        dtype = _common_dtype(down)
        self.w_down = torch.cat([m.to(dtype) for m in down], dim=0).contiguous()
        self.w_uq, self.w_o = tensors["uq"].contiguous(), tensors["o"].contiguous()
        self.q_norm = tensors["dq.norm"].to(torch.float32).contiguous()
        self.kv_norm = tensors["dkv.norm"].to(torch.float32).contiguous()
        self.k_heads = tensors["uk"].reshape(self.heads, self.head_dim, self.kv_rank).contiguous()  # q_plain [H, T, d] x this = the query in the latent's space
        self.v_heads = tensors["uv"].reshape(self.heads, self.value_dim, self.kv_rank).transpose(1, 2).contiguous()  # [H, R, e]
        self.sink = tensors["sink"].to(torch.float32).contiguous() if self.has_sink else None
        self.w_kv = torch.cat([tensors["uk"], tensors["uv"]], dim=0).contiguous() if self.expands_fresh_prompts else None  # every head's keys, then every head's values
        if self.w_kv is not None and self.w_kv.dtype == self.k_heads.dtype:  # the keys' half is what stands above, once is enough (the values' lie the other way round)
            self.k_heads = self.w_kv[: self.heads * self.head_dim].view(self.heads, self.head_dim, self.kv_rank)

    def cache_request(self):
        return PagedTokens((1,), (self.record,), 0)

    def kernel_modules(self):
        modules = [("heads_prepare", {}), ("attention_generic", {}), ("sgemm_f32", {}) if self.dtype == torch.float32 else ("gemm_tcgen05", {})]
        if self.fast:
            modules.append(("attention_latent", {"HB_RECORD": self.record, "HB_VALUE": self.kv_rank}))
        if self.expands_fresh_prompts:
            modules.append(("attention_tcgen05", {"HB_HEAD_DIM": 128, "HB_KEY_DIM": fast_attention.WIDE_KEYS}))
        return modules

    def step_plans(self):
        """Pages of the step's own for the keys and values of its prompts, and the prompts cut into tiles, where the step takes :meth:`_attend_expanded`."""
        if not self.expands_fresh_prompts:
            return {}

        def plan(rows, packer, host):
            counts = rows.counts
            pages = -(-counts // EXPANDED_PAGE)
            total = int(pages.sum())
            if (rows.positions.any() or int(counts.min()) <= fast_attention.TOKEN_SHAPE_MAX or int(counts.sum()) < EXPANDED_TOKENS * len(counts)
                    or self._expanded_bytes(total * EXPANDED_PAGE, int(counts.sum())) > EXPANDED_BYTES):
                return
            table = np.full((len(counts), int(pages.max())), -1, dtype=np.int32)
            ends = np.cumsum(pages)
            for row, (end, n) in enumerate(zip(ends.tolist(), pages.tolist())):
                table[row, :n] = np.arange(end - n, end)
            tiles, _ = fast_attention.plan_prompts(rows, fast_attention.TC_TILE_ROWS, self.heads, 2 / 3)  # whole prompts: their tiles differ in length
            host[self._expanded_key()] = (total, len(tiles) // 3)
            packer.add(f"{self._expanded_key()}_table", table.reshape(-1), table.shape)
            packer.add(f"{self._expanded_key()}_tiles", tiles)

        plan.tells_fresh_prompts = True  # the runner keeps graphs of such steps apart
        return {("latent_plan", self._expanded_key()): plan}

    def _expanded_bytes(self, slots: int, tokens: int) -> int:
        return 2 * (slots * 2 * self.heads * self.q_head + tokens * (self.heads * (self.head_dim + self.value_dim) + self.record))

    def _expanded_key(self) -> str:
        return f"latent_{self.heads}_{self.q_head}"

    def _attend_expanded(self, cq, latent, part, step, inv_freq):
        """[tokens, heads * value_dim]: attention of the step's prompts over their own keys and values."""
        key = self._expanded_key()
        pages, n_tiles = step.host[key]
        tokens = cq.shape[0]
        q = ops.project(cq, self.w_uq, None, self.dtype)
        kv = ops.project(latent, self.w_kv, None, self.dtype)
        storage = torch.empty((pages, 2, self.heads, EXPANDED_PAGE, self.q_head), dtype=self.dtype, device=cq.device)
        table = step.extra[f"{key}_table"]
        ops.latent_expand_(q, kv, part, self.heads, self.head_dim, self.value_dim, inv_freq, self.rot_dims, step.positions, step.token_row, table, storage,
                           settled=True)
        out = torch.empty((tokens, self.heads * self.value_dim), dtype=self.dtype, device=cq.device)
        fast_attention.attention_wide_keys(q, self.heads, storage, table, step.token_row, step.positions, step.extra[f"{key}_tiles"], n_tiles, self.scale, out, sinks=self.sink)
        return out

    @staticmethod
    def _batched(a: torch.Tensor, b: torch.Tensor, out_dtype: torch.dtype) -> torch.Tensor:
        if a.dtype == torch.float32 or out_dtype == a.dtype:
            return torch.bmm(a, b)
        return torch.bmm(a, b, out_dtype=out_dtype)

    def forward(self, x, step, cache, own_cache):
        if cache is None or not own_cache:
            raise ValueError("this attention writes a paged cache of its own; the schedule gave it none")
        tokens = x.shape[0]
        inv_freq = self.position.inv_freq if self.position is not None else None
        proj = ops.project(x, self.w_down, None, torch.float32)
        expands = self.expands_fresh_prompts and self._expanded_key() in step.host
        latent = torch.empty((tokens, self.kv_rank), dtype=self.dtype, device=x.device) if expands else None
        part = torch.empty((tokens, self.rot_dim), dtype=self.dtype, device=x.device) if expands else None
        cq = ops.latent_prepare(proj, 0, self.q_rank, self.q_rank, self.kv_rank, self.rot_dim, self.q_norm, self.kv_norm, self.eps, inv_freq, self.rot_dims,
                                step.positions, self.dtype, cache.kv, cache.block_table, step.token_row, cache.page_size, latent, part)
        if expands:
            return ops.project(self._attend_expanded(cq, latent, part, step, inv_freq), self.w_o, None, self.dtype, may_leave_partials=True)  # the result is a residual delta
        q = ops.project(cq, self.w_uq, None, self.dtype)
        plain = q.view(tokens, self.heads, self.q_head)[:, :, : self.head_dim].transpose(0, 1)
        q_lat = self._batched(plain, self.k_heads.to(q.dtype) if self.k_heads.dtype != q.dtype else self.k_heads, torch.float32)
        query = ops.latent_query(q, q_lat, self.heads, self.head_dim, self.rot_dim, inv_freq, self.rot_dims, step.positions)
        if self.fast:
            # a step replayed from a CUDA graph fixes its launch shape for every context its tables can hold
            longest = step.host.get("context_cap") or step.rows.longest_context
            attn = fast_attention.attention_latent(query, self.heads, self.record, self.kv_rank, cache.kv, cache.block_table, step.row_start, step.positions,
                                                   len(step.rows), int(step.rows.counts.max()), int(longest), self.scale, sinks=self.sink)
        else:
            attn = ops.attention_general(query, self.heads, 1, self.record, self.kv_rank, cache.kv, cache.block_table, step.token_row, step.positions,
                                         cache.page_size, self.scale, sinks=self.sink, value_prefix=True)
        core = torch.empty((tokens, self.heads, self.value_dim), dtype=self.dtype, device=x.device)
        v_heads = self.v_heads.to(attn.dtype) if self.v_heads.dtype != attn.dtype else self.v_heads
        torch.bmm(attn.view(tokens, self.heads, self.kv_rank).transpose(0, 1), v_heads, out=core.transpose(0, 1))
        return ops.project(core.view(tokens, self.heads * self.value_dim), self.w_o, None, self.dtype, may_leave_partials=True)  # the result is a residual delta


register_mixer("latent_attention", LatentAttention)
