"""Gated linear attention: a recurrence over a float32 state per sequence instead of keys and values.

Per head, with q and k of ``head_dim`` channels and v of ``value_dim``:

    S_t = diag(alpha_t) S_(t-1) + k_t v_t^T,    o_t = S_t^T (q_t * q_scale)
    alpha_t = sigmoid(z_t)^(1/tau),              z_t = A2 (A1 x_t) + b        (one decay per key channel)

then each head's o_t is divided by its root mean square over ``value_dim`` and multiplied by one weight vector
shared by the heads, the heads side by side are multiplied by silu(G x_t), and the output projection follows.
The state starts at zero (the cache zeroes a slot's state when it hands the slot out) and is carried from step
to step in the cache line's state area, which holds two copies per slot so that a step of one token reads one
and writes the other (see gla.cu).  q, k, v, the gate and A1 x come from one product; everything between that
product and the output projection is one kernel in float32 for single tokens, three for a prompt, whose tokens run in
chunks as matrix products (gla_chunks.cu) or, at other sizes, are cut into segments that run side by side (gla.cu).
"""
from __future__ import annotations

from typing import Optional

import torch

from ..cache import CacheNeed, LineView
from ..csrc import ops
from ..weights.loader import MATRIX, VECTOR, TensorNeed, TensorSource
from .base import Mixer, register_part
from .linear import part_linear


# From this many tokens of the longest prompt on a step may run in chunks as matrix products (gla_chunks.cu).  Measured on a B200, the
# kernels alone, microseconds, token by token | in chunks: 16 heads of 128 x 128, one prompt of 64 tokens 103 | 62, of 1,024 tokens
# 329 | 87, 16 prompts of 65 tokens 128 | 143, of 130 tokens 257 | 213, one of 128 tokens beside 63 of five 273 | 265; 16 heads of 64 x 64,
# 16 of 65 tokens 90 | 79, of 130 tokens 162 | 114; 64 heads of 64 x 64, one of 128 beside 63 of five 329 | 436; 64 heads of 128 x 64, 64 of 128
# tokens 2841 | 1490.
CHUNKED_TOKENS = 64
SEGMENT_TOKENS = 128        # other sizes: a long prompt's tokens run in segments of this many, side by side (see gla.cu)


class GatedLinearAttention(Mixer):
    replayable = True
    kernel_groups = ("common", "streams", "recurrent")

    def __init__(self, spec, dtype):
        super().__init__(spec, dtype)
        a = spec.args
        self.hidden_size = int(a["hidden_size"])
        self.num_heads = int(a["num_heads"])
        self.head_dim = int(a["head_dim"])
        self.value_dim = int(a.get("value_dim") or self.head_dim)
        self.decay_rank = int(a["decay_rank"])
        self.tau = float(a["tau"])
        self.q_scale = float(a.get("q_scale", self.head_dim ** -0.5))
        self.norm_eps = float(a.get("norm_eps", 1e-6))
        if min(self.num_heads, self.head_dim, self.value_dim, self.decay_rank) < 1:
            raise ValueError("gated linear attention needs heads, head_dim, value_dim and decay_rank of at least 1")
        if not self.tau > 0.0:
            raise ValueError(f"a decay exponent 1/tau with tau = {self.tau}")
        self.qk_width = self.num_heads * self.head_dim
        self.v_width = self.num_heads * self.value_dim
        # rows of the joint projection: q | k | v | gate | decay's inner rows
        self.offsets = (0, self.qk_width, 2 * self.qk_width, 2 * self.qk_width + self.v_width,
                        2 * self.qk_width + 2 * self.v_width)
        self.w_in: Optional[torch.Tensor] = None
        self.w_decay: Optional[torch.Tensor] = None
        self.decay_bias: Optional[torch.Tensor] = None
        self.norm_weight: Optional[torch.Tensor] = None
        self.w_o: Optional[torch.Tensor] = None

    def _needs(self) -> dict[str, TensorNeed]:
        d = self.hidden_size
        return {
            "q_proj": TensorNeed(self.name_of("q_proj"), (self.qk_width, d), MATRIX, "normal"),
            "k_proj": TensorNeed(self.name_of("k_proj"), (self.qk_width, d), MATRIX, "normal"),
            "v_proj": TensorNeed(self.name_of("v_proj"), (self.v_width, d), MATRIX, "normal"),
            "gate_proj": TensorNeed(self.name_of("gate_proj"), (self.v_width, d), MATRIX, "normal"),
            "decay_in": TensorNeed(self.name_of("decay_in"), (self.decay_rank, d), MATRIX, "normal"),
            "decay_out": TensorNeed(self.name_of("decay_out"), (self.qk_width, self.decay_rank), MATRIX, "normal"),
            "decay_bias": TensorNeed(self.name_of("decay_bias"), (self.qk_width,), VECTOR, "bias"),
            "out_norm": TensorNeed(self.name_of("out_norm"), (self.value_dim,), VECTOR, "around_one"),
            "o_proj": TensorNeed(self.name_of("o_proj"), (d, self.v_width), MATRIX, "normal"),
        }

    def tensor_needs(self):
        return list(self._needs().values())

    def load(self, source: TensorSource) -> None:
        needs = self._needs()
        self.w_in = torch.cat([source.fetch(needs[n]) for n in ("q_proj", "k_proj", "v_proj", "gate_proj", "decay_in")],
                              dim=0).contiguous()
        self.w_decay = source.fetch(needs["decay_out"])
        self.decay_bias = source.fetch(needs["decay_bias"])
        self.norm_weight = source.fetch(needs["out_norm"])
        self.w_o = source.fetch(needs["o_proj"])

    def cache_need(self) -> CacheNeed:
        return CacheNeed(state_shape=(2, self.num_heads, self.head_dim, self.value_dim), state_dtype="float32")

    def chunks_pay(self, ctx) -> bool:
        """Whether a step of prompts is faster in chunks: microseconds of both ways, fitted to 144 steps of eight head counts and sizes
        (the measurements above among them; no step of them is slower this way than token by token)."""
        if ctx.is_decode or ctx.max_q_len < CHUNKED_TOKENS:
            return False
        size = self.head_dim * self.value_dim / 2 ** 14                     # as a share of 128 x 128
        tokens = ctx.num_tokens * self.num_heads
        serial = max((1.26 + 0.35 * size) * ctx.max_q_len, (0.0042 + 0.0036 * size) * tokens)
        items = ctx.chunk_count(ops.GLA_CHUNK_TOKENS) * self.num_heads
        return ops.chunks_pay(max(39 + 24 * size, 23 + (0.05 + 0.19 * size) * items + 0.00056 * tokens), serial)

    def forward(self, ctx, act: torch.Tensor, line: LineView, writes_cache: bool) -> torch.Tensor:
        if not writes_cache:
            raise ValueError("a recurrent layer cannot read another layer's state: it has to write its own")
        proj = part_linear(act, self.w_in)                                  # float32 [T, 2 qk + 2 v + rank]
        out = ctx.buffer("linear_attention.out", (act.shape[0], self.v_width), self.dtype)
        sizes = dict(heads=self.num_heads, dim=self.head_dim, vdim=self.value_dim, tau=self.tau, q_scale=self.q_scale, eps=self.norm_eps)
        args = (proj, self.offsets, self.w_decay, self.decay_bias, self.norm_weight, line.state, ctx.seq_slot, ctx.seq_start, ctx.cu_q_len, out)
        if self.chunks_pay(ctx) and ops.gla_chunks_take(self.head_dim, self.value_dim, self.decay_rank, proj.shape[1], self.offsets):
            chunks = ctx.token_chunks(ops.GLA_CHUNK_TOKENS)
            floats = ops.gla_chunks_scratch_floats(chunks[0].numel(), act.shape[0], self.num_heads, self.head_dim, self.value_dim)
            ops.gla_chunks(*args, chunks=chunks, scratch=ctx.buffer("linear_attention.segments", (floats,), torch.float32), **sizes)
            return part_linear(out, self.w_o)
        segments = scratch = None
        # a long prompt whose heads give the device fewer than two blocks an SM
        if (not ctx.is_decode and ctx.max_q_len >= 2 * SEGMENT_TOKENS
                and ctx.num_seqs * self.num_heads < 2 * ops.sm_count(ctx.device)):
            segments = ctx.token_chunks(SEGMENT_TOKENS)
            floats = ops.gla_scratch_floats(segments[0].numel(), self.num_heads, self.head_dim, self.value_dim)
            scratch = ctx.buffer("linear_attention.segments", (floats,), torch.float32)
        ops.gla_scan(*args, segments=segments, scratch=scratch, **sizes)
        return part_linear(out, self.w_o)


register_part("mixer", "gated_linear_attention", GatedLinearAttention, replace=True)
