"""Gated linear attention: a recurrent mixer whose state per head is a matrix that decays per key channel.

With H heads, keys and queries of size dim and values of size vdim:

    q = W_q x * dim^-1/2,  k = W_k x,  v = W_v x
    a = sigmoid(W_a2 (W_a1 x) + b)^(1/tau)                      one decay per head and key channel (W_a1 narrow, W_a2 wide)
    S_t = diag(a_t) S_(t-1) + k_t v_t^T;   o_t = S_t^T q_t      S starts at zero
    out = W_o (o / rms(o) per head * w_norm * silu(W_g x))      w_norm [vdim], shared by the heads

The five projections q, k, v, g and W_a1 x are ONE product with float32 results; the wide half of the decays' projection, the
decays (through their logarithm), the state and the output's norm are float32.  A request's state lives in its state slot and is
carried from step to step.  Long segments of a bfloat16 step run the recurrence in chunks on the tensor cores (float32 operands in parts, float32
sums); short ones (decoded tokens among them, whatever stands beside them), float32 and heads the chunks do not take run it token after
token.  All launches depend on the step's counts and device arrays alone.
"""
from __future__ import annotations

import torch

from .. import ops
from ..cache.manager import LayerCacheView, StateSpec
from .base import ChunkRule, Mixer, StepContext, chunked_segments


class GatedLinearAttention(Mixer):
    def __init__(self, hidden: int, num_heads: int, dim: int, vdim: int, tau: float, w_in: torch.Tensor, w_a2: torch.Tensor, a_bias: torch.Tensor,
                 norm_weight: torch.Tensor, w_out: torch.Tensor, eps: float):
        """w_in: W_q | W_k | W_v | W_g | W_a1 stacked by rows ([2 H dim + 2 H vdim + rank, hidden], compute dtype); w_a2 [H dim, rank] and
        a_bias [H dim] (kept in float32); norm_weight [vdim]."""
        H = num_heads
        rank = w_a2.shape[1]
        if w_in.shape != (2 * H * dim + 2 * H * vdim + rank, hidden) or w_out.shape != (hidden, H * vdim) or w_a2.shape != (H * dim, rank):
            raise ValueError("the gated linear attention's weights do not fit the head counts")
        if a_bias.shape != (H * dim,) or norm_weight.shape != (vdim,):
            raise ValueError("the gated linear attention's vectors do not fit the head counts")
        if not tau > 0:
            raise ValueError("the decays' temperature is positive")
        if dim > ops.gla_max_dim():
            raise ValueError(f"keys of {dim} values: the recurrence keeps a column of the state in registers, up to {ops.gla_max_dim()} rows")
        self.hidden, self.H, self.dim, self.vdim, self.tau, self.eps, self.rank = hidden, H, dim, vdim, float(tau), float(eps), rank
        self.w_in, self.w_out = w_in.contiguous(), w_out.contiguous()
        self.a2t = w_a2.to(torch.float32).t().contiguous()          # [rank, H dim]: neighbouring threads read neighbouring channels
        self.a_bias = a_bias.to(torch.float32).contiguous()
        self.norm_weight = norm_weight.to(torch.float32).contiguous()
        # Measured, us a mixer, token after token / in chunks, 4 heads of 64 x 256 and 8 of 128 x 256:  one segment of 288: 64 / 72, 86 / 109; of 352: 80 / 72, 96 / 112; of
        # 448: 84 / 73, 119 / 118;  eight of 100: 65 / 78, 160 / 169;  sixteen of 64: 81 / 83, 184 / 184;  eight of 150: 88 / 82, 210 / 188;  one of 512 beside 32
        # single tokens: 99 / 87, 171 / 212; beside 64: 105 / 108, 198 / 309; of 2,048 beside 64: 426 / 152, 544 / 428.  In chunks
        # with the single ones / those token after token:  512 beside 8: 75 / 95, 131 / 161; 1,024 beside 32: 101 / 124, 253 / 242; beside 64: 122 / 141, 352 / 294; 2,048
        # beside 64: 152 / 159, 428 / 351.
        self.chunk_rule = ChunkRule(320 if dim <= 64 else 432, total=1024, a_single=H * vdim // 256, few=max(1, 4718592 // (H * dim * vdim)))
        self.gate_off = 2 * H * dim + H * vdim
        self.a_off = self.gate_off + H * vdim

    def tensors(self):
        return [self.w_in, self.a2t, self.a_bias, self.norm_weight, self.w_out]

    def cache_spec(self):
        return StateSpec((ops.gla_state_floats(self.H, self.dim, self.vdim),), torch.float32)

    def forward(self, xn: torch.Tensor, ctx: StepContext, cache: LayerCacheView, residual: torch.Tensor, write_cache: bool = True,
                norm=None) -> None:
        if not write_cache:
            raise ValueError("a recurrent mixer has no cache that another run could read")
        T, ws, HV = ctx.num_tokens, ctx.workspace, self.H * self.vdim
        proj = ops.linear(xn, self.w_in, ws.rows("gla.proj", T, self.w_in.shape[0], torch.float32), ops.LINEAR_F32)
        plan = (ctx.chunk_plan(self.chunk_rule) if ctx.dtype == torch.bfloat16 and ops.memory_chunked_takes(proj.shape[1], self.dim, self.vdim, self.rank)
                else None)
        scratch = None if plan is None else ws.flat(f"gla.chunks/{self.H}/{self.dim}/{self.vdim}",
                                                    ops.gla_chunked_scratch_bytes(ws.max_tokens, chunked_segments(ws, self.chunk_rule), self.H, self.dim, self.vdim), torch.uint8)
        out = ops.gla(proj, self.a_off, self.a2t, self.a_bias, self.tau, self.norm_weight, self.eps, ctx, cache.state,
                      ws.rows("gla.decay", T, self.H * self.dim, torch.float32), ws.rows("gla.o", T, HV, torch.float32),
                      ws.rows("gla.out", T, HV, ctx.dtype), self.H, self.dim, self.vdim, self.gate_off, scratch, *(plan or ()))
        ops.linear(out, self.w_out, residual, ops.LINEAR_ACC_F32)
