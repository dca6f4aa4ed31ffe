"""Mixers that carry a fixed-size state from token to token instead of keys and values."""

from __future__ import annotations

import torch

import numpy as np

from ..kernels import api as K
from ..tracing import scope
from .base import LayerCache, Mixer, StateNeed, StepContext, StepShape, as_rows, register_part
from .conv import ResidualShortConv
from .linear import linear


class InputConvMixer(Mixer):
    """Base of mixers whose input may first pass a short convolution (``input_conv``): they take the normed rows
    unrounded, and the convolution's state is the first of their states."""

    needs_f32_input = True
    input_conv: ResidualShortConv | None = None

    def own_state_needs(self) -> tuple:
        return ()

    def state_needs(self) -> tuple:
        conv = self.input_conv.state_need() if self.input_conv is not None else None
        return (() if conv is None else (conv,)) + tuple(self.own_state_needs())

    def sub_parts(self):
        return () if self.input_conv is None else (self.input_conv,)

    def read_input(self, ctx: StepContext, h32: torch.Tensor, cache: LayerCache):
        """(rows in the activations' type, the mixer's own state slabs)."""
        states = cache.states
        if self.input_conv is None:
            return h32.to(ctx.runtime.dtype), states
        if self.input_conv.state_need() is None:
            return self.input_conv.forward(ctx, h32, None), states
        return self.input_conv.forward(ctx, h32, states[0]), states[1:]


SEGMENT_TOKENS = 256  # tokens of a long portion that one block of the recurrence kernel walks


def plan_scan_segments(shape: StepShape) -> dict:
    """The step planner of the recurrences: when a request brings a long portion (at least two segments), the step's
    tokens cut into segments of SEGMENT_TOKENS, int32 [n, 4] = (request, first row, end row, flags: 1 = the request's
    first segment, 2 = the request has several).  A recurrence over time gives the GPU only its state's parallelism;
    segments scanned at once from a zero state, and corrected afterwards, multiply it by their number.  Steps of short
    portions and single tokens get no list (their tokens are walked in order, one block per request and head)."""
    if max(shape.q_lens) < 2 * SEGMENT_TOKENS:
        return {}
    segs, n0 = [], 0
    for r, T in enumerate(shape.q_lens):
        if T >= 2 * SEGMENT_TOKENS:
            for c in range(0, T, SEGMENT_TOKENS):
                segs.append((r, n0 + c, n0 + min(T, c + SEGMENT_TOKENS), (1 if c == 0 else 0) | 2))
        else:
            segs.append((r, n0, n0 + T, 1))
        n0 += T
    return {"scan_segments": np.array(segs, dtype=np.int32).reshape(-1, 4)}


# Portions of at least so many tokens may go through the chunk kernels (three launches of 50 us together at 16 heads, then
# 65 ns per token; the walk: 145 ns per token and no start).  Measured, us, walk and chunks: 16 heads 256 tokens 46 and 50,
# 512 tokens 81 and 52, 2048 tokens 297 and 144; 32 heads 512 tokens 108 and 81; 8 requests of 256 tokens, 32 heads, 288 and 290.
CHUNK_FROM_TOKENS = 384
# When they take the decayed recurrences' portions:
# * Two launches more and their arguments are 20 us of the host's time, which such a layer is bound by at few tokens, and requests
#   beside the portions are walked all the same.  So the portions must be worth CHUNK_WORK heads x tokens, or CHUNK_LEAD tokens; beside
#   others, what the longest is ahead of them counts.  A layer's pass, us, walk and chunks: 16 heads 400 tokens (retention, gated, time
#   mixing) 121 and 138, 153 and 164, 215 and 224; 768 tokens 167 and 140, 184 and 166, 216 and 224; 1024 tokens 216 and 141, 233 and
#   168, 249 and 225; 640 beside 360 tokens 196 and 215, 213 and 231, 236 and 253; 32 heads 400 tokens 208 and 161, 229 and 180, 221 and 223.
# * The chunk kernels work on 128 x 128 whatever a head's sizes, the walk on what there is, over more heads and requests at once: from
#   heads of CHUNK_AREA on chunks are ahead at any number of them (112 x 112, 8 to 64 heads, 1 to 16 requests of 384 to 2048
#   tokens: 0.32 to 1.02 of the walk's time); smaller ones take them for portions worth CHUNK_WORK_SMALL and up to CHUNK_CHAINS heads
#   of the longest (72 x 72 and 96 x 96, 8 to 32 heads: 0.29 to 0.98; 32 heads, 384 tokens 1.03 to 1.07); beyond, 72 x 72 took 0.97 to
#   1.73 of the walk's time at 2 to 16 requests of 32 to 64 heads, and 96 x 96 0.87 to 1.31.
CHUNK_WORK, CHUNK_LEAD = 12288, 1024
CHUNK_AREA, CHUNK_WORK_SMALL, CHUNK_CHAINS = 112 * 112, 16384, 32


def plan_scan_chunks(shape: StepShape) -> dict:
    """The step planner of the decayed recurrences: when a request brings a long portion, its tokens in chunks of
    ``K.CHUNK_TOKENS``: ``scan_chunks`` int32 [n, 3] = (request, first row, end row) and ``scan_chunk_requests`` [m, 3] =
    (request, its first chunk, its chunks).  Shorter portions and single tokens are walked in order."""
    if max(shape.q_lens) < CHUNK_FROM_TOKENS:
        return {}
    chunks, requests, n0 = [], [], 0
    for r, T in enumerate(shape.q_lens):
        if T >= CHUNK_FROM_TOKENS:
            requests.append((r, len(chunks), -(-T // K.CHUNK_TOKENS)))
            chunks += [(r, n0 + c, n0 + min(T, c + K.CHUNK_TOKENS)) for c in range(0, T, K.CHUNK_TOKENS)]
        n0 += T
    return {"scan_chunks": np.array(chunks, dtype=np.int32).reshape(-1, 3), "scan_chunk_requests": np.array(requests, dtype=np.int32).reshape(-1, 3)}


def step_chunks(ctx: StepContext) -> "K.Chunks | None":
    """The step's long portions in chunks, if it has any (and was planned with ``plan_scan_chunks``)."""
    chunks = ctx.arrays.get("scan_chunks")
    if chunks is None:
        return None
    requests = ctx.arrays["scan_chunk_requests"]
    m = requests.numel() // 3
    return K.Chunks(chunks, requests, chunks.numel() // 3, m, CHUNK_FROM_TOKENS, m < ctx.n_requests)


def decay_chunks_pay(lens, heads: int, dk: int, dv: int) -> bool:
    """Whether a step's long portions go through the chunk kernels rather than the decayed recurrences' walk (see CHUNK_WORK)."""
    long, rest = [n for n in lens if n >= CHUNK_FROM_TOKENS], max((n for n in lens if n < CHUNK_FROM_TOKENS), default=0)
    lead = max(long) - rest
    small = dk * dv < CHUNK_AREA
    if lead < CHUNK_LEAD and heads * (lead if rest else sum(long)) < (CHUNK_WORK_SMALL if small else CHUNK_WORK):
        return False
    return not small or heads * sum(long) <= CHUNK_CHAINS * max(long)


def scan_chunks(ctx: StepContext, heads: int, dk: int, dv: int, pays=None) -> "tuple[K.Chunks | None, torch.Tensor | None]":
    """The step's chunks and the scratch of their states, if it has long portions of heads that the chunk kernels take, and if
    ``pays(lengths, heads, dk, dv)`` says so."""
    if "scan_chunks" not in ctx.arrays or not K.chunk_scan_supported(dk, dv) or (pays is not None and not pays(ctx.host_q_lens, heads, dk, dv)):
        return None, None
    chunks = step_chunks(ctx)
    need = K.chunk_scan_scratch(chunks.n, heads, dk, dv)
    return chunks, ctx.workspace.get("chunk_scan", need, torch.float32) if ctx.workspace is not None else \
        torch.empty(need, dtype=torch.float32, device=chunks.chunks.device)


class HGRN2(InputConvMixer):
    """Gated linear recurrence with a matrix state per head, whose forget gate f doubles as the write gate 1 - f
    (keys do not exist in this form):  q = silu(W_q h), v = W_v h, f = lower + (1 - lower) * sigmoid(W_f h + b_f);
    S_t = diag(f_t) S_(t-1) + (1 - f_t) v_t^T;  o_t = S_t^T q_t;  each head's o is RMS-normed over its value size with
    one weight shared by the heads, and the heads go through W_o.  Gates, state and norm are float32.

    ``w_qfv``: [2 H dk + H dv, D], the q, f and v projections stacked in that order."""

    kernel_libraries = ("recurrent", "chunk_scan", "gemm_simt")
    kernel_libraries_bf16 = ("gemm_stream",)

    def __init__(self, w_qfv: torch.Tensor, f_bias: torch.Tensor, lower: torch.Tensor, norm_weight: torch.Tensor,
                 w_o: torch.Tensor, heads: int, dim: int, vdim: int, eps: float, input_conv: ResidualShortConv | None = None):
        if w_qfv.shape[0] != heads * (2 * dim + vdim) or w_o.shape[1] != heads * vdim or f_bias.numel() != heads * dim \
                or lower.numel() != heads * dim or norm_weight.numel() != vdim:
            raise ValueError(f"HGRN2 weights do not fit {heads} heads of {dim} x {vdim}: qfv {tuple(w_qfv.shape)}, o {tuple(w_o.shape)}")
        self.w_qfv, self.w_o = w_qfv, w_o
        self.f_bias, self.lower = f_bias.to(torch.float32).contiguous(), lower.to(torch.float32).contiguous()
        self.norm_weight = norm_weight.to(torch.float32).contiguous()
        self.heads, self.dim, self.vdim, self.eps = heads, dim, vdim, float(eps)
        self.input_conv = input_conv

    def own_state_needs(self):
        return (StateNeed((self.heads, self.dim, self.vdim), torch.float32),)

    def step_planners(self):
        return (plan_scan_chunks,) if K.chunk_scan_supported(self.dim, self.vdim) else (plan_scan_segments,)

    def forward(self, ctx: StepContext, h, cache: LayerCache, h32: torch.Tensor | None = None):
        a, (state,) = self.read_input(ctx, h32, cache)
        with scope("qkv_matmul"):
            qfv = as_rows(linear(ctx, a, self.w_qfv, torch.float32, partials=True))
        o = torch.empty((a.shape[0], self.heads * self.vdim), dtype=ctx.runtime.dtype, device=a.device)
        with scope("attention"):
            chunks, chunk_scratch = scan_chunks(ctx, self.heads, self.dim, self.vdim)
            segs = ctx.arrays.get("scan_segments") if chunks is None else None
            n_seg = 0 if segs is None else segs.numel() // 4
            need = K.hgrn2_scan_scratch(a.shape[0], self.heads, self.dim, self.vdim, n_seg)
            scratch = ctx.workspace.get("hgrn2_scan", need, torch.float32) if ctx.workspace else None
            K.hgrn2_scan(qfv.data, qfv.splits, self.f_bias, self.lower, state, ctx.cu_q, ctx.slot_ids, self.norm_weight,
                         self.eps, o, self.heads, self.dim, self.vdim, scratch, segs if n_seg else None, n_seg, SEGMENT_TOKENS, chunks, chunk_scratch)
        with scope("projection"):
            return linear(ctx, o, self.w_o, torch.float32, partials=True)


register_part("mixer", "hgrn2", HGRN2)
