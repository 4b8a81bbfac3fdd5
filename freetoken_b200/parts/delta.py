"""Gated delta rule: a recurrent mixer whose matrix state is corrected towards each token's value.

One projection of the input gives ``[q | k | v | g | b | a]``: queries and keys for ``n_kv_heads`` heads of
``head_dim``, values and an output gate for ``n_heads`` heads of ``v_head_dim`` (head ``h`` reads q/k head
``h // (n_heads / n_kv_heads)``), and two logits per head.  ``q``, ``k`` and ``v`` pass a short causal convolution
over time per channel (no bias) and ``silu``; ``q`` and ``k`` are then made unit vectors per head,
``x / sqrt(sum(x^2) + 1e-6)``, and ``q`` is multiplied by ``head_dim^-1/2``.  Per token and head::

    beta = sigmoid(b)         g = exp(-exp(A_log) softplus(a + dt_bias))
    S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q

so the read-out sees the token's own write.  Each head's ``o`` is divided by its root mean square, multiplied by
one plain weight ``[v_head_dim]`` for all heads and by ``silu`` (or ``sigmoid``) of the gate, and projected.

With ``decay_rank`` every key channel of a head has a decay of its own, through a low rank: ``a`` is then a row of
``decay_rank`` entries, ``z = W_a2 a``, ``g[d] = exp(-exp(A_log) softplus(z[d] + dt_bias[d]))``, acting on the rows of ``S`` that
belong to key channels.  With ``gate_rank`` the gate's logits are ``W_g2 g``, ``g`` a row of ``gate_rank`` entries.

Unit norms, ``beta``, ``g``, the state and all of the recurrence's sums are 32-bit (:func:`ops.delta_scan`, which
takes the logits and the convolved rows as they lie and runs a request's tokens in order, the state's columns
spread over threads); the output norm and gate are :func:`ops.gated_heads`.  Per request the layer keeps the state
``S`` (stored column by column, ``[n_heads, v_head_dim, head_dim]``) and the convolution's last ``taps - 1`` inputs in one
slot of the cache manager's state pool; both start from zero.  The reference has no recurrent mixer.
"""

from __future__ import annotations

import functools
import math
from typing import Any, Dict, List, Optional, Sequence, Tuple

import torch

from ..config.spec import ParamSpec, PartSpec, StateNeed
from ..errors import ConfigError
from ..kernels import ops
from .base import MIXERS, BuildEnv, Mixer, StepState

CHUNK_MIN_TOKENS = 80  # no request of fewer tokens goes in chunks: see chunks_pay
SMS = 148

UNIT_EPS = 1e-6  # inside the root of the unit norms of q and k: fixed by the design


def token_time(states: float, wide: bool, v_dim: int) -> float:
    """Microseconds a token of the kernel that takes a request's tokens one by one, with ``states`` (request, head) pairs at work."""
    rounds = lambda cols: math.ceil(states * -(-v_dim // cols) / SMS)  # noqa: E731  (blocks of so many value columns an SM)
    if wide and states * v_dim >= 32 * SMS:  # (as csrc/delta.cu: launch_delta)
        return (0.43, 0.61, 1.2)[rounds(64) - 1] if rounds(64) < 4 else 0.305 * rounds(64)
    if wide:
        return 0.27 if rounds(16) == 1 else 0.34
    return 0.26 if rounds(16) <= 2 else max(0.36, 0.086 * rounds(16))


def chunk_time(lens: Sequence[int], n_heads: int, n_kv_heads: int, head_dim: int, v_dim: int) -> float:
    """Microseconds of requests of ``lens`` tokens in chunks (``csrc/delta_chunk.cu``), in one pass."""
    longest = max(lens)
    states = sum(lens) / longest * n_heads  # (request, head) pairs at work, on average
    rounds = lambda cols: math.ceil(states * -(-v_dim // cols) / SMS)  # noqa: E731  (blocks of so many value columns an SM)
    chunks = -(-longest // ops.DELTA_CHUNK)
    large = rounds(64) * (3 + 5 * chunks) < rounds(16) * 3 * chunks  # (blocks of 64 columns: csrc/delta_chunk.cu: launch_delta_chunks)
    chain = rounds(64) * (4.3 + 6.4 * chunks) if large else rounds(16) * 4.2 * chunks
    blocks = sum(lens) / longest * chunks * n_kv_heads * -(-(n_heads // n_kv_heads) // 2)  # (that prepare)
    return 22.4 + chain * (1.0 if head_dim > 64 else 0.88) + 13.7 * max(0.0, blocks / (2 * SMS) - 0.35)


def chunk_passes(lens: Sequence[int], most: int) -> List[Tuple[int, int, int, int, int]]:
    """Requests of ``lens`` tokens in passes of at most ``most`` rows (of 64 tokens): first request and how many, rows from .. to of each of
    them, and how many rows that is.

    All requests side by side, each as far as all of them can, where that is eight rows and more; else whole ones, as many as there are
    rows for, and one that is longer by itself in pieces (a block's start and end, its state from memory and back, take as long as
    two rows).  48 heads on 8 of 128, 64 rows: four requests of 2,048 tokens 747 us in one pass, 789 side by side, 927 as whole ones;
    102 of 80 1,339, 1,745 and 1,389."""
    rows = [-(-n // ops.DELTA_CHUNK) for n in lens]
    out: List[Tuple[int, int, int, int, int]] = []

    def far(left: Sequence[int]) -> int:
        low, high = 0, max(left)
        while low < high:
            m = (low + high + 1) // 2
            low, high = (m, high) if sum(min(r, m) for r in left) <= most else (low, m - 1)
        return low

    if far(rows) >= min(8, max(rows)):
        done = 0
        while any(r > done for r in rows):
            left = [max(r - done, 0) for r in rows]
            step = far(left)
            out.append((0, len(rows), done, done + step, sum(min(r, step) for r in left)))
            done += step
        return out
    first = total = longest = 0
    for i, n in enumerate(rows):
        if total and total + n > most:
            out.append((first, i - first, 0, longest, total))
            total = longest = 0
        if not total:
            first = i
        if n > most:
            out.extend((i, 1, r, min(r + most, n), min(most, n - r)) for r in range(0, n, most))
        else:
            total, longest = total + n, max(longest, n)
    if total:
        out.append((first, len(rows) - first, 0, longest, total))
    return out


def chunks_pay(lens: Sequence[int], beside: bool, n_heads: int, n_kv_heads: int, head_dim: int, v_dim: int, most: Optional[int] = None) -> bool:
    """Whether requests of ``lens`` tokens are through sooner in chunks (``csrc/delta_chunk.cu``) than token by token
    (``csrc/delta.cu``); ``beside``: the step has others, which then take a launch of their own; ``most``: rows of scratch.

    Both kernels are chains (of chunks, of tokens) until a step has more blocks than the GPU holds at once, then waves or a
    rate; the chunks also have a launch that prepares them, two blocks an SM.  Fitted to 620 timings of both (heads of 64 and 128, 4 to 48 of
    them, 1 to 32 requests of 80 to 2,048 tokens, most of at most 192, 16 to 256 value columns): the slower one is named in 27, 0.4 % lost on
    average, a third at most (16 requests of 112 tokens, 48 heads of 64 on 24, 48 columns: 149 and 201).  One request, 48 heads of 128, token
    by token against chunks: 39 and 38 us for 80 tokens, 46 and 32 for 96, 59 and 37 for 128, 213 and 69 for 512; 16 heads of 64: 23
    and 26, 27 and 26, 35 and 31, 127 and 40.  Many requests: 48 heads, 16 of 80 tokens 311 and 222, four of 512 604 and 199; 48 heads
    of 64 columns that share no keys, 16 of 80 160 and 188, of 128 244 and 198."""
    return _chunks_pay(tuple(lens), beside, n_heads, n_kv_heads, head_dim, v_dim, most)  # (a step's layers ask the same)


@functools.lru_cache(maxsize=256)
def _chunks_pay(lens: Tuple[int, ...], beside: bool, n_heads: int, n_kv_heads: int, head_dim: int, v_dim: int, most: Optional[int]) -> bool:
    parts: List[Sequence[int]] = [lens]
    if most is not None and sum(-(-n // ops.DELTA_CHUNK) for n in lens) > most:
        parts = [[max(0, min(n, row1 * ops.DELTA_CHUNK) - row0 * ops.DELTA_CHUNK) for n in lens[first:first + count]]
                 for first, count, row0, row1, _ in chunk_passes(lens, most)]
    in_chunks = sum(chunk_time(p, n_heads, n_kv_heads, head_dim, v_dim) for p in parts) + (6.0 if beside else 0.0)
    longest = max(lens)
    return in_chunks < 8.0 + longest * token_time(sum(lens) / longest * n_heads, head_dim > 64, v_dim)


@MIXERS.register("gated_delta")
class GatedDelta(Mixer):
    """params: ``hidden``, ``n_heads``, ``n_kv_heads``, ``head_dim``, ``v_head_dim``, ``taps``, ``eps`` (of the output
    norm), ``decay_rank`` (None: one decay a head), ``gate_rank`` (None: the gate is projected straight), ``gate`` ("silu" |
    "sigmoid"), ``init_std``."""

    graph_safe = False  # running a step twice would advance the state twice
    graph_recordable = True  # everything a step does is decided on the device

    def __init__(self, spec: PartSpec, env: BuildEnv):
        super().__init__(spec, env)
        g = lambda k: int(spec[k])  # noqa: E731
        self.hidden, self.n_heads, self.head_dim = g("hidden"), g("n_heads"), g("head_dim")
        self.n_kv_heads = int(spec.get("n_kv_heads") or self.n_heads)
        self.v_dim = int(spec.get("v_head_dim") or self.head_dim)
        self.taps = int(spec.get("taps", 4))
        self.eps = float(spec.get("eps", 1e-6))
        if min(self.hidden, self.n_heads, self.n_kv_heads, self.v_dim) < 1 or not 1 <= self.head_dim <= 256:
            raise ConfigError("gated_delta: heads and head sizes must be positive, keys at most 256")
        if self.n_heads % self.n_kv_heads:
            raise ConfigError("gated_delta: n_heads must be a multiple of n_kv_heads")
        if not 1 <= self.taps <= 16:
            raise ConfigError(f"gated_delta: {self.taps} taps (1 to 16 taken)")
        self.decay_rank = None if spec.get("decay_rank") is None else int(spec["decay_rank"])
        self.gate_rank = None if spec.get("gate_rank") is None else int(spec["gate_rank"])
        if any(r is not None and r < 1 for r in (self.decay_rank, self.gate_rank)):
            raise ConfigError("gated_delta: a low rank is positive")
        self.gate = spec.get("gate", "silu")
        if self.gate not in ops.GATE_CODES:
            raise ConfigError(f"gated_delta: unknown gate '{self.gate}'")
        H, G, D, Dv = self.n_heads, self.n_kv_heads, self.head_dim, self.v_dim
        self.k_col = G * D
        self.v_col = 2 * G * D
        self.conv_dim = self.v_col + H * Dv
        self.g_col = self.conv_dim
        self.b_col = self.g_col + (self.gate_rank or H * Dv)
        self.a_col = self.b_col + H
        self.proj_rows = self.a_col + (self.decay_rank or H)
        # scratch of the longest step: its rows, and what one takes
        self.most_rows, size = self.chunk_scratch(env.max_step_tokens, env.max_step_tokens // CHUNK_MIN_TOKENS)
        self.row_bytes = size // max(self.most_rows, 1)

    def param_specs(self) -> Dict[str, ParamSpec]:
        std = self.spec.get("init_std")
        std_in, std_out = (float(std[0]), float(std[1])) if std else (0.02, 0.02)
        H, D, Dv = self.n_heads, self.head_dim, self.v_dim
        f32 = dict(dtype="float32", store="bfloat16")
        out = {
            "in_proj.weight": ParamSpec((self.proj_rows, self.hidden), init=("normal", 0.0, std_in)),
            "conv.weight": ParamSpec((self.conv_dim, self.taps), init=("normal", 0.0, 0.4 if std else 0.02), **f32),
            "A_log": ParamSpec((H,), init=("normal", -1.0 if std else 0.0, 0.5 if std else 0.02), **f32),
            "dt_bias": ParamSpec((H * D if self.decay_rank else H,), init=("normal", -1.0 if std else 0.0, 0.5 if std else 0.02), **f32),
            "norm.weight": ParamSpec((Dv,), init=("normal", 1.0, 0.2 if std else 0.02), **f32),
            "o_proj.weight": ParamSpec((self.hidden, H * Dv), init=("normal", 0.0, std_out)),
        }
        for name, rows, rank in (("decay_proj.weight", H * D, self.decay_rank), ("gate_proj.weight", H * Dv, self.gate_rank)):
            if rank:
                out[name] = ParamSpec((rows, rank), init=("normal", 0.0, rank ** -0.5 if std else 0.02))
        return out

    def cache_need(self):
        tensors = [("s", (self.n_heads, self.v_dim, self.head_dim), "float32")]  # S column by column
        if self.taps > 1:
            tensors.append(("conv", (self.taps - 1, self.conv_dim), "float32"))
        return StateNeed(tuple(tensors))

    def workspace_bytes(self, n_tokens: int) -> int:
        item = 4 if self.env.dtype == torch.float32 else 2
        H, D, Dv = self.n_heads, self.head_dim, self.v_dim
        own = (self.proj_rows + self.conv_dim + H * Dv + self.hidden + (H * Dv if self.gate_rank else 0)) * item
        return n_tokens * (own + (H * Dv + (H * D if self.decay_rank else 0)) * 4) + self.chunk_scratch(n_tokens, n_tokens // CHUNK_MIN_TOKENS)[1]

    def chunk_scratch(self, n_tokens: int, n_long: int):
        """``(rows, bytes)`` of scratch for ``n_long`` requests of a step of so many tokens to go in chunks (0 bytes: they do not).

        A row of 64 tokens takes 50 KB a head and 16 or 32 a key head, 2.68 MB for 48 heads on 8 of 128.  All rows of the longest step
        would be 617 MB at 8,192 tokens, so larger steps than 32 rows get half of them (:func:`chunk_passes`): 172 MB, 343 MB at
        16,384 tokens, 86 MB below 4,096.  A pass more costs two launches."""
        if self.decay_rank:
            return 0, 0
        rows = n_tokens // ops.DELTA_CHUNK + n_long
        size = ops.delta_chunk_scratch(self.env.dtype, n_tokens, n_long, self.n_heads, self.n_kv_heads, self.head_dim, self.v_dim)
        most = min(rows, max(32, self.env.max_step_tokens // (2 * ops.DELTA_CHUNK)))
        return most, size // max(rows, 1) * most

    def forward(self, h: torch.Tensor, step: StepState, cache: Any, writes_cache: bool) -> torch.Tensor:
        if not writes_cache:
            raise ConfigError("gated_delta: a state cannot be shared between layers")
        T = h.shape[0]
        ws, dt, cap = self.env.workspace, self.env.dtype, self.env.max_step_tokens
        H, D, Dv = self.n_heads, self.head_dim, self.v_dim
        n_segs = len(step.segments)
        proj = ws.get("delta.proj", (T, self.proj_rows), dt, (cap, self.proj_rows))
        ops.linear(h, self.params["in_proj.weight"], proj)
        qkv = ws.get("delta.qkv", (T, self.conv_dim), dt, (cap, self.conv_dim))
        ops.conv_act(proj[:, : self.conv_dim], self.params["conv.weight"], None, "silu",
                     cache.tensors["conv"] if self.taps > 1 else None, step.state_slots, step.seg_info, n_segs, qkv)
        a, z = proj[:, self.a_col:], None
        if self.decay_rank:
            z = ws.get("delta.z", (T, H * D), torch.float32, (cap, H * D))
            ops.linear_f32(a, self.params["decay_proj.weight"], z)
            a = None
        o32 = ws.get("delta.o32", (T, H, Dv), torch.float32, (cap, H, Dv))
        args = dict(z=z)
        long = [seg.q_len for seg in step.segments if seg.q_len >= CHUNK_MIN_TOKENS] if z is None and h.is_cuda else []
        n_long = len(long)
        if long and self.row_bytes:
            need = T // ops.DELTA_CHUNK + n_long
            rows = min(need, self.most_rows)
            if chunks_pay(long, n_long < n_segs, H, self.n_kv_heads, D, Dv, rows):
                # (by rows: layers of other sizes have a buffer of their own, and no step asks for more rows)
                args = dict(scratch=ws.get("delta.chunks", (rows, self.row_bytes), torch.uint8, (self.most_rows, self.row_bytes)),
                            long_from=CHUNK_MIN_TOKENS, n_long=n_long)
                if rows < need:
                    args["passes"] = chunk_passes(long, rows)
        ops.delta_scan(qkv[:, : self.k_col], qkv[:, self.k_col: self.v_col], qkv[:, self.v_col:],
                       proj[:, self.b_col: self.a_col], a, self.params["A_log"], self.params["dt_bias"],
                       D ** -0.5, UNIT_EPS, cache.tensors["s"], step.state_slots, step.seg_info, n_segs, o32, **args)
        gate = proj[:, self.g_col: self.b_col]
        if self.gate_rank:
            low, gate = gate, ws.get("delta.gate", (T, H * Dv), dt, (cap, H * Dv))
            ops.linear(low, self.params["gate_proj.weight"], gate)
        o = ws.get("delta.o", (T, H, Dv), dt, (cap, H, Dv))
        ops.gated_heads(o32, gate, o, Dv, self.gate, self.params["norm.weight"], self.eps)
        out = ws.get("delta.out", (T, self.hidden), dt, (cap, self.hidden))
        ops.linear(o.view(T, H * Dv), self.params["o_proj.weight"], out)
        return out
