"""Attention whose keys and values are made from a cached low-rank latent."""
from __future__ import annotations

import math

import torch

from ..kernels import ops
from ..weights.tensor_spec import TensorSpec
from .base import Mixer, PagedLatent, register_mixer
from .linear import linear_partials

PER_HEAD_LIBRARY_ROWS = 32    # above this many bfloat16 rows the per-head products are the library's batched product

# Portions of prompts: keys and values of every head made from the gathered latent rows first, or attention over the latent
# rows themselves.  The former costs one product over the rows that the requests hold (at EXPAND_FLOPS a microsecond) and
# then 320 multiply-adds a (row, key, head) at EXPANDED_FLOPS; the latter none and 2 rank + 64 at LATENT_FLOPS (measured at
# 16 heads, a latent of 512: 2,048 rows of a prompt 11 + 39.5 us, with 4 for the gathering, against 611; the two products
# per head around the latter, 19 us, are saved too).  Both write into buffers of the step.
EXPAND_FLOPS, EXPANDED_FLOPS, LATENT_FLOPS = 1.0e9, 4.0e8, 1.2e8
EXPAND_OVERHEAD_US = 15.0     # two more launches, and the first tiles of an attention of few blocks
# Keys and values that are held at once (512 bytes a row and head), and gathered rows.  They are taken in the middle of a step,
# beside a cache that was sized before: no more than the buffers of a step of a few thousand rows over the latent rows take.
# Where the heads' keys and values take more, some heads at a time are made and attended to: 128 heads, 256 rows behind 8,000
# keys, captured: 891 us (572 with all of them at once, in 805 MB) against 4,540 over the latent rows.
EXPAND_MAX_BYTES = 1 << 28


def _size_class(rows: int) -> int:
    """``rows`` rounded up to half a power of two: captured steps are kept by it, so a prompt in portions meets two classes for
    every doubling of its context (four had nearly every portion captured anew), and the product makes at most half as many
    rows again as there are.  Steps launched one by one make the rows that there are."""
    step = max(64, 1 << max(0, (rows - 1).bit_length() - 2))
    return -(-rows // step) * step

_DEFAULT_NAMES = {"q_down": "dq", "q_down_norm": "dq.norm", "q_up": "uq", "q": "q", "kv_down": "dkv",
                  "kv_down_norm": "dkv.norm", "k_up": "uk", "v_up": "uv", "sink": "sink", "gate": "g", "out": "o"}


def rotary_frequencies(rot: dict) -> tuple[torch.Tensor, float]:
    """Frequencies (float64 [dims / 2]) and the factor on cos and sin of a rotary description ``{base, dims,
    scaling}``.  Without ``scaling``: f_i = base^(-2i / dims), factor 1.  With ``scaling`` = {factor s, original n,
    fast, slow} (the scheme known as YaRN): with pair(t) = dims ln(n / (2 pi t)) / (2 ln base) the index of the pair
    that makes t turns over n positions, lo = max(floor(pair(fast)), 0), hi = min(ceil(pair(slow)), dims - 1) and
    ramp_i = clamp((i - lo) / max(hi - lo, 0.001), 0, 1), the frequency is f_i / s * ramp_i + f_i (1 - ramp_i):
    fast pairs keep theirs, slow pairs are stretched by s; cos and sin are multiplied by 0.1 ln(s) + 1."""
    dims, base = int(rot["dims"]), float(rot["base"])
    index = torch.arange(dims // 2, dtype=torch.float64)
    freq = base ** (-2.0 * index / dims)
    scaling = rot.get("scaling")
    if not scaling:
        return freq, 1.0
    factor, original = float(scaling["factor"]), float(scaling["original"])

    def pair(turns: float) -> float:
        return dims * math.log(original / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

    lo = max(math.floor(pair(float(scaling["fast"]))), 0)
    hi = min(math.ceil(pair(float(scaling["slow"]))), dims - 1)
    ramp = ((index - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return freq / factor * ramp + freq * (1.0 - ramp), 0.1 * math.log(factor) + 1.0


@register_mixer("latent_attention")
class LatentAttention(Mixer):
    """params: ``heads``, ``dim`` (unrotated query/key size of a head), ``rot_dim`` (rotated size), ``vdim``,
    ``kv_rank`` (the latent), ``q_rank`` (0: queries are projected directly; else they go through a normed latent of
    this size), ``scale`` (on the scores), ``rot`` ({base, dims, scaling}: see :func:`rotary_frequencies`; the first
    ``dims`` of the ``rot_dim`` values are rotated in interleaved pairs), ``eps`` (of the latent norms), ``sink`` (a
    learned number per head in the softmax's denominator), ``gate`` (true, or "head": head h's output times sigmoid(W_g x)_h;
    "elements": the concatenated heads times sigmoid(W_g x), W_g with a row per value), ``window`` (> 0: a row reads its last
    ``window`` keys, itself included; older pages are given back),
    ``own_cache`` (false: the layer reads the latent rows of another layer, ``LayerSpec.cache_from``, and has no
    down-projection of its own), ``tensor_names``.

    c = norm(W_dkv x)[:kv_rank] and the rotated last rot_dim values of W_dkv x (shared by the heads) are the cached
    row of a token; head h's key is [W_uk,h c | shared part], its value W_uv,h c.  The per-head maps are folded
    around the attention: q' = W_uk,h^T q_unrotated before it, W_uv,h after it, so that the attention runs over the
    cached rows themselves (``csrc/attention_latent.cu``)."""

    graph_safe = True
    kernel_sources = ("attention_latent", "attention_latent_mma", "gemm_heads", "attention_expanded_tcgen05",)

    def __init__(self, params, weights, ctx) -> None:
        super().__init__(params, weights, ctx)
        p = params
        self.heads, self.dim, self.rot_dim = int(p["heads"]), int(p["dim"]), int(p["rot_dim"])
        self.vdim, self.rank, self.q_rank = int(p["vdim"]), int(p["kv_rank"]), int(p.get("q_rank") or 0)
        self.scale, self.eps = float(p["scale"]), float(p["eps"])
        self.window = int(p.get("window", 0))
        self.own_cache = bool(p.get("own_cache", True))
        self.rot_dims = int(p["rot"]["dims"])
        if self.rot_dims > self.rot_dim or self.rot_dims % 2:
            raise ops.KernelError(f"latent attention: {self.rot_dims} rotated values of {self.rot_dim}")
        freq, self.rot_factor = rotary_frequencies(p["rot"])
        self.freq = freq.to(ctx.device)
        names = {**_DEFAULT_NAMES, **p.get("tensor_names", {})}
        stacked, self.q_off, self.kv_off, self.g_off = [], 0, -1, -1
        width = 0
        if self.q_rank:
            stacked.append(weights[names["q_down"]])
            self.q_norm = weights[names["q_down_norm"]].to(torch.float32).contiguous()
            self.q_up = weights[names["q_up"]].contiguous()
            width += self.q_rank
        else:
            stacked.append(weights[names["q"]])
            width += self.heads * (self.dim + self.rot_dim)
        self.kv_norm = None
        if self.own_cache:
            stacked.append(weights[names["kv_down"]])
            self.kv_norm = weights[names["kv_down_norm"]].to(torch.float32).contiguous()
            self.kv_off = width
            width += self.rank + self.rot_dim
        self.gates = self._gates(p)
        if self.gates:
            stacked.append(weights[names["gate"]])
            self.g_off = width
            width += self.gates
        if self.gates > self.heads and width % 16:       # whole tiles of the product, aligned rows of its result
            stacked.append(stacked[0].new_zeros((-width % 16, stacked[0].shape[1])))
        self.in_weight = torch.cat(stacked, dim=0).contiguous()
        self.kv_up = torch.cat([weights[names["k_up"]], weights[names["v_up"]]], dim=0).contiguous()
        self.k_up = self.kv_up[:self.heads * self.dim].view(self.heads, self.dim, self.rank)
        self.v_up = self.kv_up[self.heads * self.dim:].view(self.heads, self.vdim, self.rank).transpose(1, 2)
        self.sink = weights[names["sink"]].to(torch.float32).contiguous() if p.get("sink", False) else None
        self.out_weight = weights[names["out"]].contiguous()
        self._tile: int | None = None      # keys of a tile of the expanded attention, 0: not for this layer (see _key_tile)

    @staticmethod
    def _gates(params) -> int:
        """Rows of the gate's matrix: none, one per head, or one per value."""
        kind = params.get("gate", False)
        if kind not in (False, None, True, "head", "elements"):
            raise ops.KernelError(f"latent attention: gate {kind!r} must be false, head or elements")
        return int(params["heads"]) * (int(params["vdim"]) if kind == "elements" else 1) if kind else 0

    @classmethod
    def expected_tensors(cls, params, hidden_size):
        p = params
        heads, dim, rot, vdim, rank = int(p["heads"]), int(p["dim"]), int(p["rot_dim"]), int(p["vdim"]), int(p["kv_rank"])
        q_rank = int(p.get("q_rank") or 0)
        names = {**_DEFAULT_NAMES, **p.get("tensor_names", {})}
        out = {}
        if q_rank:
            out[names["q_down"]] = TensorSpec((q_rank, hidden_size))
            out[names["q_down_norm"]] = TensorSpec((q_rank,), "norm")
            out[names["q_up"]] = TensorSpec((heads * (dim + rot), q_rank))
        else:
            out[names["q"]] = TensorSpec((heads * (dim + rot), hidden_size))
        if p.get("own_cache", True):
            out[names["kv_down"]] = TensorSpec((rank + rot, hidden_size))
            out[names["kv_down_norm"]] = TensorSpec((rank,), "norm")
        out[names["k_up"]] = TensorSpec((heads * dim, rank))
        out[names["v_up"]] = TensorSpec((heads * vdim, rank))
        if p.get("sink", False):
            out[names["sink"]] = TensorSpec((heads,), "bias")
        if cls._gates(p):
            out[names["gate"]] = TensorSpec((cls._gates(p), hidden_size))
        out[names["out"]] = TensorSpec((hidden_size, heads * vdim))
        return out

    @classmethod
    def cache_requirement(cls, params, hidden_size):
        return PagedLatent(int(params["kv_rank"]) + int(params["rot_dim"]), int(params.get("window", 0)))

    def _key_tile(self) -> int:
        """Keys of a tile of the attention over expanded keys and values, 0 if it does not take this layer."""
        if self._tile is None:
            taken = self.gates <= self.heads and self.scale > 0.0 and ops.attention_expanded_supported(
                self.dim, self.rot_dim, self.vdim, self.rank, self.ctx.dtype)
            self._tile = ops.attention_expanded_tile() if taken else 0
        return self._tile

    def _expanded_rows(self, segment_counts: list[int], contexts: list[int]) -> int:
        """How many rows of keys and values are made for a step of this shape (a size class), or 0: the attention runs over
        the latent rows.  ``contexts``: keys of each request after the step."""
        return _size_class(rows) if (rows := self._worth_expanding(segment_counts, contexts)) else 0

    def _worth_expanding(self, segment_counts: list[int], contexts: list[int]) -> int:
        """The same without the size class: the rows that there are, each request's rounded up to whole key tiles.  Whether it is
        worth it goes by the class."""
        tile = self._key_tile() if self._tile is None else self._tile
        if min(segment_counts) == 1 or not tile:
            return 0
        window, exact, pairs = self.window, 0, 0
        for count, context in zip(segment_counts, contexts):
            first = max(0, context - count + 1 - window) if window > 0 else 0
            exact += -(-(context - first) // tile) * tile
            pairs += count * (min(context, window) if window > 0 else context - count // 2)
        rows = _size_class(exact)
        expanded = (2.0 * rows * self.kv_up.numel() / EXPAND_FLOPS
                    + 2.0 * pairs * self.heads * (self.dim + self.rot_dim + self.vdim) / EXPANDED_FLOPS + EXPAND_OVERHEAD_US)
        latent = 2.0 * pairs * self.heads * (2 * self.rank + self.rot_dim) / LATENT_FLOPS
        fits = 2 * rows * max(self.dim + self.vdim, self.rank + self.rot_dim) <= EXPAND_MAX_BYTES      # a head, the gathered rows
        return exact if fits and expanded < latent else 0

    def launch_signature_at(self, segment_counts, contexts):
        rows = self._expanded_rows(segment_counts, contexts)
        return ("expanded", rows) if rows else ()

    def _expanded_attention(self, q_plain, q_wide, step, cache, gate, rows: int):
        gathered = ops.latent_gather(cache.keys, cache.block_tables, step.segment_first_position, step.segment_context, rows, self.window)
        latent, dim = gathered[:, :self.rank], self.dim
        at_once = EXPAND_MAX_BYTES // (4 * rows * dim)      # heads whose keys and values are made together
        if at_once >= self.heads:
            kv = torch.mm(latent, self.kv_up.t()).view(rows, 2 * self.heads, dim)
            values = torch.empty((q_plain.shape[0], self.heads, self.vdim), dtype=q_plain.dtype, device=q_plain.device)
            return ops.attention_expanded(q_plain, q_wide, gathered, kv, values, step.segment_start, step.segment_first_position,
                                          step.segment_context, self.scale, self.window, self.sink, gate)
        values = torch.empty((q_plain.shape[0], self.heads, self.vdim), dtype=q_plain.dtype, device=q_plain.device)
        buffer = torch.empty(rows * 2 * at_once * dim, dtype=q_plain.dtype, device=q_plain.device)
        for first in range(0, self.heads, at_once):
            count = min(at_once, self.heads - first)
            kv = buffer[:rows * 2 * count * dim].view(rows, 2 * count * dim)
            keys, vals = (self.kv_up[at:at + count * dim] for at in (first * dim, (self.heads + first) * dim))
            torch.mm(latent, keys.t(), out=kv[:, :count * dim])
            torch.mm(latent, vals.t(), out=kv[:, count * dim:])
            ops.attention_expanded(q_plain, q_wide, gathered, kv.view(rows, 2 * count, dim), values, step.segment_start,
                                   step.segment_first_position, step.segment_context, self.scale, self.window, self.sink, gate, first)
        return values

    def _fold_queries(self, q_plain, q_wide) -> None:
        """q_wide[t, h, :rank] = W_uk,h^T q_plain[t, h]: many bfloat16 rows go to the library's batched product (the tensor
        cores), few rows and float32 to the engine's own kernel (true float32, one summation order)."""
        if q_plain.dtype == torch.bfloat16 and q_plain.shape[0] > PER_HEAD_LIBRARY_ROWS:
            torch.bmm(q_plain.transpose(0, 1), self.k_up, out=q_wide[:, :, :self.rank].transpose(0, 1))
        else:
            ops.head_gemm(q_plain, self.k_up, q_wide[:, :, :self.rank])

    def _expand_values(self, attended, values, gate, proj) -> None:
        """values[t, h] = gate * W_uv,h attended[t, h]; ``gate`` [T, heads], [T, heads, vdim], or None (without gates, or when
        the gate columns of ``proj`` are still to be taken)."""
        if attended.dtype == torch.bfloat16 and attended.shape[0] > PER_HEAD_LIBRARY_ROWS:
            if gate is None and self.g_off < 0:
                torch.bmm(attended.transpose(0, 1), self.v_up, out=values.transpose(0, 1))
                return
            product = torch.bmm(attended.transpose(0, 1), self.v_up)            # [heads, T, vdim], float32 accumulation
            if gate is None:
                ops.gate_heads(product, proj, self.g_off, values)
            else:
                torch.mul(product.transpose(0, 1), gate if gate.dim() == 3 else gate.unsqueeze(-1), out=values)
        else:
            ops.head_gemm(attended, self.v_up, values, gate)

    def forward(self, x, step, cache):
        tokens, heads = x.shape[0], self.heads
        proj = linear_partials(x, self.in_weight)
        wide = self.rank + self.rot_dim
        q_plain = torch.empty((tokens, heads, self.dim), dtype=x.dtype, device=x.device)
        q_wide = torch.empty((tokens, heads, wide), dtype=x.dtype, device=x.device)
        # many rows: the kernel behind the values' product takes the gates from the projection itself
        late_gates = self.gates > heads and x.dtype == torch.bfloat16 and proj.dim() == 2 and tokens > PER_HEAD_LIBRARY_ROWS
        gate = (torch.empty((tokens, self.gates), dtype=torch.float32, device=x.device)
                if self.gates and not late_gates else None)
        if not self.q_rank and self.own_cache:
            ops.latent_front(proj, step.positions, cache.slot_mapping, self.eps, q_off=self.q_off, heads=heads, dim=self.dim,
                             rot=self.rot_dim, rot_dims=self.rot_dims, freq=self.freq, rot_factor=self.rot_factor,
                             kv_off=self.kv_off, rank=self.rank, kv_norm=self.kv_norm, q_plain=q_plain, q_wide=q_wide,
                             cache=cache.keys, g_off=self.g_off, gate=gate)
        else:
            q_latent = torch.empty((tokens, self.q_rank), dtype=x.dtype, device=x.device) if self.q_rank else None
            if self.q_rank or self.own_cache or gate is not None:
                ops.latent_prepare(proj, step.positions, cache.slot_mapping, self.eps,
                                   q_off=self.q_off, q_rank=self.q_rank, q_norm=self.q_norm if self.q_rank else None,
                                   q_latent=q_latent, kv_off=self.kv_off, rank=self.rank, kv_norm=self.kv_norm,
                                   rot=self.rot_dim, rot_dims=self.rot_dims, freq=self.freq, rot_factor=self.rot_factor,
                                   cache=cache.keys, g_off=self.g_off, heads=self.gates, gate=gate)
            queries = linear_partials(q_latent, self.q_up) if self.q_rank else proj
            ops.latent_query(queries, 0, heads, self.dim, self.rot_dim, self.rot_dims, self.freq, self.rot_factor,
                             step.positions, step.segment_of_token, q_plain, q_wide, self.rank)
        expanded = 0
        if not step.decode_only:
            shape = ([segment.count for segment in step.segments], [segment.first_position + segment.count for segment in step.segments])
            expanded = self._worth_expanding(*shape)
            if expanded and step.max_context is None:      # a step that is captured for its class
                expanded = _size_class(expanded)
        if expanded:
            values = self._expanded_attention(q_plain, q_wide, step, cache, gate, expanded)
            return linear_partials(values.view(tokens, heads * self.vdim), self.out_weight)
        self._fold_queries(q_plain, q_wide)
        attended = torch.empty((tokens, heads, self.rank), dtype=x.dtype, device=x.device)
        ops.latent_attention(q_wide, cache.keys, attended, cache.block_tables, step.segment_of_token, step.positions,
                             self.scale, self.sink, self.window, segment_start=step.segment_start,
                             segment_first_position=step.segment_first_position)
        values = torch.empty((tokens, heads, self.vdim), dtype=x.dtype, device=x.device)
        if gate is not None and self.gates > heads:
            gate = gate.view(tokens, heads, self.vdim)
        self._expand_values(attended, values, gate, proj)
        return linear_partials(values.view(tokens, heads * self.vdim), self.out_weight)
