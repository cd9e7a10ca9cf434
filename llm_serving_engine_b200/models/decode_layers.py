"""A decode step of a whole model in one launch.

Models made of pre-norm layers of grouped-query attention (rotary positions, head size 128) and a SiLU-gated
feed-forward, in bfloat16, run a step of few single tokens through ``ops.decode_layers``: one kernel walks all layers and
the LM head (reference ``src/llmserve/model.py:270-309``, a step of single tokens).  Everything else (prompt portions, more
rows, other parts, float32, a hook between layers) runs launch by launch through the parts.
"""
from __future__ import annotations

import os

import torch

from ..config.model_config import ModelSpec
from ..kernels import ops
from ..parts.attention import GroupedQueryAttention
from ..parts.base import BLOCKS, FEED_FORWARDS, MIXERS, NORMS, POSITION_ENCODINGS
from ..parts.block import PreNormResidualBlock
from ..parts.mlp import SwiGLU
from ..parts.norm import RMSNorm
from ..parts.rope import RotaryEncoding

HEAD = 128     # head size of the kernel

# LSE_DECODE_LAYERS=0: decode steps launch by launch, for comparisons and for the timeline of single kernels
ENABLED = os.environ.get("LSE_DECODE_LAYERS", "1") != "0"


# Steps of at most so many values of the residual (rows x hidden size), and of at most the kernel's four rows, go through the
# one launch.  It saves a layer's nine hand-overs (1.3 to 1.9 us each), and costs the exchange of every phase's rows between all
# blocks, which grows with them.  One launch against launch by launch, microseconds a step with its upload: 28 layers of the 1.5B
# sizes (hidden 1,536), one request of 100 keys 920 / 1,232, of 30,000 1,316 / 1,615, two of 2,048 1,064 / 1,313, four of 500
# 1,138 / 1,257, of 4,000 1,216 / 1,371, of 30,000 1,673 / 1,888 (eight of 2,048 keys 1,338 / 1,310); four layers of the 7B sizes
# (3,584) and the head, one 519 / 617, two 556 / 620 (three 600 / 603); four of the 14B sizes (5,120), two 693 / 756 (four 823 /
# 754).  The contexts do not change the answer: four layers of the 1.5B sizes, one request of 8,000 keys 250 / 316, of 100,000
# 397 / 422, two of 100,000 423 / 437, four of 8,000 302 / 335; of the 7B sizes, two of 100,000 811 / 886; of the 14B sizes, two of
# 8,000 751 / 801, of 100,000 1,159 / 1,279.
MOST_VALUES = 10240


# A part whose class or instance has another ``forward`` (wrapped to look at what passes, replaced in a trial) is called, not read.
_CALLED = {PreNormResidualBlock: "forward", GroupedQueryAttention: "forward", SwiGLU: "forward", RMSNorm: "forward",
           RotaryEncoding: "encode_and_store"}
_AS_WRITTEN = {cls: getattr(cls, name) for cls, name in _CALLED.items()}


def _plain(part, cls) -> bool:
    name = _CALLED[cls]
    return type(part) is cls and name not in vars(part) and getattr(cls, name) is _AS_WRITTEN[cls]


def _matrix(tensor, rows: int, columns: int) -> bool:
    return (tensor.dtype == torch.bfloat16 and tensor.shape == (rows, columns) and tensor.is_contiguous() and tensor.data_ptr() % 16 == 0)


def _vector(tensor, size: int) -> bool:
    return tensor.dtype == torch.float32 and tensor.shape == (size,) and tensor.is_contiguous() and tensor.data_ptr() % 16 == 0


class DecodeLayers:
    """Decode steps of a model whose layers the one-launch kernel can run.  Nothing is kept of the layers: every step that is
    launched (a captured one: when it is captured) reads the parts as they are then."""

    def __init__(self, model) -> None:
        self.model = model
        self.refused = False     # the device did not take the launch: it will not take the next one either

    @staticmethod
    def described(spec: ModelSpec, dtype: torch.dtype) -> bool:
        """Whether models of this description may be of that kind: then they have the kernel loaded when they are built."""
        if (not ENABLED or dtype != torch.bfloat16 or spec.residual_streams != 1 or spec.position_table_name or spec.embedding_again
                or NORMS.get(spec.final_norm.kind) is not RMSNorm):
            return False
        for layer in spec.layers:
            mixer, ff = layer.mixer, layer.feed_forward
            if (ff is None or layer.feed_forward_norm is None or BLOCKS.get(layer.block.kind) is not PreNormResidualBlock
                    or MIXERS.get(mixer.kind) is not GroupedQueryAttention or FEED_FORWARDS.get(ff.kind) is not SwiGLU
                    or NORMS.get(layer.mixer_norm.kind) is not RMSNorm or NORMS.get(layer.feed_forward_norm.kind) is not RMSNorm
                    or POSITION_ENCODINGS.get(mixer.params["position"]["kind"]) is not RotaryEncoding
                    or int(mixer.params["head_dim"]) != HEAD):
                return False
        return True

    @classmethod
    def of(cls, model) -> "DecodeLayers | None":
        """For a model whose layers are of that kind, else None."""
        if model.device.type != "cuda" or not cls.described(model.spec, model.dtype):
            return None
        made = cls(model)
        return made if made._layers() is not None and made._asked(ops.decode_layers_fits, 1) else None

    def _layers(self):
        """(weights, both norms' eps) of every layer run, from the parts as they are now; None where one is not what the kernel runs."""
        model = self.model
        hidden, final, first = model.spec.hidden_size, model.final_norm, self._first.mixer
        if not (_plain(final, RMSNorm) and _vector(final.weight, hidden) and _matrix(model.lm_head, len(model.lm_head), hidden)
                and _matrix(model.embedding, len(model.embedding), hidden)):
            return None
        weights, eps = [], []
        for index in model.spec.order:
            block = model.blocks[index]
            if not _plain(block, PreNormResidualBlock):
                return None
            mixer, ff, norm1, norm2 = block.mixer, block.feed_forward, block.mixer_norm, block.feed_forward_norm
            if not (_plain(mixer, GroupedQueryAttention) and _plain(ff, SwiGLU) and _plain(norm1, RMSNorm) and _plain(norm2, RMSNorm)
                    and _plain(mixer.position, RotaryEncoding)):
                return None
            n_q, n_kv, inter, position = mixer.n_q, mixer.n_kv, ff.inter, mixer.position
            if (mixer.head_dim != HEAD or mixer.window or ff.activation != "silu" or ff.float32_output
                    or (n_q, n_kv, mixer.scale) != (first.n_q, first.n_kv, first.scale) or inter != self.inter
                    or position.pairing != first.position.pairing or position.params.get("theta") != first.position.params.get("theta")):
                return None
            rows = (n_q + 2 * n_kv) * HEAD
            if not (_matrix(mixer.qkv_weight, rows, hidden) and _matrix(mixer.o_weight, hidden, n_q * HEAD)
                    and _matrix(ff.gate_up_weight, 2 * inter, hidden) and _matrix(ff.down_weight, hidden, inter)
                    and _vector(norm1.weight, hidden) and _vector(norm2.weight, hidden)
                    and (mixer.qkv_bias is None or _vector(mixer.qkv_bias, rows))):
                return None
            weights.append((mixer.qkv_weight, mixer.o_weight, ff.gate_up_weight, ff.down_weight, mixer.qkv_bias, norm1.weight, norm2.weight))
            eps += [norm1.eps, norm2.eps]
        return weights, eps

    @property
    def _first(self):
        return self.model.blocks[self.model.spec.order[0]]

    @property
    def inter(self) -> int:
        return self._first.feed_forward.inter

    def supported(self, rows: int) -> bool:
        return self._asked(ops.decode_layers_supported, rows)

    def _asked(self, question, rows: int) -> bool:
        spec, mixer = self.model.spec, self._first.mixer
        return question(len(spec.order), rows, spec.hidden_size, self.inter, mixer.n_q, mixer.n_kv, len(self.model.lm_head))

    def wanted(self, rows: int) -> bool:
        """Whether a step of so many single tokens goes through the one launch."""
        return rows * self.model.spec.hidden_size <= MOST_VALUES and self.supported(rows)

    def forward(self, step, caches) -> torch.Tensor | None:
        """float32 logits of every row of a step of single tokens; None where the step has to go launch by launch."""
        model = self.model
        first = caches[0]
        if self.refused or step.num_tokens * model.spec.hidden_size > MOST_VALUES or first.keys.shape[2] % 16 or first.keys.dtype != torch.bfloat16:
            return None
        if any(cache.group != first.group or cache.keys.shape != first.keys.shape for cache in caches):
            return None
        layers = self._layers()
        if layers is None or not self.supported(step.num_tokens):
            return None
        weights, eps = layers
        pointers = [[None if tensor is None else tensor.data_ptr() for tensor in of_layer] + [cache.keys.data_ptr(), cache.values.data_ptr()]
                    for of_layer, cache in zip(weights, caches)]
        mixer = self._first.mixer
        logits = ops.decode_layers(pointers, eps, model.embedding, model.spec.embedding_scale, model.lm_head,
                                   model.final_norm.weight, model.final_norm.eps, mixer.position.inv_freq, mixer.position.pairing,
                                   step.token_ids, step.positions, step.segment_of_token, first.slot_mapping, first.block_tables,
                                   first.keys, self.inter, mixer.n_q, mixer.scale)
        self.refused = logits is None
        return logits
