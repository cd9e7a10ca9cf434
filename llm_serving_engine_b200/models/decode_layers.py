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

# LSE_DECODE_LAYERS=0: decode steps launch by launch, for comparisons and for the timeline of single kernels
ENABLED = os.environ.get("LSE_DECODE_LAYERS", "1") != "0"


# Steps of at most so many values of the residual (rows x hidden size), and of at most the kernel's four rows, go through the
# one launch.  It saves a layer's nine hand-overs (1.3 to 1.9 us each), and costs the exchange of every phase's rows between all
# blocks, which grows with them.  One launch against launch by launch, microseconds a step: 28 layers of the 1.5B sizes (hidden
# 1,536), one request of 100 keys 879 / 1,158, two of 2,048 keys 1,056 / 1,238, four of 500 1,109 / 1,215, of 4,000 1,192 / 1,357
# (eight of 2,048 keys 1,338 / 1,310); four layers of the 7B sizes (3,584) and the head, one 511 / 597, two 543 / 594 (three
# 600 / 603); four of the 14B sizes (5,120), two 670 / 729 (four 823 / 754).
MOST_VALUES = 10240


class DecodeLayers:
    """The layers of a model whose decode steps the one-launch kernel can run."""

    def __init__(self, model) -> None:
        self.model = model
        first = model.blocks[model.spec.order[0]]
        self.mixer, self.inter = first.mixer, first.feed_forward.inter
        self.weights, self.eps = [], []
        for index in model.spec.order:
            block = model.blocks[index]
            mixer, ff = block.mixer, block.feed_forward
            self.weights.append([mixer.qkv_weight, mixer.o_weight, ff.gate_up_weight, ff.down_weight, mixer.qkv_bias,
                                 block.mixer_norm.weight, block.feed_forward_norm.weight])
            self.eps += [block.mixer_norm.eps, block.feed_forward_norm.eps]

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
                    or int(mixer.params["head_dim"]) != 128):
                return False
        return True

    @classmethod
    def of(cls, model) -> "DecodeLayers | None":
        """For a model whose layers are of that kind, else None."""
        spec = model.spec
        if model.device.type != "cuda" or not cls.described(spec, model.dtype):
            return None
        if model.embedding.dtype != torch.bfloat16 or model.lm_head.dtype != torch.bfloat16:
            return None
        first = model.blocks[spec.order[0]]
        for block in model.blocks:
            mixer, ff = block.mixer, block.feed_forward
            if (type(block) is not PreNormResidualBlock or type(mixer) is not GroupedQueryAttention or type(ff) is not SwiGLU
                    or type(block.mixer_norm) is not RMSNorm or type(block.feed_forward_norm) is not RMSNorm
                    or type(mixer.position) is not RotaryEncoding):
                return None
            if (mixer.head_dim != 128 or mixer.window or ff.activation != "silu" or ff.float32_output
                    or (mixer.n_q, mixer.n_kv, ff.inter) != (first.mixer.n_q, first.mixer.n_kv, first.feed_forward.inter)
                    or mixer.position.pairing != first.mixer.position.pairing
                    or mixer.position.params.get("theta") != first.mixer.position.params.get("theta")):
                return None
            matrices = (mixer.qkv_weight, mixer.o_weight, ff.gate_up_weight, ff.down_weight)
            if any(matrix.dtype != torch.bfloat16 for matrix in matrices):
                return None
        made = cls(model)
        tensors = [tensor for layer in made.weights for tensor in layer if tensor is not None] + [model.lm_head]
        if any(tensor.data_ptr() % 16 or not tensor.is_contiguous() for tensor in tensors) or not made.supported(1):
            return None
        return made

    def supported(self, rows: int) -> bool:
        spec = self.model.spec
        return ops.decode_layers_supported(len(spec.order), rows, spec.hidden_size, self.inter, self.mixer.n_q, self.mixer.n_kv,
                                           self.model.lm_head.shape[0])

    def wanted(self, rows: int) -> bool:
        """Whether a step of so many single tokens goes through the one launch."""
        return rows * self.model.spec.hidden_size <= MOST_VALUES and self.supported(rows)

    def forward(self, step, caches) -> torch.Tensor | None:
        """float32 logits of every row of a step of single tokens; None where the step has to go launch by launch."""
        model = self.model
        first = caches[0]
        if not self.wanted(step.num_tokens) or first.keys.shape[2] % 16 or first.keys.dtype != torch.bfloat16:
            return None
        if any(cache.group != first.group or cache.keys.shape != first.keys.shape for cache in caches):
            return None
        pointers = [[None if tensor is None else tensor.data_ptr() for tensor in weights] + [cache.keys.data_ptr(), cache.values.data_ptr()]
                    for weights, cache in zip(self.weights, caches)]
        return ops.decode_layers(pointers, self.eps, model.embedding, model.spec.embedding_scale, model.lm_head,
                                 model.final_norm.weight, model.final_norm.eps, self.mixer.position.inv_freq,
                                 self.mixer.position.pairing, step.token_ids, step.positions, step.segment_of_token,
                                 first.slot_mapping, first.block_tables, first.keys, self.inter, self.mixer.n_q, self.mixer.scale)
