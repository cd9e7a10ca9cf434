"""A decode step in one launch (``models/decode_layers.py``): steps of single tokens at the sizes where the kernel's layout
changes, against the plain implementation; and the same steps launch by launch."""
import random

import pytest
import torch

import helpers
from plain import qwen2_plain

pytestmark = pytest.mark.gpu

# hidden, feed-forward, query heads, key/value heads, vocabulary: a k range of one piece and few units; pieces and parts of
# different sizes in every product, eight heads a group; one head a group, more units than blocks
SIZES = {
    "small": (192, 320, 2, 1, 528),
    "odd": (1600, 4672, 16, 2, 1040),
    "wide": (576, 3136, 4, 4, 4112),
}
CONTEXTS = [0, 1, 15, 16, 17, 31, 127, 128, 129, 300, 64, 5, 48, 200, 33, 3]


def _build(name, pairing="interleaved"):
    from llm_serving_engine_b200.config import load_config
    from llm_serving_engine_b200.models import DecoderModel, expected_tensors

    hidden, inter, n_q, n_kv, vocab = SIZES[name]
    config = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "vocab_size": vocab, "hidden_size": hidden, "head_dim": 128,
              "intermediate_size": inter, "num_hidden_layers": 3, "num_attention_heads": n_q, "num_key_value_heads": n_kv,
              "max_position_embeddings": 1024, "rope_theta": 10000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": False}
    _, _, spec = load_config(config)
    for layer in spec.layers:
        layer.mixer.params["position"]["params"]["pairing"] = pairing
    generator = torch.Generator().manual_seed(hidden)
    weights = {}
    for tensor_name, tensor in expected_tensors(spec).items():
        value = torch.randn(tensor.shape, generator=generator) * (0.5 / tensor.shape[-1] ** 0.5 if tensor.kind == "matrix" else 0.05)
        weights[tensor_name] = (value if tensor.kind != "norm" else value + 1.0).to(torch.bfloat16)
    held = {key: (value.cuda() if value.dim() > 1 else value.float().cuda()) for key, value in weights.items()}
    return config, DecoderModel(spec, held, torch.bfloat16, "cuda"), {key: value.float() for key, value in weights.items()}


def _decode(model, sequences, steps, one_launch, use_graphs=False):
    """Logits of the last ``steps`` tokens of every sequence, decoded together; the tokens before them come as portions."""
    from llm_serving_engine_b200.cache import CacheManager
    from llm_serving_engine_b200.config import CacheConfig
    from llm_serving_engine_b200.engine import StepEntry, StepRunner
    from llm_serving_engine_b200.models import cache_requirements

    held, model._decode_layers = model._decode_layers, model._decode_layers if one_launch else None
    try:
        cache = CacheManager(cache_requirements(model.spec), CacheConfig(16, 16 * 40), model.dtype, "cuda", 1024, num_state_slots=16)
        for group in cache.groups:         # whatever lies behind a request's keys must not matter
            group.storage.fill_(float("nan"))
        runner = StepRunner(model, cache, max_tokens_per_step=1024, max_segments=16, use_graphs=use_graphs)
        for index, tokens in enumerate(sequences):
            cache.create(str(index))
            if len(tokens) > steps:
                runner.run([StepEntry(str(index), tokens[:-steps], [])])
        out = []
        for step in range(steps):
            entries = [StepEntry(str(index), [tokens[len(tokens) - steps + step]], [0]) for index, tokens in enumerate(sequences)]
            out.append(runner.run(entries).clone())
        return torch.stack(out, dim=1).cpu()      # [requests, steps, vocab]
    finally:
        model._decode_layers = held


@pytest.mark.parametrize("name,rows,first", [("small", 1, 0), ("small", 3, 1), ("small", 4, 4), ("small", 4, 8), ("odd", 1, 9), ("odd", 2, 2),
                                             ("odd", 4, 0), ("odd", 4, 6), ("wide", 1, 7), ("wide", 3, 3), ("wide", 4, 12)])
def test_against_the_plain_implementation(name, rows, first):
    from llm_serving_engine_b200.kernels import library

    config, model, weights = _build(name)
    assert model._decode_layers is not None and model._decode_layers.wanted(rows)
    rng = random.Random(rows)
    steps = 2
    sequences = [helpers.random_tokens(rng, config["vocab_size"], context + steps) for context in CONTEXTS[first:first + rows]]
    before = library.launches()
    got = _decode(model, sequences, steps, True, use_graphs=rows == 3)
    assert library.load().lse_decode_layers_status() == 0
    assert library.launches() > before
    repeated = _decode(model, sequences, steps, True)
    assert torch.equal(got, repeated)              # every sum has its order
    for index, tokens in enumerate(sequences):
        want = qwen2_plain.forward_full(config, weights, tokens)[-steps:]
        limit = helpers.tolerance("bfloat16", want)
        assert float((got[index] - want).abs().max()) <= limit, (name, rows, index)
        assert helpers.rms_ratio(got[index], want) <= helpers.RMS_RATIO_LARGE_LAYERS


@pytest.mark.parametrize("name,rows", [("small", 4), ("odd", 3)])
def test_halves_turned_as_launch_by_launch(name, rows):
    config, model, _ = _build(name, "half")
    rng = random.Random(rows)
    sequences = [helpers.random_tokens(rng, config["vocab_size"], context + 1) for context in CONTEXTS[2:2 + rows]]
    got, want = (_decode(model, sequences, 1, one_launch) for one_launch in (True, False))
    assert float((got - want).abs().max()) <= helpers.tolerance("bfloat16", want)


def test_some_rows_wanted():
    """A step launch by launch (no graph) that asks for some requests' logits only gives those, in their order."""
    from llm_serving_engine_b200.cache import CacheManager
    from llm_serving_engine_b200.config import CacheConfig
    from llm_serving_engine_b200.engine import StepEntry, StepRunner
    from llm_serving_engine_b200.models import cache_requirements

    _, model, _ = _build("small")

    def run(wants):
        cache = CacheManager(cache_requirements(model.spec), CacheConfig(16, 16), model.dtype, "cuda", 1024, num_state_slots=4)
        runner = StepRunner(model, cache, 64, 4, use_graphs=False)
        for index in range(3):
            cache.create(str(index))
        return runner.run([StepEntry(str(index), [7 + index], want) for index, want in enumerate(wants)]).clone()

    whole = run([[0], [0], [0]])
    assert torch.equal(run([[0], [], [0]]), whole[[0, 2]])
    assert torch.equal(run([[], [0, 0], [0]]), whole[[1, 1, 2]])
    assert run([[], [], []]).shape == (0, whole.shape[1])
