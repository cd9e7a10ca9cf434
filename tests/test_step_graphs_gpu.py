"""Captured steps replayed at other contexts of their class, through the step function."""
import pytest
import torch

from llm_serving_engine_b200.cache import CacheManager
from llm_serving_engine_b200.config import CacheConfig
from llm_serving_engine_b200.engine import StepEntry, StepRunner
from llm_serving_engine_b200.models import cache_requirements
from llm_serving_engine_b200.parts import latent_attention
from test_launch_signature_cpu import latent_model

pytestmark = pytest.mark.gpu


def runner_for(model, use_graphs, positions=2048, page=16, pages=200, tokens=512, segments=8):
    cache = CacheManager(cache_requirements(model.spec), CacheConfig(page, pages), model.dtype, "cuda", positions, num_state_slots=segments)
    return StepRunner(model, cache, tokens, segments, use_graphs=use_graphs)


def in_portions(runner, rid, tokens, size):
    """The logits of every token of a request that is run alone in portions of ``size``."""
    runner.cache.create(rid)
    out = []
    for lo in range(0, len(tokens), size):
        part = tokens[lo:lo + size]
        out.append(runner.run([StepEntry(rid, part, list(range(len(part))))]).clone())
    runner.cache.free(rid)
    return torch.cat(out)


def test_a_captured_step_is_not_replayed_where_a_layer_launches_something_else(monkeypatch):
    """A windowed and a full latent layer, room bounded so that the full layer makes keys and values up to 128 keys only, a head at
    a time: the second portions of two requests capture the step, the later portions of a third have the windowed layer's buffer of the same
    size, but a full layer that goes over the latent rows.  Every logit against the latent rows' kernel launch by launch."""
    model = latent_model([64, 0], heads=2, rank=64, device="cuda", scale=0.07)
    generator = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, 64, (length,), generator=generator).tolist() for length in (128, 128, 448)]
    plain = runner_for(model, use_graphs=False)
    monkeypatch.setattr(latent_attention, "LATENT_FLOPS", 1.0e30)      # never worth it
    want = [in_portions(plain, "r", tokens, 64) for tokens in prompts]
    monkeypatch.setattr(latent_attention, "LATENT_FLOPS", 1.0)         # always worth it, where it fits
    monkeypatch.setattr(latent_attention, "EXPAND_MAX_BYTES", 128 * 512)
    graphs = runner_for(model, use_graphs=True)
    for index, tokens in enumerate(prompts):
        got = in_portions(graphs, "r", tokens, 64)
        # bfloat16 at other places of two layers: a few units in the last place of the largest logit
        assert float((got - want[index]).abs().max()) <= 2.0 ** -4 * float(want[index].abs().max()), index
    assert graphs.portion_graph_replays >= 4


def test_warmup_runs_the_kernels_of_a_portion_alone(monkeypatch):
    """A latent layer's portion alone goes over expanded keys and values, beside a single token over the latent rows: both are run
    once before the first request, and the cache is left empty."""
    from llm_serving_engine_b200.kernels import ops

    calls = []
    for name in ("attention_expanded", "latent_attention"):
        def recorded(*args, _real=getattr(ops, name), _name=name, **more):
            calls.append(_name)
            return _real(*args, **more)

        monkeypatch.setattr(ops, name, recorded)
    monkeypatch.setattr(latent_attention, "LATENT_FLOPS", 1.0)
    runner = runner_for(latent_model([0], heads=1, rank=64, device="cuda", scale=0.07), use_graphs=True, segments=2)
    runner.warmup()
    assert calls[:2] == ["latent_attention", "attention_expanded"] and not runner.cache.requests
    assert runner.cache.groups[0].pool.used_pages == 0


def test_captured_steps_beyond_the_bound_make_room_for_each_other():
    """Three classes of steps in turn where two graphs are kept: captured, dropped, captured again, and always the same logits;
    the class used last stays."""
    model = latent_model([0], heads=1, rank=64, device="cuda", scale=0.07)
    generator = torch.Generator().manual_seed(7)
    prompts = [torch.randint(0, 64, (length,), generator=generator).tolist() for length in (16, 30, 45)]
    plain, graphs = runner_for(model, use_graphs=False), runner_for(model, use_graphs=True)
    graphs.MAX_PORTION_GRAPHS = 2
    want = [in_portions(plain, "r", tokens, 64) for tokens in prompts]
    for index in (0, 0, 1, 1, 0, 2, 2, 0, 1, 1, 1, 2, 2, 2, 0):
        got = in_portions(graphs, "r", prompts[index], 64)
        assert float((got - want[index]).abs().max()) <= 2.0 ** -5 * float(want[index].abs().max()), index
        assert len(graphs._portion_graphs) <= 2
    assert [key[1] for key in graphs._portion_graphs] == [32, 48] or [key[1] for key in graphs._portion_graphs] == [48, 32]
    assert graphs.portion_graph_replays >= 6


def attention_model(heads=(12, 2), layers=1):
    """Grouped-query attention layers of 128 values a head in bfloat16, as the large models have them, with a narrow feed-forward."""
    config = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": layers, "hidden_size": 128 * heads[0],
              "intermediate_size": 64, "num_attention_heads": heads[0], "num_key_value_heads": heads[1],
              "vocab_size": 64, "max_position_embeddings": 4096, "rope_theta": 10000.0, "rms_norm_eps": 1e-6,
              "tie_word_embeddings": True, "attention_bias": True}
    from llm_serving_engine_b200.config import load_config
    from llm_serving_engine_b200.models import DecoderModel, expected_tensors

    _, _, spec = load_config(config)
    generator = torch.Generator().manual_seed(2)
    weights = {}
    for name, tensor in expected_tensors(spec).items():
        values = torch.randn(tensor.shape, generator=generator)
        weights[name] = ((values * tensor.shape[-1] ** -0.5).bfloat16() if tensor.kind == "matrix" else 1.0 + 0.1 * values).cuda()
    return DecoderModel(spec, weights, torch.bfloat16, "cuda")


def test_decode_steps_split_their_keys_by_the_contexts_and_not_by_the_tables(monkeypatch):
    """64 requests in tables of 4,096 keys, captured: whole while the longest context is below 1,024 keys, in two splits from
    there on, each from a graph of its own that the warm-up has made, with the logits of the step launched one by one."""
    from llm_serving_engine_b200.kernels import ops

    model, splits, real = attention_model(), [], ops.paged_attention_decode
    assert model.decode_depends_on_keys(64) and not model.decode_depends_on_keys(1)

    def recorded(*args, **more):
        splits.append(args[8])
        return real(*args, **more)

    monkeypatch.setattr(ops, "paged_attention_decode", recorded)
    sizes = dict(positions=4096, pages=6000, tokens=2100, segments=64)
    graphs, plain = runner_for(model, use_graphs=True, **sizes), runner_for(model, use_graphs=False, **sizes)
    graphs.warmup([64])
    assert {1, 2} <= set(splits) and len(graphs._graphs) == 2
    generator = torch.Generator().manual_seed(9)
    lengths = [1006 if index == 5 else 20 + index for index in range(64)]      # + 1: 63 pages of 16 keys; then 1,008 and 1,009
    tokens = [torch.randint(0, 64, (length + 3,), generator=generator).tolist() for length in lengths]
    for runner in (graphs, plain):
        for index, length in enumerate(lengths):
            runner.cache.create(str(index))
            runner.run([StepEntry(str(index), tokens[index][:length], [])])
    for turn, (eager, kind) in enumerate(((1, 0), (1, 0), (1, 1))):
        entries = [StepEntry(str(index), tokens[index][length + turn:length + turn + 1], [0]) for index, length in enumerate(lengths)]
        splits.clear()
        replays = graphs.graph_replays
        got, want = graphs.run(entries).clone(), plain.run(entries)
        assert splits == [eager] and graphs.graph_replays == replays + 1 and len(graphs._graphs) == 2
        assert graphs._decode_key(64, graphs._pages_after([StepEntry(e.request_id, [], []) for e in entries]))[2] == kind, turn
        assert float((got - want).abs().max()) <= 2.0 ** -5 * float(want.abs().max())      # bfloat16, another order of sums


_ROUNDED_UP = """
import random, torch
from llm_serving_engine_b200.cache import CacheManager
from llm_serving_engine_b200.config import CacheConfig, load_config
from llm_serving_engine_b200.engine import StepEntry, StepRunner
from llm_serving_engine_b200.kernels import library, ops
from llm_serving_engine_b200.models import DecoderModel, cache_requirements, expected_tensors

config = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "vocab_size": 512, "hidden_size": 1536, "intermediate_size": 8960,
          "num_hidden_layers": 2, "num_attention_heads": 12, "num_key_value_heads": 2, "max_position_embeddings": 2048,
          "rope_theta": 1e6, "rms_norm_eps": 1e-6, "tie_word_embeddings": True}
_, _, spec = load_config(config)
torch.manual_seed(1)
weights = {}
for name, tensor in expected_tensors(spec).items():
    value = torch.randn(tensor.shape, device="cuda") * (tensor.shape[-1] ** -0.5 if tensor.kind == "matrix" else 0.05)
    weights[name] = value.bfloat16() if tensor.kind == "matrix" else value + (tensor.kind == "norm")
model = DecoderModel(spec, weights, torch.bfloat16, "cuda")
assert library.load().source_loaded("gemm_pairs") and library.load().source_loaded("decode_layers")
calls = []
product = ops.gated_product
ops.gated_product = lambda *given: calls.append(1) or product(*given)
rng = random.Random(1)
prompts = [[rng.randrange(512) for _ in range(1200)] for _ in range(3)]
logits, counts = {}, []
for graphs in (True, False):
    cache = CacheManager(cache_requirements(spec), CacheConfig(16, 80), model.dtype, "cuda", 2048, num_state_slots=2)
    runner = StepRunner(model, cache, 1280, 2, use_graphs=graphs)
    logits[graphs] = []
    for prompt in prompts:
        cache.create("r")
        logits[graphs].append(runner.run([StepEntry("r", prompt, [1199])]).clone())
        cache.free("r")
        counts.append(len(calls))
    if graphs:
        assert runner.portion_graph_replays == 2
assert counts == [0, 2, 2, 2, 2, 2], counts        # met first while a step is captured, of 1,280 rows, and replayed
for got, want in zip(logits[True], logits[False]):
    error = float((got - want).abs().max() / want.abs().max())
    assert error <= 2.0 ** -5, error
print("as launch by launch")
"""


def test_a_product_that_only_the_rows_of_a_captured_step_take():
    """A portion of 1,200 rows runs launch by launch at first, then captured with 1,280: only there are the rows enough for the product
    with its gate.  In a process of its own, without a warm-up, so that this is the product's first use."""
    import subprocess
    import sys
    from pathlib import Path

    run = subprocess.run([sys.executable, "-c", _ROUNDED_UP], capture_output=True, text=True, timeout=600, cwd=Path(__file__).parents[1])
    assert run.returncode == 0 and "as launch by launch" in run.stdout, run.stderr
