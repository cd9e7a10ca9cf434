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
    """A windowed and a full latent layer, keys and values bounded so that the full layer makes its own up to 128 keys only: the
    second portions of two requests capture the step, the later portions of a third have the windowed layer's buffer of the same
    size, but a full layer that goes over the latent rows.  Every logit against the latent rows' kernel launch by launch."""
    model = latent_model([64, 0], heads=2, rank=64, device="cuda", scale=0.07)
    generator = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, 64, (length,), generator=generator).tolist() for length in (128, 128, 448)]
    plain = runner_for(model, use_graphs=False)
    monkeypatch.setattr(latent_attention, "LATENT_FLOPS", 1.0e30)      # never worth it
    want = [in_portions(plain, "r", tokens, 64) for tokens in prompts]
    monkeypatch.setattr(latent_attention, "LATENT_FLOPS", 1.0)         # always worth it, where it fits
    monkeypatch.setattr(latent_attention, "EXPAND_MAX_BYTES", 2 * 128 * model.blocks[0].mixer.kv_up.shape[0])
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
