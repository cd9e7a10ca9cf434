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
    "two_heads": (192, 320, 4, 2, 528),
    "eight_heads": (256, 320, 16, 8, 528),
    "many_heads": (256, 320, 36, 36, 528),
    "square": (2560, 320, 2, 1, 2560),
}
CONTEXTS = [0, 1, 15, 16, 17, 31, 127, 128, 129, 300, 64, 5, 48, 200, 33, 3]


def _build(name, pairing="interleaved", layers=3):
    from llm_serving_engine_b200.config import load_config
    from llm_serving_engine_b200.models import DecoderModel, expected_tensors

    hidden, inter, n_q, n_kv, vocab = SIZES[name]
    config = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "vocab_size": vocab, "hidden_size": hidden, "head_dim": 128,
              "intermediate_size": inter, "num_hidden_layers": layers, "num_attention_heads": n_q, "num_key_value_heads": n_kv,
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


def _decode(model, sequences, steps, one_launch, use_graphs=False, launches=None):
    """Logits of the last ``steps`` tokens of every sequence, decoded together; the tokens before them come as portions.  The steps
    take the one launch where they are meant to and nowhere else: ``launches`` of it, by default one a step (with graphs: ahead of
    the capture and in it) or none."""
    from llm_serving_engine_b200.cache import CacheManager
    from llm_serving_engine_b200.config import CacheConfig
    from llm_serving_engine_b200.engine import StepEntry, StepRunner
    from llm_serving_engine_b200.kernels import ops
    from llm_serving_engine_b200.models import cache_requirements

    held, model._decode_layers = model._decode_layers, model._decode_layers if one_launch else None
    launch, calls = ops.decode_layers, []
    ops.decode_layers = lambda *given: calls.append(1) or launch(*given)
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
        calls.clear()
        for step in range(steps):
            entries = [StepEntry(str(index), [tokens[len(tokens) - steps + step]], [0]) for index, tokens in enumerate(sequences)]
            out.append(runner.run(entries).clone())
        if launches is None:
            launches = (2 if use_graphs else steps) if one_launch else 0
        assert len(calls) == launches
        return torch.stack(out, dim=1).cpu()      # [requests, steps, vocab]
    finally:
        model._decode_layers, ops.decode_layers = held, launch


@pytest.mark.parametrize("name,rows,first", [("small", 1, 0), ("small", 3, 1), ("small", 4, 4), ("small", 4, 8), ("odd", 1, 9), ("odd", 2, 2),
                                             ("odd", 4, 0), ("odd", 4, 6), ("wide", 1, 7), ("wide", 3, 3), ("wide", 4, 12)])
def test_against_the_plain_implementation(name, rows, first):
    from llm_serving_engine_b200.kernels import library

    config, model, weights = _build(name)
    assert model._decode_layers is not None and model._decode_layers.wanted(rows)
    rng = random.Random(rows)
    steps = 2
    sequences = [helpers.random_tokens(rng, config["vocab_size"], context + steps) for context in CONTEXTS[first:first + rows]]
    got = _decode(model, sequences, steps, True, use_graphs=rows == 3)
    assert library.load().lse_decode_layers_status() == 0
    repeated = _decode(model, sequences, steps, True)
    assert torch.equal(got, repeated)              # every sum has its order
    for index, tokens in enumerate(sequences):
        want = qwen2_plain.forward_full(config, weights, tokens)[-steps:]
        limit = helpers.tolerance("bfloat16", want)
        assert float((got[index] - want).abs().max()) <= limit, (name, rows, index)
        assert helpers.rms_ratio(got[index], want) <= helpers.RMS_RATIO["bfloat16"]      # largest measured: 7.2e-3


@pytest.mark.parametrize("name,rows", [("small", 4), ("odd", 3)])
def test_halves_turned_as_launch_by_launch(name, rows):
    config, model, _ = _build(name, "half")
    rng = random.Random(rows)
    sequences = [helpers.random_tokens(rng, config["vocab_size"], context + 1) for context in CONTEXTS[2:2 + rows]]
    got, want = (_decode(model, sequences, 1, one_launch) for one_launch in (True, False))
    assert float((got - want).abs().max()) <= helpers.tolerance("bfloat16", want)


def _plain_step(config, weights, kept, context, token):
    """Logits of ``token`` behind ``context`` cached keys and values (``kept``: [layers, 2, context, heads, 128], turned)."""
    n_q, n_kv, eps, positions = config["num_attention_heads"], config["num_key_value_heads"], config["rms_norm_eps"], torch.tensor([context])
    h = qwen2_plain.embedding(weights["model.embed_tokens.weight"], torch.tensor([token]))
    for index in range(config["num_hidden_layers"]):
        base = f"model.layers.{index}."
        x = qwen2_plain.rms_norm(h, weights[base + "input_layernorm.weight"], eps)
        q, k, v = (qwen2_plain.linear(x, weights[base + f"self_attn.{part}_proj.weight"], weights[base + f"self_attn.{part}_proj.bias"])
                   .view(1, -1, 128) for part in "qkv")
        q, k = (qwen2_plain.rope(part, positions, config["rope_theta"]) for part in (q, k))
        keys, values = torch.cat([kept[index, 0], k]), torch.cat([kept[index, 1], v])
        scores = torch.einsum("hgd,khd->hgk", q.view(n_kv, n_q // n_kv, 128), keys) / 128 ** 0.5
        out = torch.einsum("hgk,khd->hgd", scores.softmax(-1), values).reshape(1, n_q * 128)
        h = h + qwen2_plain.linear(out, weights[base + "self_attn.o_proj.weight"])
        h = h + qwen2_plain.swiglu(qwen2_plain.rms_norm(h, weights[base + "post_attention_layernorm.weight"], eps), weights, base + "mlp.")
    return qwen2_plain.linear(qwen2_plain.rms_norm(h, weights["model.norm.weight"], eps), weights["lm_head.weight"])[0]


# the ring (18 tiles) just filled and refilled, shares of many stages, one request's keys in more than ten shares and in as many as
# there may be, eight key/value heads, requests of very different lengths, a share of more tiles than are looked up ahead
@pytest.mark.parametrize("name,layers,contexts", [
    ("small", 3, [1280]), ("small", 3, [1281, 3072]), ("small", 3, [6912, 6913, 31, 7200]), ("two_heads", 3, [8192]),
    ("two_heads", 3, [30000]), ("two_heads", 2, [30000, 16]), ("eight_heads", 2, [4000, 3985]),
    ("eight_heads", 2, [6000, 129, 5999, 2650]), ("many_heads", 1, [17000, 20, 15, 33])])
def test_long_contexts(name, layers, contexts, monkeypatch):
    """Against the plain implementation and launch by launch.  The cached keys are large enough (scores of a spread of two) that some
    hundreds of them carry the result: a share that is lost or read twice moves it by a tenth and more.  Such scores carry the
    queries' rounding to bfloat16 (2^-9) into the probabilities a few times over, whichever way the step runs: hence the wider of
    the two bounds."""
    from llm_serving_engine_b200.cache import CacheManager
    from llm_serving_engine_b200.config import CacheConfig
    from llm_serving_engine_b200.engine import StepEntry, StepRunner
    from llm_serving_engine_b200.kernels import library, ops
    from llm_serving_engine_b200.models import cache_requirements

    config, model, weights = _build(name, layers=layers)
    n_kv, rows = config["num_key_value_heads"], len(contexts)
    assert model._decode_layers is not None and model._decode_layers.wanted(rows)
    generator = torch.Generator().manual_seed(sum(contexts))
    spread = torch.tensor([4.0, 1.0]).view(1, 2, 1, 1, 1)
    kept = [(torch.randn((layers, 2, context, n_kv, 128), generator=generator) * spread).bfloat16() for context in contexts]
    tokens = [7 + index for index in range(rows)]
    pages = sum(-(-(context + 1) // 16) for context in contexts)
    calls = []
    launch = ops.decode_layers
    monkeypatch.setattr(ops, "decode_layers", lambda *given: calls.append(1) or launch(*given))

    def run():
        cache = CacheManager(cache_requirements(model.spec), CacheConfig(16, pages), model.dtype, "cuda", 40000, num_state_slots=rows)
        cache.groups[0].storage.fill_(float("nan"))
        runner = StepRunner(model, cache, max_tokens_per_step=rows, max_segments=rows, use_graphs=False)
        for index, context in enumerate(contexts):
            cache.create(str(index))
            cache.reserve(str(index), context)
            slots = torch.from_numpy(cache.slot_mapping(0, str(index), 0, context)).cuda().long()
            for position in range(layers):
                view = cache.layer_view(position)
                view.keys[slots // 16, :, slots % 16] = kept[index][position, 0].cuda()
                view.values[slots // 16, :, slots % 16] = kept[index][position, 1].cuda()
        return runner.run([StepEntry(str(index), [token], [0]) for index, token in enumerate(tokens)]).cpu()

    got, again = run(), run()
    assert len(calls) == 2 and library.load().lse_decode_layers_status() == 0
    assert torch.equal(got, again)
    model._decode_layers = None
    chain = run()
    assert len(calls) == 2
    for index, (context, token) in enumerate(zip(contexts, tokens)):
        want = _plain_step(config, weights, kept[index].float(), context, token)
        limit = helpers.tolerance("bfloat16", want)
        for answer in (got[index], chain[index]):
            assert float((answer - want).abs().max()) <= limit, (context, "one launch" if answer is got[index] else "launch by launch")
            assert helpers.rms_ratio(answer[None], want[None]) <= helpers.RMS_RATIO_LARGE_LAYERS


@pytest.mark.parametrize("keys", [slice(256, 384), slice(300, 301), slice(0, 1280), slice(1279, 1280), slice(1280, 1280)])
@pytest.mark.parametrize("what", ["keys", "values"])
def test_nan_in_the_cache_reaches_the_logits(keys, what):
    """As launch by launch: a share of the keys all of whose scores are NaN, a single such key, all of them, none; the same in the
    values."""
    from llm_serving_engine_b200.cache import CacheManager
    from llm_serving_engine_b200.config import CacheConfig
    from llm_serving_engine_b200.engine import StepEntry, StepRunner
    from llm_serving_engine_b200.models import cache_requirements

    _, model, _ = _build("small", layers=1)
    kept = torch.randn(1280, 128, generator=torch.Generator().manual_seed(2)).bfloat16().cuda()
    found = []
    for one_launch in (True, False):
        if not one_launch:
            model._decode_layers = None
        cache = CacheManager(cache_requirements(model.spec), CacheConfig(16, 81), model.dtype, "cuda", 2048, num_state_slots=1)
        cache.create("a")
        cache.reserve("a", 1280)
        slots = torch.from_numpy(cache.slot_mapping(0, "a", 0, 1280)).cuda().long()
        view = cache.layer_view(0)
        for tensor in (view.keys, view.values):
            tensor[slots // 16, 0, slots % 16] = kept
        poisoned = view.keys if what == "keys" else view.values
        poisoned[slots[keys] // 16, 0, slots[keys] % 16] = float("nan")
        found.append(StepRunner(model, cache, 1, 1, use_graphs=False).run([StepEntry("a", [5], [0])]).isnan().cpu())
    assert torch.equal(found[0], found[1]) and bool(found[0].all()) == (keys.stop > keys.start)


@pytest.mark.parametrize("one_launch", [True, False])
def test_the_head_reads_rows_that_were_rounded_once(one_launch):
    """Branches that add nothing and a head that is the identity: the logits are the normed embeddings as the product reads them,
    float32 up to one rounding to bfloat16.  Float32's own rounding (a few 2^-24) puts a value on the other side of a bfloat16
    boundary once in 2^13: 5 of the 40,960 values here.  Sixteen bits on the way (2^-18 on average) would do so once in 2^9.5."""
    config, model, weights = _build("square", layers=1)
    block = model.blocks[0]
    block.mixer.o_weight.zero_()
    block.feed_forward.down_weight.zero_()
    model.lm_head.copy_(torch.eye(2560))
    model.final_norm.weight.copy_(1.0 + 0.3 * torch.randn(2560, generator=torch.Generator().manual_seed(3)))
    rng = random.Random(3)
    sequences = [helpers.random_tokens(rng, config["vocab_size"], 4) for _ in range(4)]
    got = _decode(model, sequences, 4, one_launch)
    rows = weights["model.embed_tokens.weight"][torch.tensor(sequences)].double()
    want = rows * (rows.pow(2).mean(-1, keepdim=True) + config["rms_norm_eps"]).rsqrt() * model.final_norm.weight.cpu().double()
    assert int((got != want.bfloat16().float()).sum()) <= 16


def test_the_parts_are_read_as_they_are(monkeypatch):
    """A matrix that takes another's place is used by the next step, and a part that was wrapped, on the instance or on its class, is
    called: the one launch keeps nothing of the layers as they were built."""
    from llm_serving_engine_b200.parts.mlp import SwiGLU

    config, model, _ = _build("small")
    passed = []
    sequences = [[3], [8]]
    before = _decode(model, sequences, 1, True)
    ff = model.blocks[1].feed_forward
    ff.down_weight = (torch.randn(ff.down_weight.shape, generator=torch.Generator().manual_seed(9)) * 0.1).bfloat16().cuda()
    got, want = (_decode(model, sequences, 1, one_launch) for one_launch in (True, False))
    limit = helpers.tolerance("bfloat16", want)
    assert float((got - want).abs().max()) <= limit < float((got - before).abs().max())

    mixer = model.blocks[2].mixer
    whole = mixer.forward
    mixer.forward = lambda *given: passed.append("instance") or whole(*given)
    assert torch.equal(_decode(model, sequences, 1, True, launches=0), want) and passed == ["instance"]
    del mixer.forward
    act = SwiGLU.forward
    monkeypatch.setattr(SwiGLU, "forward", lambda self, x: passed.append("class") or act(self, x))
    assert torch.equal(_decode(model, sequences, 1, True, launches=0), want) and passed[1:] == ["class"] * 3
    monkeypatch.setattr(SwiGLU, "forward", act)
    assert torch.equal(_decode(model, sequences, 1, True), got)


def test_a_launch_that_is_refused_goes_launch_by_launch(monkeypatch):
    """The step's result is that of the kernels one by one, and the launch is not tried again."""
    from llm_serving_engine_b200.kernels import library, ops

    _, model, _ = _build("small")
    asked = []
    want = _decode(model, [[3], [8]], 1, False)
    monkeypatch.setattr(library.load(), "lse_decode_layers", lambda *given: asked.append(1) or ops.DECODE_LAYERS_REFUSED)
    for use_graphs in (False, True):
        assert torch.equal(_decode(model, [[3], [8]], 1, True, use_graphs, launches=0 if use_graphs else 1), want)
    assert len(asked) == 1


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


@pytest.mark.parametrize("name,rows,layers", [("small", 1, 3), ("odd", 4, 2)])
def test_a_wait_that_runs_out_is_reported_and_the_kernel_returns(name, rows, layers):
    """A value that the first product waits for does not come, and the waits give up after a few thousand attempts: the blocks that
    wait for it, those that wait for what these would have made, and the warps whose ring nobody empties.  The launch ends, its
    status word reaches the host as the sampler reads it, and after a reset the next step is right.  Nothing faults: a value is
    simply not written."""
    from llm_serving_engine_b200.kernels import library, ops
    from llm_serving_engine_b200.sampling.sampler import GenerationConfig, Sampler

    config, model, _ = _build(name, layers=layers)
    sequences = [[5 + index, 9] for index in range(rows)]
    want = _decode(model, sequences, 1, True)
    sampler = Sampler(config["vocab_size"], rows, torch.device("cuda"))
    ops.decode_layers_test_hooks(spin_limit=2000, withhold=True)
    try:
        broken = _decode(model, sequences, 1, True)[:, 0].cuda()
        assert library.load().lse_decode_layers_status() == 1
        ticket = sampler.launch(broken, [GenerationConfig() for _ in range(rows)], [0] * rows)
        with pytest.raises(ops.KernelError, match="the decode step"):
            sampler.collect(ticket)
    finally:
        ops.decode_layers_test_hooks()
        ops.kernel_status_reset()
    assert torch.equal(_decode(model, sequences, 1, True), want)
    assert library.load().lse_decode_layers_status() == 0
