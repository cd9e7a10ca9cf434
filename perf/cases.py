"""Timed cases of the engine, over the range that it is used for.

Three kinds, each through entry points that a program of this package calls:

* ``step``: one ``StepRunner.run`` of a Qwen2 model (what ``LLMEngine`` and the trace replay do for every step): host
  packing, the upload, the CUDA graph, the logits.  The requests are taken back by the step's tokens first, so that
  every pass is the same step.
* ``block``: one decoder layer (norm, attention, norm, feed-forward and the norm that adds its output) over the rows of a
  step, launch by launch, as ``DecoderModel.forward`` runs a step beyond the graphs' size classes.
* ``part``: one mixer or feed-forward of the other designs over a prompt's rows.

Requests of a case are written "context+tokens" (tokens of this step behind a cached context), "xN" for N of them, with
contexts spread from half to one and a half times the number when ``ragged`` is set.  Weights are N(0, 0.02) like the
package's random models, queries' and keys' N(0, 0.03), so that attention is neither flat nor one-hot.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from llm_serving_engine_b200.cache import CacheManager
from llm_serving_engine_b200.config import CacheConfig, load_config
from llm_serving_engine_b200.config.model_config import LayerSpec, ModelSpec, PartSpec
from llm_serving_engine_b200.engine import StepEntry, StepRunner
from llm_serving_engine_b200.models import DecoderModel, cache_requirements, expected_tensors, parse_dtype
from llm_serving_engine_b200.parts import FEED_FORWARDS
from llm_serving_engine_b200.parts.base import BuildContext, ResidualStream

# Layer sizes of Qwen2.5 models, as the repository's benchmark has them.
SIZES = {
    "1.5b": {"hidden_size": 1536, "intermediate_size": 8960, "num_attention_heads": 12, "num_key_value_heads": 2,
             "vocab_size": 151936, "tie_word_embeddings": True, "rms_norm_eps": 1e-6},
    "7b": {"hidden_size": 3584, "intermediate_size": 18944, "num_attention_heads": 28, "num_key_value_heads": 4,
           "vocab_size": 152064, "tie_word_embeddings": False, "rms_norm_eps": 1e-6},
    "14b": {"hidden_size": 5120, "intermediate_size": 13824, "num_attention_heads": 40, "num_key_value_heads": 8,
            "vocab_size": 152064, "tie_word_embeddings": False, "rms_norm_eps": 1e-5},
}
THETA, PAGE, HEAD = 1000000.0, 16, 128
MAX_POSITIONS = 16384
EPS = 1e-5


def listed() -> list[dict]:
    return [
        # one user's chat turn: the smallest step, all launches and latency (the whole model)
        {"name": "decode_1", "kind": "step", "size": "1.5b", "layers": 28, "dtype": "bfloat16", "requests": "100+1", "ragged": False},
        # the benchmark's headline: eight requests of 2,048 tokens decoding (the whole model)
        {"name": "decode_8", "kind": "step", "size": "1.5b", "layers": 28, "dtype": "bfloat16", "requests": "2048+1x8", "ragged": False},
        # a full batch of requests at different lengths decoding: four layers and the head
        {"name": "decode_64", "kind": "step", "size": "1.5b", "layers": 4, "dtype": "bfloat16", "requests": "1900+1x64", "ragged": True},
        # short prompts in portions of 32, eight at a time: four layers and the head
        {"name": "portions_8x32", "kind": "step", "size": "1.5b", "layers": 4, "dtype": "bfloat16", "requests": "96+32x8", "ragged": False},
        # the true 32-bit path decoding (checks of a checkpoint, short evaluations): four layers and the head
        {"name": "decode_8_float32", "kind": "step", "size": "1.5b", "layers": 4, "dtype": "float32", "requests": "700+1x8", "ragged": True},
        # a layer over the benchmark's 2,048-token prompt
        {"name": "prompt_2048", "kind": "block", "size": "1.5b", "dtype": "bfloat16", "requests": "0+2048", "ragged": False},
        # a larger model under mixed traffic: a portion late in a long prompt, a short prompt, requests that decode
        {"name": "mixed_7b", "kind": "block", "size": "7b", "dtype": "bfloat16", "requests": "8000+1024 0+301 1500+1x24", "ragged": True},
        # the true 32-bit path over a prompt of odd length
        {"name": "prompt_777_float32", "kind": "block", "size": "1.5b", "dtype": "float32", "requests": "0+777", "ragged": False},
        # a mixture of eight experts with a shared one over a prompt portion
        {"name": "experts_2048", "kind": "part", "part": "experts", "width": 2048, "heads": 16, "dtype": "bfloat16", "rows": 2048},
        # linear attention with a decay per head over a prompt
        {"name": "linear_attention_2048", "kind": "part", "part": "linear", "width": 2048, "heads": 16, "dtype": "bfloat16", "rows": 2048},
        # attention over a cached latent, over a prompt
        {"name": "latent_attention_2048", "kind": "part", "part": "latent", "width": 2048, "heads": 16, "dtype": "bfloat16", "rows": 2048},
        # a matrix memory that writes differences, over a short prompt of odd length
        {"name": "delta_memory_501", "kind": "part", "part": "delta", "width": 2048, "heads": 16, "dtype": "bfloat16", "rows": 501},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_one(rng) -> dict:
    kind = rng.choice(["decode", "decode", "decode", "portions", "portions", "prompt", "prompt", "mixed", "part", "part"])
    dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
    size = rng.choice(["1.5b", "1.5b", "7b", "14b"])
    if kind == "decode":
        return {"kind": "step", "size": size, "layers": rng.randint(2, 4), "dtype": dtype,
                "requests": f"{_log(rng, 8, 4000)}+1x{_log(rng, 1, 64)}", "ragged": True}
    if kind == "portions":
        return {"kind": "step", "size": size, "layers": rng.randint(2, 4), "dtype": dtype,
                "requests": f"{_log(rng, 8, 4000)}+{_log(rng, 4, 128)}x{_log(rng, 1, 8)}", "ragged": True}
    if kind == "prompt":
        return {"kind": "block", "size": size, "dtype": dtype, "requests": f"0+{_log(rng, 100, 2048)}", "ragged": False}
    if kind == "mixed":
        return {"kind": "block", "size": size, "dtype": dtype, "ragged": True,
                "requests": f"{_log(rng, 100, 8000)}+{_log(rng, 64, 1024)} 0+{_log(rng, 16, 400)} {_log(rng, 50, 2000)}+1x{_log(rng, 2, 32)}"}
    # the designs' parts, from a short prompt to a long one; the experts are grouped from 128 rows on
    return {"kind": "part", "part": rng.choice(["experts", "linear", "latent", "delta"]), "width": 2048, "heads": 16,
            "dtype": "bfloat16", "rows": _log(rng, 130, 2300)}


def _cost(case: dict) -> float:
    """A bound on a pass, in units of time: a 32-bit operation counts thirty times a 16-bit one."""
    need = work(case)
    return need["flops"] * (30.0 if case["dtype"] == "float32" else 1.0) / 1.5e15 + need["bytes"] / 6.5e12


def draw(rng) -> dict:
    most = max(_cost(case) for case in listed())
    while True:
        case = _draw_one(rng)
        if _cost(case) <= most:
            return case


# ---------------------------------------------------------------------------------------------- inputs
def _requests(case: dict) -> list[tuple[int, int]]:
    """(cached context, tokens of this step) of every request."""
    out = []
    for group in case["requests"].split():
        context, rest = group.split("+")
        tokens, _, count = rest.partition("x")
        context, tokens, count = int(context), int(tokens), int(count or 1)
        for index in range(count):
            scale = 0.5 + index / (count - 1) if case["ragged"] and count > 1 else 1.0
            out.append((int(context * scale), tokens))
    return out


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(generator, shape, std: float, dtype=torch.float32) -> torch.Tensor:
    return (torch.randn(shape, generator=generator, device="cuda", dtype=torch.float32) * std).to(dtype)


def _qwen_config(case: dict) -> dict:
    return {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": case.get("layers", 1),
            "max_position_embeddings": MAX_POSITIONS, "rope_theta": THETA, "attention_bias": True, **SIZES[case["size"]]}


def _qwen_inputs(case: dict, seed: int) -> dict:
    """Weights, the cached keys and values of every request ([layers, 2, sum of contexts, kv heads, head size]) and the
    step's tokens or rows."""
    size, compute, generator = SIZES[case["size"]], parse_dtype(case["dtype"]), _generator(seed)
    layers, hidden, inter = case.get("layers", 1), size["hidden_size"], size["intermediate_size"]
    n_q, n_kv, vocab = size["num_attention_heads"] * HEAD, size["num_key_value_heads"] * HEAD, size["vocab_size"]
    weights = {}
    for index in range(layers):
        prefix = f"model.layers.{index}."
        for name, shape, std in (("self_attn.q_proj", (n_q, hidden), 0.03), ("self_attn.k_proj", (n_kv, hidden), 0.03),
                                 ("self_attn.v_proj", (n_kv, hidden), 0.02), ("self_attn.o_proj", (hidden, n_q), 0.02),
                                 ("mlp.gate_proj", (inter, hidden), 0.02), ("mlp.up_proj", (inter, hidden), 0.02),
                                 ("mlp.down_proj", (hidden, inter), 0.02)):
            weights[prefix + name + ".weight"] = _normal(generator, shape, std, compute)
        for name, rows in (("q", n_q), ("k", n_kv), ("v", n_kv)):
            weights[prefix + f"self_attn.{name}_proj.bias"] = _normal(generator, (rows,), 0.02)
        for name in ("input_layernorm", "post_attention_layernorm"):
            weights[prefix + name + ".weight"] = 1.0 + _normal(generator, (hidden,), 0.05)
    weights["model.norm.weight"] = 1.0 + _normal(generator, (hidden,), 0.05)
    if case["kind"] == "step":
        weights["model.embed_tokens.weight"] = _normal(generator, (vocab, hidden), 0.02, compute)
        if not size["tie_word_embeddings"]:
            weights["lm_head.weight"] = _normal(generator, (vocab, hidden), 0.02, compute)
    requests = _requests(case)
    rows, cached = sum(count for _, count in requests), sum(context for context, _ in requests)
    kv = _normal(generator, (layers, 2, cached, size["num_key_value_heads"], HEAD), 1.0, compute)
    return {"weights": weights, "requests": requests, "kv": kv,
            "tokens": torch.randint(0, vocab, (rows,), generator=generator, device="cuda"),
            "rows": _normal(generator, (rows, hidden), 1.0)}


def _experts_sizes(case: dict) -> tuple[int, int, int, int]:
    """Experts, chosen ones, columns of an expert and of the shared expert: a token's work is a dense layer's of 4 x width."""
    ff = (4 * case["width"] // 3) // 64 * 64
    return 8, 2, ff, 4 * case["width"] - 2 * ff


def _part(case: dict) -> tuple[str, dict, dict]:
    """Kind, parameters and tensor shapes (with the values' spread) of a part."""
    width, heads, dim = case["width"], case["heads"], 128
    if case["part"] == "experts":
        experts, top, ff, shared = _experts_sizes(case)
        params = {"experts": experts, "top": top, "ff": ff, "limit": 7.0, "correction": False, "shared": {"ff": shared, "limit": 7.0}}
        shapes = {"router": ((experts, width), 0.02), "shared.sg": ((1, width), 0.02)}
        for prefix, columns in [(f"e{index}.", ff) for index in range(experts)] + [("shared.", shared)]:
            shapes.update({prefix + "gate": ((columns, width), 0.02), prefix + "up": ((columns, width), 0.02),
                           prefix + "down": ((width, columns), 0.02)})
        return "clamped_moe", params, shapes
    if case["part"] == "linear":
        params = {"heads": heads, "dim": dim, "vdim": dim, "eps": EPS,
                  "decay": [1.0 - 2.0 ** -(3 + 5 * head / max(heads - 1, 1)) for head in range(heads)]}
        shapes = {name: ((heads * dim, width), 0.02) for name in ("q", "k", "v", "g")}
        shapes.update({"o": ((width, heads * dim), 0.02), "norm": ((heads * dim,), 0.05)})
        return "decayed_linear_attention", params, shapes
    if case["part"] == "latent":
        params = {"heads": heads, "dim": dim, "rot_dim": 64, "vdim": dim, "kv_rank": 512, "scale": 192 ** -0.5, "eps": EPS,
                  "rot": {"base": 500000.0, "dims": 64}}
        shapes = {"q": ((heads * 192, width), 0.03), "dkv": ((576, width), 0.03), "dkv.norm": ((512,), 0.05),
                  "uk": ((heads * dim, 512), 0.05), "uv": ((heads * dim, 512), 0.05), "o": ((width, heads * dim), 0.02)}
        return "latent_attention", params, shapes
    params = {"heads": heads, "kv_heads": heads // 2, "dim": dim, "vdim": dim, "conv": 4, "decay_rank": 64, "gate_rank": 64,
              "eps": EPS}
    shapes = {}
    for name, rows in (("q", heads // 2 * dim), ("k", heads // 2 * dim), ("v", heads * dim)):
        shapes.update({name: ((rows, width), 0.02), name + ".conv": ((rows, 4), 0.3)})
    shapes.update({"b": ((heads, width), 0.02), "A_log": ((heads,), 0.02), "norm": ((dim,), 0.05), "a1": ((64, width), 0.02),
                   "a2": ((heads * dim, 64), 0.02), "dt_bias": ((heads * dim,), 0.02), "g1": ((64, width), 0.02),
                   "g2": ((heads * dim, 64), 0.02), "o": ((width, heads * dim), 0.02)})
    return "channel_delta_memory", params, shapes


_VECTORS = ("norm", "dkv.norm", "A_log", "dt_bias", "q.conv", "k.conv", "v.conv")    # held in 32 bits, as a loader holds them


def _part_inputs(case: dict, seed: int) -> tuple[dict, torch.Tensor]:
    generator, compute = _generator(seed), parse_dtype(case["dtype"])
    weights = {}
    for name, (shape, std) in _part(case)[2].items():
        weights[name] = _normal(generator, shape, std, torch.float32 if name in _VECTORS else compute)
        if name.endswith("norm"):
            weights[name] += 1.0
    return weights, _normal(generator, (case["rows"], case["width"]), 1.0, compute)


def _runner(model, requests: list[tuple[int, int]], max_positions: int) -> StepRunner:
    """A step runner with a cache that holds the requests, each already ``context`` tokens long."""
    pages = sum(-(-(context + count) // PAGE) for context, count in requests) + 1
    cache = CacheManager(cache_requirements(model.spec), CacheConfig(PAGE, pages), model.dtype, "cuda", max_positions,
                         num_state_slots=len(requests))
    rows = sum(count for _, count in requests)
    runner = StepRunner(model, cache, max_tokens_per_step=rows, max_segments=len(requests))
    for index, (context, _) in enumerate(requests):
        cache.create(str(index))
        if context:
            cache.reserve(str(index), context)
    return runner


# ---------------------------------------------------------------------------------------------- passes
def prepare(case: dict, seed: int) -> dict:
    if case["kind"] == "part":
        return _prepare_part(case, seed)
    inputs = _qwen_inputs(case, seed)
    config = _qwen_config(case)
    _, _, spec = load_config(config)
    weights = inputs["weights"]
    if case["kind"] == "block":     # the layer alone: rows come in where an embedding would leave them
        weights = dict(weights, **{"model.embed_tokens.weight": torch.zeros((1, config["hidden_size"]), device="cuda")})
        weights["lm_head.weight"] = weights["model.embed_tokens.weight"]
    model = DecoderModel(spec, weights, parse_dtype(case["dtype"]), "cuda")
    requests = inputs["requests"]
    runner = _runner(model, requests, MAX_POSITIONS)
    slots = [runner.cache.slot_mapping(0, str(index), 0, context) for index, (context, _) in enumerate(requests) if context]
    if slots:
        flat = torch.cat([torch.from_numpy(part) for part in slots]).to("cuda").long()
        for position in range(len(spec.order)):
            view = runner.cache.layer_view(position)
            view.keys[flat // PAGE, :, flat % PAGE] = inputs["kv"][position, 0]
            view.values[flat // PAGE, :, flat % PAGE] = inputs["kv"][position, 1]
    tokens, entries, at = inputs["tokens"].tolist(), [], 0
    for index, (_, count) in enumerate(requests):
        entries.append(StepEntry(str(index), tokens[at:at + count], [count - 1]))
        at += count
    state = {"kind": case["kind"], "model": model, "runner": runner, "entries": entries}
    if case["kind"] == "step":
        for _ in range(2):          # what a server's warm-up does: the step's graph is captured
            run(state)
    else:
        state["step"], state["caches"] = runner.prepare(entries)
        state["rows"] = inputs["rows"]
    return state


def _prepare_part(case: dict, seed: int) -> dict:
    weights, x = _part_inputs(case, seed)
    kind, params, _ = _part(case)
    compute = parse_dtype(case["dtype"])
    if case["part"] == "experts":
        ctx = BuildContext(compute, torch.device("cuda"), case["width"], 0, MAX_POSITIONS)
        return {"kind": "experts", "part": FEED_FORWARDS.get(kind)(params, weights, ctx), "x": x}
    norm = PartSpec("rmsnorm", {"eps": EPS})
    layer = LayerSpec(prefix="l0.", block=PartSpec("residual_streams", {"feed_forward": False}), mixer=PartSpec(kind, params),
                      feed_forward=None, mixer_norm=norm, feed_forward_norm=None)
    spec = ModelSpec(architecture="one layer", vocab_size=16, hidden_size=case["width"], layers=(layer,), order=(0,), final_norm=norm,
                     embedding_name="embed", final_norm_prefix="final.", lm_head_name="head", tie_word_embeddings=True,
                     max_position_embeddings=MAX_POSITIONS)
    given = {"l0.mixer." + name: tensor for name, tensor in weights.items()}
    for name, tensor in expected_tensors(spec).items():
        if name not in given:
            given[name] = torch.ones(tensor.shape, device="cuda", dtype=compute if tensor.kind == "matrix" else torch.float32)
    model = DecoderModel(spec, given, compute, "cuda")
    runner = _runner(model, [(0, case["rows"])], MAX_POSITIONS)
    step, caches = runner.prepare([StepEntry("0", [0] * case["rows"])])
    return {"kind": "mixer", "mixer": model.blocks[0].mixer, "x": x, "step": step, "caches": caches, "cache": runner.cache,
            "states": runner.cache.snapshot_states(), "model": model, "runner": runner}


def run(state: dict):
    kind = state["kind"]
    if kind == "step":
        runner = state["runner"]
        for entry in state["entries"]:     # the request as it was before this step
            request = runner.cache.requests[entry.request_id]
            if state.get("ran"):
                request.length -= len(entry.tokens)
        state["ran"] = True
        return {"logits": runner.run(state["entries"])}
    if kind == "block":
        model, stream = state["model"], ResidualStream(state["rows"].clone())
        state["model"].blocks[0].forward(stream, state["step"], state["caches"][0])
        normed = model.final_norm.forward(stream)
        return {"normed": normed, "residual": stream.residual, "cache": state["runner"].cache.groups[0].storage}
    if kind == "experts":
        return {"out": state["part"].forward(state["x"])}
    state["cache"].restore_states(state["states"])     # a new request: its state is zero
    out = {"out": state["mixer"].forward(state["x"], state["step"], state["caches"][0])}
    tensors = state["cache"].states.tensors
    for index, key in enumerate(sorted(tensors, key=str)):
        out[f"state{index}"] = tensors[key]
    return out


# ---------------------------------------------------------------------------------------------- work, tolerance
def work(case: dict) -> dict:
    width_of = 4.0 if case["dtype"] == "float32" else 2.0
    if case["kind"] == "part":
        rows, width, heads = case["rows"], case["width"], case["heads"]
        held = sum(math.prod(shape) for shape, _ in _part(case)[2].values())
        flops = 2.0 * rows * held
        if case["part"] == "experts":
            experts, top, ff, _ = _experts_sizes(case)
            flops -= 2.0 * rows * 3 * width * ff * (experts - top)
        elif case["part"] == "linear":       # a state updated and read for every token
            flops += rows * heads * 128 * 128 * 4.0
        elif case["part"] == "latent":       # causal scores and sums over keys of 192 and values of 128
            flops += rows * (rows + 1) / 2 * heads * (192 + 128) * 2.0
        else:
            flops += rows * heads * 128 * 128 * 7.0
        return {"bytes": width_of * (held + 2 * rows * width), "flops": flops}
    size = SIZES[case["size"]]
    hidden, inter, layers = size["hidden_size"], size["intermediate_size"], case.get("layers", 1)
    n_q, n_kv = size["num_attention_heads"] * HEAD, size["num_key_value_heads"] * HEAD
    matrices = hidden * (n_q + 2 * n_kv) + n_q * hidden + 3 * hidden * inter
    requests = _requests(case)
    rows = sum(count for _, count in requests)
    keys = sum(context + count for context, count in requests)
    pairs = sum(count * context + count * (count + 1) / 2 for context, count in requests)
    flops = layers * (2.0 * rows * matrices + 4.0 * pairs * n_q)
    moved = layers * width_of * (matrices + 2 * n_kv * keys)
    if case["kind"] == "step":
        flops += 2.0 * len(requests) * hidden * size["vocab_size"]
        moved += width_of * hidden * size["vocab_size"] + 4.0 * len(requests) * size["vocab_size"]
    else:
        moved += rows * hidden * (4.0 + 4.0 + width_of)
    return {"bytes": moved, "flops": flops}


def tolerance(case: dict) -> dict:
    """A few times what a correct implementation at the same precision is off ``exact`` by: measured 5e-7 to 8e-6 in 32 bits
    (the rotation's angles at high positions), 2.7e-2 over 28 layers in bfloat16, 1.5e-2 over four, 2e-3 to 7e-3 for a layer."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    if case["kind"] == "step":
        return {"rel": 6e-2 if case["layers"] > 4 else 3e-2}
    return {"rel": 1.5e-2}


# ---------------------------------------------------------------------------------------------- 64 bits, plain torch
def _rms(x, weight, eps):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps) * weight


def _rotate(x, positions, base: float):
    """Neighbouring pairs (2i, 2i + 1) of the last axis turned by position * base^(-2i / D); x [T, heads, D]."""
    dim = x.shape[-1]
    # the frequencies as the model holds them: 32-bit numbers
    freq = (1.0 / (base ** (torch.arange(0, dim, 2, device=x.device).float() / dim))).double()
    angle = positions.double()[:, None] * freq[None]
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    even, odd = x[..., 0::2], x[..., 1::2]
    return torch.stack([even * cos - odd * sin, even * sin + odd * cos], dim=-1).flatten(-2)


def _attend(q, k, v, first: int, scale: float):
    """q [T, heads, D] of positions first .. on k [S, kv heads, D], v [S, kv heads, E]; causal."""
    tokens, heads, _ = q.shape
    group = heads // k.shape[1]
    hidden = torch.arange(k.shape[0], device=q.device)[None] > torch.arange(first, first + tokens, device=q.device)[:, None]
    out = torch.empty((tokens, heads, v.shape[2]), dtype=q.dtype, device=q.device)
    for head in range(heads):
        scores = (q[:, head] @ k[:, head // group].t()) * scale
        out[:, head] = torch.softmax(scores.masked_fill(hidden, -math.inf), dim=-1) @ v[:, head // group]
    return out


def _exact_layer(h, weights, prefix: str, size: dict, requests, kv):
    n_q, n_kv, eps = size["num_attention_heads"], size["num_key_value_heads"], size["rms_norm_eps"]

    def matrix(name):
        return weights[prefix + name].double()

    x = _rms(h, matrix("input_layernorm.weight"), eps)
    q, k, v = ((x @ matrix(f"self_attn.{name}_proj.weight").t() + matrix(f"self_attn.{name}_proj.bias")).view(len(x), -1, HEAD)
               for name in "qkv")
    out = torch.empty((len(x), n_q, HEAD), dtype=x.dtype, device=x.device)
    row = cached = 0
    for context, count in requests:
        positions = torch.arange(context, context + count, device=x.device)
        mine = slice(row, row + count)
        keys = torch.cat([kv[0, cached:cached + context].double(), _rotate(k[mine], positions, THETA)])
        values = torch.cat([kv[1, cached:cached + context].double(), v[mine]])
        out[mine] = _attend(_rotate(q[mine], positions, THETA), keys, values, context, HEAD ** -0.5)
        row, cached = row + count, cached + context
    h = h + out.view(len(x), n_q * HEAD) @ matrix("self_attn.o_proj.weight").t()
    x = _rms(h, matrix("post_attention_layernorm.weight"), eps)
    gate, up = x @ matrix("mlp.gate_proj.weight").t(), x @ matrix("mlp.up_proj.weight").t()
    return h + (F.silu(gate) * up) @ matrix("mlp.down_proj.weight").t()


def exact(case: dict, seed: int):
    if case["kind"] == "part":
        weights, x = _part_inputs(case, seed)
        return _EXACT_PARTS[case["part"]](case, {name: tensor.double() for name, tensor in weights.items()}, x.double())
    inputs, size = _qwen_inputs(case, seed), SIZES[case["size"]]
    weights, requests = inputs["weights"], inputs["requests"]
    h = weights["model.embed_tokens.weight"][inputs["tokens"]].double() if case["kind"] == "step" else inputs["rows"].double()
    for index in range(case.get("layers", 1)):
        h = _exact_layer(h, weights, f"model.layers.{index}.", size, requests, inputs["kv"][index])
    normed = _rms(h, weights["model.norm.weight"].double(), size["rms_norm_eps"])
    if case["kind"] == "block":
        return {"normed": normed, "residual": h, "cache": None}    # pages lie where the cache manager put them
    last = torch.cumsum(torch.tensor([count for _, count in requests]), 0) - 1
    head = weights["model.embed_tokens.weight" if size["tie_word_embeddings"] else "lm_head.weight"]
    return {"logits": normed[last.to("cuda")] @ head.double().t()}


def _exact_experts(case, w, x):
    experts, top, _, _ = _experts_sizes(case)

    def expert(prefix, rows):
        gate = (rows @ w[prefix + "gate"].t()).clamp(max=7.0)
        up = (rows @ w[prefix + "up"].t()).clamp(-7.0, 7.0)
        return (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ w[prefix + "down"].t()

    scores = torch.softmax(x @ w["router"].t(), dim=-1)
    chosen = torch.topk(scores, top, dim=-1).indices
    y = expert("shared.", x) * torch.sigmoid(x @ w["shared.sg"].t())
    for index in range(experts):
        rows = (chosen == index).any(-1).nonzero()[:, 0]
        y[rows] += scores[rows, index, None] * expert(f"e{index}.", x[rows])
    return {"out": y}


def _exact_linear(case, w, x):
    rows, heads, dim = case["rows"], case["heads"], 128
    params = _part(case)[1]
    q, k, v = (F.silu(x @ w[name].t()).view(rows, heads, dim) for name in "qkv")
    out, state = torch.empty_like(v), torch.zeros((heads, dim, dim), dtype=x.dtype, device=x.device)
    decay = torch.tensor(params["decay"], device=x.device).double()      # as the part holds them: 32-bit numbers
    step = 64                       # rows at a time: within them by the decays' powers, between them by the state
    for first in range(0, rows, step):
        n = min(step, rows - first)
        qc, kc, vc = (t[first:first + n].transpose(0, 1) for t in (q, k, v))
        index = torch.arange(n, device=x.device, dtype=x.dtype)
        apart = (index[:, None] - index[None]).clamp(min=0)
        inside = torch.tril((qc @ kc.transpose(1, 2)) * decay[:, None, None] ** apart[None])
        o = inside @ vc + (qc @ state) * decay[:, None, None] ** (index + 1)[None, :, None]
        out[first:first + n] = o.transpose(0, 1)
        state = state * decay[:, None, None] ** n + (kc * decay[:, None, None] ** (n - 1 - index)[None, :, None]).transpose(1, 2) @ vc
    merged = _rms(out.reshape(rows, heads * dim), w["norm"], EPS) * torch.sigmoid(x @ w["g"].t())
    return {"out": merged @ w["o"].t(), "state0": state[None]}


def _exact_latent(case, w, x):
    rows, heads, dim = case["rows"], case["heads"], 128
    positions = torch.arange(rows, device=x.device)
    base = _part(case)[1]["rot"]["base"]

    def rotate(t):                  # the frequencies in 64 bits
        freq = base ** (-torch.arange(0, 64, 2, device=x.device).double() / 64)
        angle = positions.double()[:, None] * freq[None]
        cos, sin = angle.cos()[:, None], angle.sin()[:, None]
        even, odd = t[..., 0::2], t[..., 1::2]
        return torch.stack([even * cos - odd * sin, even * sin + odd * cos], dim=-1).flatten(-2)

    q = (x @ w["q"].t()).view(rows, heads, dim + 64)
    down = x @ w["dkv"].t()
    latent, shared = _rms(down[:, :512], w["dkv.norm"], EPS), rotate(down[:, None, 512:])
    q = torch.cat([q[..., :dim], rotate(q[..., dim:])], dim=-1)
    k = torch.cat([(latent @ w["uk"].t()).view(rows, heads, dim), shared.expand(rows, heads, 64)], dim=-1)
    v = (latent @ w["uv"].t()).view(rows, heads, dim)
    return {"out": _attend(q, k, v, 0, 192 ** -0.5).reshape(rows, heads * dim) @ w["o"].t()}


def _exact_delta(case, w, x):
    rows, heads, dim = case["rows"], case["heads"], 128

    def convolved(name, count):
        u = x @ w[name].t()
        padded = torch.cat([u.new_zeros((3, u.shape[1])), u])
        y = sum(padded[tap:tap + rows] * w[name + ".conv"][:, tap] for tap in range(4))
        return F.silu(y).view(rows, count, dim), padded[-3:]

    def unit(t):
        return t / torch.sqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)

    (q, q_last), (k, k_last), (v, v_last) = convolved("q", heads // 2), convolved("k", heads // 2), convolved("v", heads)
    q, k = (unit(t).repeat_interleave(2, dim=1) for t in (q, k))
    q = q * dim ** -0.5
    beta = torch.sigmoid(x @ w["b"].t())
    z = (x @ w["a1"].t()) @ w["a2"].t() + w["dt_bias"]
    keep = torch.exp(-torch.exp(w["A_log"])[None, :, None] * F.softplus(z, threshold=1e9).view(rows, heads, dim))
    out, state = torch.empty_like(v), torch.zeros((heads, dim, dim), dtype=x.dtype, device=x.device)
    for t in range(rows):
        state = keep[t][:, :, None] * state
        u = beta[t][:, None] * (v[t] - (k[t][:, None] @ state)[:, 0])
        state = state + k[t][:, :, None] * u[:, None]
        out[t] = (q[t][:, None] @ state)[:, 0]
    gate = torch.sigmoid((x @ w["g1"].t()) @ w["g2"].t())
    out = _rms(out, w["norm"], EPS).reshape(rows, heads * dim) * gate
    return {"out": out @ w["o"].t(), "state0": state[None], "state1": torch.cat([q_last, k_last, v_last], dim=1)[None]}


_EXACT_PARTS = {"experts": _exact_experts, "linear": _exact_linear, "latent": _exact_latent, "delta": _exact_delta}
