"""The Givelix design through the engine against the plain implementation (``tests/plain/givelix_plain.py``):
every mixer alone and together, whole prompts, decoding through the cache and the state, portions down to two
tokens, mixed batches with pages and state slots that are used again, other sizes, both precisions, and greedy
generation through ``LLMEngine``."""
import json
import random
import tempfile
from pathlib import Path

import numpy as np
import pytest
import torch

import helpers
from plain import givelix_plain as plain

pytestmark = pytest.mark.gpu

ROT = {"base": 10000.0, "dims": 8}
ROT_SCALED = {"base": 50000.0, "dims": 12, "scaling": {"factor": 4.0, "original": 64, "fast": 16.0, "slow": 2.0}}


def lightning(heads=3, dim=24, vdim=40, decay=(0.5, 0.97, 0.9995), mlp=None):
    return {"type": "lightning", "mixer": {"heads": heads, "dim": dim, "vdim": vdim, "decay": list(decay)}, "mlp": mlp}


def latent(heads=3, dim=24, rot_dim=8, vdim=20, kv_rank=40, q_rank=36, rot=ROT, kv_from=None, mlp=None):
    mixer = {"heads": heads, "dim": dim, "rot_dim": rot_dim, "vdim": vdim, "kv_rank": kv_rank, "q_rank": q_rank,
             "scale": 1.7 / (dim + rot_dim) ** 0.5, "rot": dict(rot)}
    if kv_from is not None:
        mixer["kv_from"] = kv_from
    return {"type": "latent_attention", "mixer": mixer, "mlp": mlp}


def latent2(heads=5, dim=16, rot_dim=12, vdim=24, kv_rank=56, rot=ROT_SCALED, mlp=None):
    return {"type": "latent_attention_2", "mlp": mlp,
            "mixer": {"heads": heads, "dim": dim, "rot_dim": rot_dim, "vdim": vdim, "kv_rank": kv_rank,
                      "scale": 2.1 / (dim + rot_dim) ** 0.5, "rot": dict(rot)}}


def model(layers, width=72, vocab=211, streams=3, mult=0.4, logit_scale=0.7):
    config = {"architecture": "Givelix", "vocab": vocab, "width": width, "layers": layers, "norm": {"eps": 1e-5},
              "residual_mult": mult, "logit_scale": logit_scale}
    if streams is not None:
        config["streams"] = streams
    return config


DENSE = {"kind": "dense", "ff": 104}
CONFIGS = {
    "lightning_only": model([lightning(mlp=DENSE), lightning(heads=1, dim=40, vdim=8, decay=(0.8,))]),
    "latent_only": model([latent(mlp=DENSE), latent(kv_from=0)], streams=None),
    "latent2_only": model([latent2(), latent2(heads=2, dim=8, rot_dim=4, vdim=8, kv_rank=24,
                                          rot={"base": 100.0, "dims": 4}, mlp=DENSE)], streams=1),
    "all_kinds": model([latent(mlp=DENSE), lightning(), latent(kv_from=0, heads=2, dim=16, vdim=8, q_rank=20, mlp=DENSE),
                        latent2(mlp=DENSE), lightning(heads=2, dim=36, vdim=16, decay=(0.6, 0.999), mlp=DENSE), latent2()],
                       width=80, streams=4),
    # values that many models make equal or one: one head, one stream with tables, dim = vdim = rank, no layer scale
    "equal_sizes": model([latent(heads=1, dim=16, rot_dim=16, vdim=16, kv_rank=16, q_rank=16, rot={"base": 300.0, "dims": 16}),
                          lightning(heads=1, dim=32, vdim=32, decay=(0.9,), mlp=DENSE)], width=64, streams=1, mult=1.0,
                         logit_scale=1.0),
    # sizes that no vector load, tensor-core tile or few-rows product takes: every kernel's plain path
    "odd_sizes": model([lightning(heads=2, dim=48, vdim=20, decay=(0.7, 0.99)),
                        latent(heads=5, dim=20, rot_dim=6, vdim=12, kv_rank=36, q_rank=30, rot={"base": 777.0, "dims": 6},
                               mlp={"kind": "dense", "ff": 90}),
                        latent2(heads=3, dim=10, rot_dim=6, vdim=14, kv_rank=22,
                                rot={"base": 1000.0, "dims": 6, "scaling": {"factor": 3.0, "original": 40, "fast": 8.0, "slow": 1.0}},
                                mlp={"kind": "dense", "ff": 50}),
                        # a reader of a cache that is not the first layer's, with other heads and sizes of its own
                        latent(heads=9, dim=8, rot_dim=6, vdim=10, kv_rank=36, q_rank=14, rot={"base": 777.0, "dims": 6}, kv_from=1)],
                       width=102, vocab=333, streams=2),
    # heads of 128 and 64 rotated values: the attention over keys and values made from the latent
    "expanded": model([latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=64, rot={"base": 500.0, "dims": 64}, mlp=DENSE),
                       latent2(heads=3, dim=128, rot_dim=64, vdim=128, kv_rank=72, rot={"base": 900.0, "dims": 48}),
                       latent(heads=1, dim=128, rot_dim=64, vdim=128, kv_rank=64, q_rank=24, rot={"base": 500.0, "dims": 64}, kv_from=0)],
                      width=96),
}
NO_LAYER_SCALE = {"equal_sizes"}
# bfloat16: the random models are made with large gains so that every mechanism matters; their rounding noise is
# a few hundredths of the logits, a wrong mechanism moves them by tenths and more (and float32 pins the rest)
RMS_LIMIT = {"float32": 1.0e-5, "bfloat16": 1.0e-1}
_MODELS: dict = {}


def folder_of(name: str):
    if name not in _MODELS:
        holder = tempfile.TemporaryDirectory(prefix=f"givelix_{name}_")
        plain.write_model(holder.name, CONFIGS[name], seed=11 + len(_MODELS), layer_scale=name not in NO_LAYER_SCALE)
        _MODELS[name] = (holder, Path(holder.name), plain.load_folder(holder.name))
    return _MODELS[name][1]


def reference(name: str, tokens):
    folder_of(name)
    config, weights = _MODELS[name][2]
    return plain.forward_full(config, weights, tokens).to(torch.float32)


def replay(name: str, dtype: str, steps, max_tokens: int, page: int = 16, max_requests: int = 4):
    from llm_serving_engine_b200.engine.trace_replay import replay as run

    with tempfile.TemporaryDirectory(prefix="givelix_out_") as out:
        run(folder_of(name), dtype, out, max_tokens, [json.dumps(step) for step in steps], block_size=page,
            max_requests=max_requests)
        return helpers.collect(steps, Path(out))


def compare(name, dtype, requests, got, what):
    for rid, tokens in requests.items():
        want = reference(name, tokens)
        assert got[rid].shape == want.shape, f"{what}: {rid}: shape {tuple(got[rid].shape)} against {tuple(want.shape)}"
        centred = want - want.mean(-1, keepdim=True)
        per_row = (got[rid] - want).double().pow(2).mean(-1).sqrt() / centred.double().pow(2).mean().sqrt()
        worst = float(per_row.max())
        assert worst <= RMS_LIMIT[dtype], (f"{what}: {name} {dtype} request {rid}: row error / logit size {worst:.2e} at "
                                           f"position {int(per_row.argmax())}, first above the limit "
                                           f"{int((per_row > RMS_LIMIT[dtype]).nonzero()[0])}")


def some_requests(name, lengths, seed=5):
    rng = random.Random(seed)
    vocab = CONFIGS[name]["vocab"]
    return {f"r{index}": helpers.random_tokens(rng, vocab, length) for index, length in enumerate(lengths)}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", sorted(CONFIGS))
def test_whole_prompts(name, dtype):
    requests = some_requests(name, [1, 2, 17, 70])
    got = replay(name, dtype, helpers.trace_whole(requests), helpers.max_tokens_for(requests))
    compare(name, dtype, requests, got, "whole")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", sorted(CONFIGS))
def test_prompt_then_token_by_token(name, dtype):
    """Decoding reads the pages and the state that the prompt step left; the single tokens are replayed from a
    captured graph, whose warm-up run must leave the state as it was."""
    requests = some_requests(name, [40, 9, 3], seed=6)
    got = replay(name, dtype, helpers.trace_tail_decode(requests, tail=24), helpers.max_tokens_for(requests))
    compare(name, dtype, requests, got, "tail decoded")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_portions_of_changing_size(dtype):
    requests = some_requests("all_kinds", [150, 33], seed=7)
    for sizes in ((7, 2, 13, 3, 2, 31, 5, 16, 2, 64, 17), (2,), (16, 16, 1, 15, 17)):
        got = replay("all_kinds", dtype, helpers.trace_portions(requests, sizes), helpers.max_tokens_for(requests))
        compare("all_kinds", dtype, requests, got, f"portions {sizes}")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("page", [16, 8])
def test_mixed_batches_reuse_pages_and_state_slots(dtype, page):
    """Nine requests through four state slots and a pool sized for the live ones only: a slot's state must be
    zero for its next request, and a page's old rows must not be read."""
    requests = some_requests("all_kinds", [61, 5, 90, 33, 2, 47, 130, 18, 64], seed=8)
    steps, peak = helpers.trace_mixed(requests, seed=3, max_live=4)
    got = replay("all_kinds", dtype, steps, peak, page=page)
    compare("all_kinds", dtype, requests, got, "mixed")


def test_a_batch_gives_what_each_request_gives_alone():
    requests = some_requests("all_kinds", [37, 12, 80, 5], seed=9)
    steps, peak = helpers.trace_mixed(requests, seed=4, max_live=4)
    together = replay("all_kinds", "float32", steps, peak)
    for rid, tokens in requests.items():
        alone = replay("all_kinds", "float32", helpers.trace_whole({rid: tokens}), helpers.max_tokens_for({rid: tokens}))
        assert float((together[rid] - alone[rid]).abs().max()) <= 2e-5 * float(alone[rid].abs().max())


def test_long_decoding_carries_the_state_and_crosses_key_chunks():
    """600 single tokens after a short prompt: the lightning state is carried through 600 graph replays, the latent
    attention's keys pass the borders of its tiles (32), chunks (256) and many pages."""
    requests = some_requests("all_kinds", [610], seed=10)
    got = replay("all_kinds", "float32", helpers.trace_tail_decode(requests, tail=600), 640)
    compare("all_kinds", "float32", requests, got, "long decoding")


def test_greedy_generation_through_the_engine_and_its_scheduler():
    """More requests than the scheduler keeps live, prompts cut into portions: every request's greedy tokens equal
    the plain implementation's (float32; a request whose top two logits are closer than the arithmetic's noise is
    skipped from that token on)."""
    from llm_serving_engine_b200.config import CacheConfig, SchedulerConfig
    from llm_serving_engine_b200.engine.llm_engine import LLMEngine
    from llm_serving_engine_b200.sampling.sampler import GenerationConfig
    from llm_serving_engine_b200.models import load_model

    name = "all_kinds"
    engine = LLMEngine(load_model(folder_of(name), dtype="float32"), None,
                       cache_config=CacheConfig(block_size=16, num_blocks=40),
                       scheduler_config=SchedulerConfig(max_batch_size=3, max_tokens_per_step=48), prefill_chunk_size=20)
    prompts = list(some_requests(name, [30, 7, 55, 2, 19, 41], seed=12).values())
    new_tokens = 12
    produced = engine.generate_many(prompts, GenerationConfig(max_new_tokens=new_tokens, temperature=0.0))
    for prompt, tokens in zip(prompts, produced):
        assert len(tokens) == new_tokens
        logits = reference(name, prompt + tokens)
        for index, token in enumerate(tokens):
            row = logits[len(prompt) + index - 1]
            top = torch.topk(row, 2).values
            if float(top[0] - top[1]) < 1e-3 * float(row.abs().max()):
                break
            assert int(row.argmax()) == token, f"token {index} of a {len(prompt)}-token prompt"


# ------------------------------------------------------------------ the mechanisms' kernels alone
def _latent_plain(q, rows, positions, scale, rank, sink, window=0):
    out = torch.zeros(q.shape[0], q.shape[1], rank, dtype=torch.float64)
    for t, pos in enumerate(positions):
        first = max(0, pos + 1 - window) if window else 0
        keys = rows[first:pos + 1].double()
        scores = torch.einsum("hd,jd->hj", q[t].double(), keys) * scale
        top = scores.max(-1, keepdim=True).values
        if sink is not None:
            top = torch.maximum(top, sink.double()[:, None])
        weights = torch.exp(scores - top)
        total = weights.sum(-1, keepdim=True)
        if sink is not None:
            total = total + torch.exp(sink.double()[:, None] - top)
        out[t] = (weights / total) @ keys[:, :rank]
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("use_sink", [False, True])
def test_latent_attention_finds_one_far_key_at_every_border(dtype, use_sink):
    """One key among hundreds is made to stand out (its row is a multiple of the query); it sits at, just before and
    just after the borders of pages, tiles of 32 and chunks of 256, as the first key and as the row's own.  Rows are
    single tokens (keys split over blocks and merged) and rows of a portion (one block per row)."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(3)
    heads, rank, rot, page = 3, 40, 8, 16
    width, context = rank + rot, 530
    pages = -(-context // page)
    order = torch.randperm(pages + 5)[:pages].to(torch.int32)          # pages scattered over a larger pool
    for special in (0, 15, 16, 31, 32, 255, 256, 257, 511, 512, 529):
        rows = torch.randn(context, width) * 0.3
        q = torch.randn(1, heads, width)
        rows[special] = q[0, 1] * 2.0                                    # head 1 looks at `special`
        rows, q = rows.to(dtype).float(), q.to(dtype).float()
        pool = torch.full((pages + 5, page, width), float("nan"))      # unowned pages hold anything
        for logical in range(pages):
            chunk = rows[logical * page:(logical + 1) * page]
            pool[int(order[logical])].zero_()
            pool[int(order[logical]), :chunk.shape[0]] = chunk
        sink = torch.tensor([0.5, -1.0, 2.0]) if use_sink else None
        for positions in ([context - 1], [special], list(range(special, min(context, special + 70)))):
            count = len(positions)
            queries = q.expand(count, heads, width).contiguous()
            want = _latent_plain(queries, rows, positions, 0.9, rank, sink)
            got = torch.empty(count, heads, rank, dtype=dtype, device="cuda")
            ops.latent_attention(queries.to(dtype).cuda(), pool.to(dtype).cuda(), got, order.view(1, -1).cuda(),
                                 torch.zeros(count, dtype=torch.int32, device="cuda"),
                                 torch.tensor(positions, dtype=torch.int32, device="cuda"), 0.9,
                                 None if sink is None else sink.cuda(), split=count == 1)
            limit = 2e-5 if dtype == torch.float32 else 2e-2
            assert float((got.float().cpu() - want).abs().max()) <= limit, (special, positions[:3], count)


def test_tensor_core_latent_attention_against_the_general_kernel():
    """Portions of several requests beside single tokens, pages scattered, odd numbers of heads, with and without a
    sink, whole and split by chunks: the tensor-core kernel against the float32-arithmetic kernel on the same
    bfloat16 inputs, and one far key that must be found."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(8)
    page = 16
    for heads, rank, rot in ((3, 64, 16), (16, 128, 32), (40, 192, 16), (6, 24, 8)):
        width = rank + rot
        counts, firsts = [70, 1, 33, 1, 5], [300, 519, 0, 0, 63]
        contexts = [first + count for first, count in zip(firsts, counts)]
        pages_each = [-(-context // page) for context in contexts]
        pool = (torch.randn(sum(pages_each) + 3, page, width) * 0.5).to(torch.bfloat16).cuda()
        order = torch.randperm(sum(pages_each) + 3).to(torch.int32)
        table = torch.full((len(counts), max(pages_each)), -1, dtype=torch.int32)
        cursor = 0
        for index, count in enumerate(pages_each):
            table[index, :count] = order[cursor:cursor + count]
            cursor += count
        total = sum(counts)
        q = (torch.randn(total, heads, width) * 0.5).to(torch.bfloat16)
        pool[int(table[0, 1]), 3] = (q[5, heads - 1] * 4.0).cuda()          # key 19 of request 0 stands out for one head
        starts = torch.tensor([0] + list(np.cumsum(counts)), dtype=torch.int32).cuda()
        seg = torch.cat([torch.full((count,), index, dtype=torch.int32) for index, count in enumerate(counts)]).cuda()
        pos = torch.cat([torch.arange(first, first + count, dtype=torch.int32) for first, count in zip(firsts, counts)]).cuda()
        first_pos = torch.tensor(firsts, dtype=torch.int32).cuda()
        for sink in (None, torch.linspace(-1.0, 2.0, heads).cuda()):
            for split in (False, True):
                want = torch.empty(total, heads, rank, dtype=torch.bfloat16, device="cuda")
                got = torch.empty_like(want)
                ops.latent_attention(q.cuda(), pool, want, table.cuda(), seg, pos, 0.3, sink, split=split, tensor_cores=False)
                ops.latent_attention(q.cuda(), pool, got, table.cuda(), seg, pos, 0.3, sink, split=split,
                                     segment_start=starts, segment_first_position=first_pos)
                assert ops.latent_attention_mma_supported(width, rank, torch.bfloat16) == (rank % 8 == 0 and width % 16 == 0)
                error = float((got.float() - want.float()).abs().max())
                assert error <= 2e-2 * max(1.0, float(want.float().abs().max())), (heads, rank, rot, sink is not None, split, error)


def test_latent_attention_window_edges():
    """The kernel's window parameter: the key just inside the window is seen, the one just outside is not."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(4)
    heads, rank, rot, page, context, window = 2, 24, 8, 8, 300, 37
    width = rank + rot
    rows = torch.randn(context, width) * 0.3
    q = torch.randn(1, heads, width)
    pool = rows.view(-1, page, width).contiguous() if context % page == 0 else None
    if pool is None:
        pool = torch.zeros(-(-context // page) * page, width)
        pool[:context] = rows
        pool = pool.view(-1, page, width)
    table = torch.arange(pool.shape[0], dtype=torch.int32).view(1, -1)
    for pos in (window - 2, window - 1, window, 255, 256, 299):
        for offset in (window - 1, window):          # the last key inside, the first outside
            if pos - offset < 0:
                continue
            marked = rows.clone()
            marked[pos - offset] = q[0, 0] * 3.0
            marked_pool = pool.clone().view(-1, width)
            marked_pool[pos - offset] = marked[pos - offset]
            want = _latent_plain(q, marked, [pos], 1.0, rank, None, window)
            got = torch.empty(1, heads, rank, device="cuda")
            ops.latent_attention(q.cuda(), marked_pool.view(-1, page, width).cuda(), got, table.cuda(),
                                 torch.zeros(1, dtype=torch.int32, device="cuda"),
                                 torch.tensor([pos], dtype=torch.int32, device="cuda"), 1.0, None, window=window)
            assert float((got.cpu() - want).abs().max()) <= 2e-5, (pos, offset)


def test_linear_attention_scan_against_the_recurrence():
    """Odd sizes (dim beyond one thread's 32 rows, columns beyond one block), two requests of unequal length from
    non-zero states in slots that are not in order, decays from fast to almost none."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(5)
    for heads, dim, vdim in ((2, 24, 40), (3, 72, 136), (1, 130, 8)):
        width = heads * (2 * dim + 2 * vdim)
        counts, slots = [19, 1, 150], [2, 0, 3]
        proj = torch.randn(sum(counts), width)
        decay = torch.tensor([0.3, 0.95, 0.9999][:heads])
        state = torch.randn(4, heads, dim, vdim) * 0.5
        want_state = state.double().clone()
        want = torch.zeros(sum(counts), heads * vdim, dtype=torch.float64)
        row = 0
        for count, slot in zip(counts, slots):
            for t in range(row, row + count):
                z = proj[t].double()
                act = z * torch.sigmoid(z)
                q = act[:heads * dim].view(heads, dim)
                k = act[heads * dim:2 * heads * dim].view(heads, dim)
                v = act[2 * heads * dim:2 * heads * dim + heads * vdim].view(heads, vdim)
                for h in range(heads):
                    want_state[slot, h] = float(decay[h]) * want_state[slot, h] + torch.outer(k[h], v[h])
                    want[t, h * vdim:(h + 1) * vdim] = want_state[slot, h].t() @ q[h]
            row += count
        starts = torch.tensor([0, 19, 20, 170, 170], dtype=torch.int32).cuda()       # a fourth, empty request
        for chunked in (False, True):      # row by row, and in chunks of 64 rows scanned side by side (19, 1, 64 + 64 + 22)
            got = torch.empty(sum(counts), heads * vdim, device="cuda")
            device_state = state.cuda()
            ops.linear_attention_scan(proj.cuda(), 0, heads * dim, 2 * heads * dim, decay.cuda(), device_state, starts,
                                      torch.tensor(slots + [1], dtype=torch.int32).cuda(), got, heads, dim, vdim, "silu",
                                      chunked=chunked)
            scale = float(want.abs().max())
            assert float((got.cpu() - want).abs().max()) <= 2e-5 * scale, (heads, dim, vdim, chunked)
            assert float((device_state.cpu() - want_state).abs().max()) <= 2e-5 * float(want_state.abs().max())
            assert torch.equal(device_state[1].cpu(), state[1])                  # the empty request's slot is untouched


def test_expanded_latent_attention_in_a_model(monkeypatch):
    """Prompts in portions through the step function, layer by layer over expanded keys and values: launch by launch, from
    a graph captured at a size class, and from that graph again with other contexts of the class; beside a decoding request the
    layers go over the latent rows.  Every logit against the plain implementation."""
    from llm_serving_engine_b200.kernels import ops
    from llm_serving_engine_b200.parts import latent_attention

    monkeypatch.setattr(latent_attention, "LATENT_FLOPS", 1.0)      # always worth it, whatever the sizes
    sizes, real = [], ops.attention_expanded

    def recorded(q_plain, q_wide, rows, *rest):
        sizes.append((q_plain.shape[0], rows.shape[0]))
        return real(q_plain, q_wide, rows, *rest)

    monkeypatch.setattr(ops, "attention_expanded", recorded)
    requests = some_requests("expanded", [230, 230, 215, 31])
    steps, ids = [], list(requests)

    def add(entries, end=()):
        steps.append({"step": len(steps), "end": list(end),
                      "entries": [{"id": rid, "tokens": requests[rid][lo:hi], "want": list(range(hi - lo))} for rid, lo, hi in entries]})

    for rid in ids[:3]:                        # the same classes three times: launches, capture, replay
        add([(rid, 0, 120)])
        add([(rid, 120, len(requests[rid]))], end=[rid] if rid != ids[2] else ())
    add([(ids[3], 0, 30)])
    add([(ids[3], 30, 31)], end=[ids[2], ids[3]])
    got = replay("expanded", "bfloat16", steps, 1024)
    compare("expanded", "bfloat16", requests, got, "expanded")
    assert sizes and len(sizes) % 3 == 0 and len(sizes) < 3 * 7      # some steps were replayed: nothing was launched from here
    assert any(tokens > 120 for tokens, _ in sizes)                  # a captured class has padding rows


@pytest.mark.parametrize("heads, rank, page, window, portions", [
    (2, 64, 16, 0, [(0, 2), (0, 64), (63, 129), (700, 66)]), (3, 512, 8, 0, [(0, 300)]), (1, 24, 64, 37, [(0, 200), (500, 3), (36, 2)]),
    (2, 512, 16, 512, [(1000, 130), (0, 640)]), (5, 72, 1, 1, [(5, 70)])])
def test_latent_attention_over_expanded_keys_and_values(heads, rank, page, window, portions):
    """Portions (first position, rows) behind prefixes, cut at the edges of row tiles (128) and key tiles (64), windows that
    end inside a tile, a sink and a gate: the gathered rows exactly, the attention against float64 over the same bfloat16
    keys and values.  Pages that no request owns hold NaN."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(rank + page)
    rng = random.Random(rank)
    width, tokens = rank + 64, sum(count for _, count in portions)
    contexts = [first + count for first, count in portions]
    pages = [-(-context // page) for context in contexts]
    order = list(range(sum(pages) + 3))
    rng.shuffle(order)
    cache = torch.full((len(order), page, width), float("nan"), dtype=torch.bfloat16)
    tables = torch.full((len(portions), max(pages)), -1, dtype=torch.int32)
    dense = [torch.randn(context, width).bfloat16() for context in contexts]
    for s, rows in enumerate(dense):
        for logical in range(pages[s]):
            tables[s, logical] = physical = order.pop()
            part = rows[logical * page:(logical + 1) * page]
            cache[physical, :len(part)] = part
    starts = torch.tensor([0] + [count for _, count in portions] + [0]).cumsum(0).to(torch.int32).cuda()      # an empty request at the end
    firsts = torch.tensor([first for first, _ in portions] + [0], dtype=torch.int32).cuda()
    ends = torch.tensor(contexts + [0], dtype=torch.int32).cuda()
    tables = torch.cat([tables, torch.full_like(tables[:1], -1)]).cuda()
    low = [max(0, first + 1 - window) if window else 0 for first, _ in portions]
    kept = [-(-(context - lo) // 64) * 64 for context, lo in zip(contexts, low)]
    capacity = sum(kept) + 70
    rows = ops.latent_gather(cache.cuda(), tables, firsts, ends, capacity, window)
    want_rows = torch.zeros(capacity, width, dtype=torch.bfloat16)
    at = 0
    for part, lo, size in zip(dense, low, kept):
        want_rows[at:at + len(part) - lo] = part[lo:]
        at += size
    assert torch.equal(rows.cpu(), want_rows)
    kv = torch.randn(capacity, 2 * heads, 128).bfloat16()
    q_plain, q_wide = torch.randn(tokens, heads, 128).bfloat16() * 0.4, torch.randn(tokens, heads, width).bfloat16()
    sink, gate = torch.randn(heads), torch.rand(tokens, heads)
    for with_extras in (False, True):
        got = torch.empty(tokens, heads, 128, dtype=torch.bfloat16, device="cuda")
        ops.attention_expanded(q_plain.cuda(), q_wide.cuda(), rows, kv.cuda(), got, starts, firsts, ends, 0.1, window,
                               sink.cuda() if with_extras else None, gate.cuda() if with_extras else None)
        assert int(ops.library.load().lse_attention_expanded_status()) == 0
        row = at = 0
        for (first, count), lo, size in zip(portions, low, kept):
            keys = kv[at:at + size].double()
            for t in sorted({0, 1, count // 2, min(127, count - 1), count - 1}):
                pos = first + t
                seen = slice(max(0, pos + 1 - window) - lo if window else 0, pos + 1 - lo)
                scores = (torch.einsum("hd,khd->hk", q_plain[row + t].double(), keys[seen, :heads])
                          + q_wide[row + t, :, rank:].double() @ want_rows[at:at + size][seen, rank:].double().t()) * 0.1
                if with_extras:
                    scores = torch.cat([scores, sink.double()[:, None]], dim=1)
                weights = torch.softmax(scores, dim=1)[:, :keys[seen].shape[0]]
                want = torch.einsum("hk,khd->hd", weights, keys[seen, heads:])
                if with_extras:
                    want = want * gate[row + t].double()[:, None]
                # weights rounded to bfloat16, the result again: 2^-8 of the largest value each
                assert float((got[row + t].cpu().double() - want).abs().max()) <= 2.0 ** -7 * max(1.0, float(want.abs().max())), (first, t)
            row, at = row + count, at + size


@pytest.mark.parametrize("window", [0, 330])
@pytest.mark.parametrize("per_tile", [5.0, 9.5, 40.0, 90.0])
def test_expanded_latent_attention_while_the_maximum_grows(per_tile, window):
    """Scores that grow along the keys, by 2^5 a tile of 64 (a tile's probabilities stay relative to an older maximum), 2^9.5 and
    2^40 (the sums are taken over to the new maximum a tile later) and 2^90 (at once), in the unrotated and the rotated part, over
    enough tiles for both groups and all their accumulators; the values shrink as the weights grow (up to 2^9.5 a tile), so that
    every tile counts and a factor that is lost or applied twice shows.  Against float64 over the same bfloat16 keys and values."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(int(per_tile) + window)
    heads, rank, portions = 2, 64, [(0, 600), (500, 130)]
    contexts = [first + count for first, count in portions]
    low = [max(0, first + 1 - window) if window else 0 for first, _ in portions]
    kept = [-(-(context - lo) // 64) * 64 for context, lo in zip(contexts, low)]
    tokens, capacity, scale = sum(count for _, count in portions), sum(kept), 0.1
    sign, rot_sign = torch.randint(0, 2, (heads, 128)) * 2.0 - 1, torch.randint(0, 2, (64,)) * 2.0 - 1
    q_plain = (sign * 0.5).expand(tokens, heads, 128).contiguous().bfloat16()
    q_wide = torch.cat([torch.randn(tokens, heads, rank), (rot_sign * 0.5).expand(tokens, heads, 64)], dim=2).bfloat16()
    rows, kv = torch.zeros(capacity, rank + 64), torch.zeros(capacity, 2 * heads, 128)
    at = 0
    for lo, context, size in zip(low, contexts, kept):
        n = context - lo
        growth = torch.arange(n) * per_tile / 64                       # of the score, in powers of two
        natural = growth * 0.6931471805599453 / scale
        kv[at:at + n, :heads] = (natural * 0.6 / 64)[:, None, None] * sign + torch.randn(n, heads, 128) * 0.02
        rows[at:at + n, rank:] = (natural * 0.4 / 32)[:, None] * rot_sign + torch.randn(n, 64) * 0.02
        shrink = torch.exp2(-growth if per_tile < 10 else torch.zeros(n))
        kv[at:at + n, heads:] = (1.0 + torch.rand(n, heads, 128)) * shrink[:, None, None]
        at += size
    rows, kv = rows.bfloat16(), kv.bfloat16()
    starts = torch.tensor([0, 600, 730], dtype=torch.int32).cuda()
    firsts, ends = (torch.tensor(values, dtype=torch.int32).cuda() for values in ([0, 500], contexts))
    got = torch.empty(tokens, heads, 128, dtype=torch.bfloat16, device="cuda")
    ops.attention_expanded(q_plain.cuda(), q_wide.cuda(), rows.cuda(), kv.cuda(), got, starts, firsts, ends, scale, window)
    assert int(ops.library.load().lse_attention_expanded_status()) == 0
    row = at = 0
    for (first, count), lo, size in zip(portions, low, kept):
        keys, rotated = kv[at:at + size].double(), rows[at:at + size, rank:].double()
        for t in sorted({0, 63, 64, 127, min(128, count - 1), min(200, count - 1), min(400, count - 1), count - 1}):
            pos = first + t
            seen = slice(max(0, pos + 1 - window) - lo if window else 0, pos + 1 - lo)
            scores = (torch.einsum("hd,khd->hk", q_plain[row + t].double(), keys[seen, :heads])
                      + q_wide[row + t, :, rank:].double() @ rotated[seen].t()) * scale
            want = torch.einsum("hk,khd->hd", torch.softmax(scores, dim=1), keys[seen, heads:])
            # weights rounded to bfloat16 and the result again, all values positive: 2^-8 each of the value
            error = ((got[row + t].cpu().double() - want).abs() / want).max()
            assert float(error) <= 2.0 ** -6, (first, t, float(error))
        row, at = row + count, at + size


@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_a_latent_that_is_not_finite_reaches_the_rows_that_read_it_only(value, window, monkeypatch):
    """One cached row of 300 with a value that is not finite in its latent, through the layer: rows before it, and rows whose
    window has passed it, are what they are without it, bit for bit; rows that read it are NaN, as over the latent rows.  Then an
    infinite rotated value: the same rows are left alone."""
    from llm_serving_engine_b200.kernels import ops
    from llm_serving_engine_b200.parts import latent_attention
    from test_launch_signature_cpu import latent_model
    from test_step_graphs_gpu import runner_for
    from llm_serving_engine_b200.engine import StepEntry

    monkeypatch.setattr(latent_attention, "LATENT_FLOPS", 1.0)
    mixer = latent_model([window], heads=2, rank=72, device="cuda", scale=0.07).blocks[0].mixer
    torch.manual_seed(3)
    x = torch.randn(300, 64, device="cuda").bfloat16()
    real, at = ops.latent_gather, 193

    def outputs(column):
        runner = runner_for(latent_model([window], heads=2, rank=72, device="cuda"), use_graphs=False)
        runner.cache.create("r")
        step, caches = runner.prepare([StepEntry("r", [0] * 300, [])])

        def gather(cache, tables, *rest):
            if column is not None:
                cache[tables[0, at // 16], at % 16, column] = value
            return real(cache, tables, *rest)

        monkeypatch.setattr(ops, "latent_gather", gather)
        out = mixer.forward(x, step, caches[0])
        return (out.sum(0) if out.dim() == 3 else out).float()

    clean = outputs(None)
    readers = torch.zeros(300, dtype=torch.bool, device="cuda")
    readers[at:at + window if window else 300] = True
    for column in (0, 71, 80):
        got = outputs(column)
        assert bool(clean.isfinite().all()) and torch.equal(got[~readers], clean[~readers]), column
        if column < 72:
            assert bool(got[readers].isnan().all()), column


def test_expanded_latent_attention_some_heads_at_a_time():
    """Five heads, two, two and one at a time, with a sink and gates, bit for bit as all of them at once; a launch leaves the other
    heads' outputs alone."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(8)
    heads, rank, counts, first = 5, 72, [130, 65], [0, 63]
    contexts = [a + b for a, b in zip(first, counts)]
    tokens, capacity = sum(counts), sum(-(-context // 64) * 64 for context in contexts)
    rows, kv = torch.randn(capacity, rank + 64).bfloat16().cuda(), torch.randn(capacity, 2, heads, 128).bfloat16().cuda()
    q_plain, q_wide = torch.randn(tokens, heads, 128).bfloat16().cuda(), torch.randn(tokens, heads, rank + 64).bfloat16().cuda()
    starts, firsts, ends = (torch.tensor(values, dtype=torch.int32).cuda() for values in ([0, 130, 195], first, contexts))
    sink, gate = torch.randn(heads).cuda(), torch.rand(tokens, heads).cuda()
    want, got = torch.empty_like(q_plain), torch.full_like(q_plain, 9.0)
    rest = (starts, firsts, ends, 0.1, 0, sink, gate)
    ops.attention_expanded(q_plain, q_wide, rows, kv.view(capacity, 2 * heads, 128), want, *rest)
    for at, count in ((3, 2), (0, 2), (2, 1)):
        part = kv[:, :, at:at + count].reshape(capacity, 2 * count, 128).contiguous()
        before = got.clone()
        ops.attention_expanded(q_plain, q_wide, rows, part, got, *rest, first_head=at)
        assert torch.equal(got[:, at:at + count], want[:, at:at + count])
        others = [head for head in range(heads) if not at <= head < at + count]
        assert torch.equal(got[:, others], before[:, others])
    assert int(ops.library.load().lse_attention_expanded_status()) == 0


def test_a_gather_without_room_for_the_requests_rows_is_reported():
    """Contexts of 100 and 130 keys are 128 and 192 rows: room for one row fewer is reported, and nothing behind it is written."""
    from llm_serving_engine_b200.kernels import ops

    cache = torch.randn(16, 16, 88).bfloat16().cuda()
    tables = torch.arange(16, dtype=torch.int32).view(2, 8).cuda()
    tables = torch.cat([tables, tables], dim=1)
    firsts, contexts = torch.tensor([40, 0], dtype=torch.int32).cuda(), torch.tensor([100, 130], dtype=torch.int32).cuda()
    library = ops.library.load()
    for capacity, want in ((320, 0), (319, ops.EXPANDED_ROWS_LEFT_OUT), (400, 0)):
        rows = ops.latent_gather(cache, tables, firsts, contexts, capacity)
        assert library.lse_attention_expanded_status() == want and rows.shape[0] == capacity
        ops.kernel_status_reset()
    assert library.lse_attention_expanded_status() == 0


@pytest.mark.parametrize("heads, dim, vdim, counts, dtype", [(2, 128, 128, [64, 65, 1, 130], "bfloat16"), (3, 68, 130, [127, 63], "float32"),
                                                             (1, 127, 5, [200, 2], "bfloat16"), (2, 96, 256, [128], "float32")])
def test_linear_attention_in_chunks_as_products(heads, dim, vdim, counts, dtype):
    """The products over chunks of 64 rows at the edges of their tiles, against the recurrence in float64, from states that
    are not zero; a decay that is gone within a chunk; and an infinite value in a request's last row, which must not reach
    the rows before it."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(dim)
    rows, width = sum(counts), heads * (2 * dim + 2 * vdim) + 3
    proj = torch.randn(rows, width).to(getattr(torch, dtype))
    v_last = 2 * heads * dim + heads * vdim - 1
    proj[counts[0] - 1, v_last] = float("inf")
    decay = torch.tensor([0.999, 0.02, 0.9][:heads])
    state = torch.randn(len(counts), heads, dim, vdim) * 0.5
    z = proj.double()
    act = z * torch.sigmoid(z)
    q, k = (act[:, i * heads * dim:(i + 1) * heads * dim].view(rows, heads, dim) for i in (0, 1))
    v = act[:, 2 * heads * dim:2 * heads * dim + heads * vdim].view(rows, heads, vdim)
    want, want_state, row = torch.zeros(rows, heads, vdim, dtype=torch.float64), state.double().clone(), 0
    for request, count in enumerate(counts):
        for t in range(row, row + count):
            want_state[request] = decay.double()[:, None, None] * want_state[request] + k[t][:, :, None] * v[t][:, None, :]
            want[t] = torch.einsum("hde,hd->he", want_state[request], q[t])
        row += count
    starts = torch.tensor([0] + counts).cumsum(0).to(torch.int32).cuda()
    got, device_state = torch.empty(rows, heads * vdim, device="cuda"), state.cuda()
    ops.linear_attention_scan(proj.cuda(), 0, heads * dim, 2 * heads * dim, decay.cuda(), device_state, starts,
                              torch.arange(len(counts), dtype=torch.int32).cuda(), got, heads, dim, vdim, "silu", chunked=True)
    got = got.cpu().view(rows, heads, vdim).double()
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), finite) and int((~finite).sum()) == 1
    # sums of up to 130 rows of 128 products, each a few units of 2^-24 of the largest terms
    assert float((got - want)[finite].abs().max()) <= 2e-5 * float(want[finite].abs().max())
    good = torch.isfinite(want_state)
    assert float((device_state.cpu() - want_state)[good].abs().max()) <= 2e-5 * float(want_state[good].abs().max())


@pytest.mark.parametrize("counts", [[32, 33, 1, 80, 3], [1] * 40, [5], [300] + [1] * 9, [32], [33]])
def test_short_requests_beside_chunks_are_scanned_row_by_row(counts):
    """Requests of up to 32 rows do not pay for a chunk of 64: beside longer ones and alone they give the row-by-row scan's bits,
    outputs and states; the longer ones' agree with it up to rounding."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(len(counts))
    heads, dim, vdim, rows = 2, 96, 130, sum(counts)
    proj = torch.randn(rows, heads * (2 * dim + 2 * vdim)).bfloat16().cuda()
    decay, first = torch.tensor([0.97, 0.5]).cuda(), torch.randn(len(counts), heads, dim, vdim).cuda()
    starts = torch.tensor([0] + counts).cumsum(0).to(torch.int32).cuda()
    slots = torch.arange(len(counts), dtype=torch.int32).flip(0).cuda()
    results = []
    for chunked in (False, True):
        out, state = torch.full((rows, heads * vdim), float("nan"), device="cuda"), first.clone()
        ops.linear_attention_scan(proj, 0, heads * dim, 2 * heads * dim, decay, state, starts, slots, out, heads, dim, vdim, "silu",
                                  chunked=chunked)
        results.append((out, state))
    (want, want_state), (got, got_state) = results
    for index, count in enumerate(counts):
        mine, slot = slice(int(starts[index]), int(starts[index + 1])), int(slots[index])
        if count <= 32:
            assert torch.equal(got[mine], want[mine]) and torch.equal(got_state[slot], want_state[slot]), index
        # sums of up to 300 rows of 96 products, each a few units of 2^-24 of the largest terms
        assert float((got[mine] - want[mine]).abs().max()) <= 2e-5 * float(want[mine].abs().max()), index
        assert float((got_state[slot] - want_state[slot]).abs().max()) <= 2e-5 * float(want_state[slot].abs().max()), index


@pytest.mark.parametrize("rows, n, off, partials", [(3, 100, 4, 1), (5, 508, 0, 1), (5, 512, 8, 1), (300, 512, 3, 1), (2, 2052, 4, 1),
                                                    (7, 4096, 0, 1), (4, 4100, 0, 1), (9, 1024, 4, 3)])
@pytest.mark.parametrize("proj_type, out_type", [("float32", "float32"), ("bfloat16", "bfloat16"), ("float32", "bfloat16")])
def test_gated_norm_on_either_side_of_its_rules(rows, n, off, partials, proj_type, out_type):
    """Widths below and above the one-pass kernel's, gates at columns that are not aligned, stacks of partial sums; rows of no
    request are left alone."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(n + rows)
    kind = getattr(torch, proj_type if partials == 1 else "float32")
    values, weight = torch.randn(rows, n).cuda(), (torch.rand(n) + 0.5).cuda()
    proj = torch.randn(*((partials,) if partials > 1 else ()), rows, n + off + -(n + off) % 4).to(kind).cuda()
    segments = torch.zeros(rows, dtype=torch.int32)
    segments[rows // 2] = -1
    got = torch.full((rows, n), 9.0, dtype=getattr(torch, out_type)).cuda()
    ops.gated_rmsnorm(values, proj, off, weight, 1e-5, got, segments.cuda())
    z = proj.double().sum(0) if partials > 1 else proj.double()
    x = values.double()
    want = x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * weight.double() * torch.sigmoid(z[:, off:off + n])
    kept = segments >= 0
    assert bool((got[~kept] == 9.0).all())
    bound = 2.0 ** -8 if out_type == "bfloat16" else 2e-6
    assert float((got.double() - want)[kept].abs().max()) <= bound * float(want.abs().max())


def test_residual_copies_update_and_norm():
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(6)
    rows, copies, width = 9, 3, 50
    x = torch.randn(rows, copies, width)
    delta = torch.randn(2, rows, width)              # two partial sums
    scale, mix = torch.rand(width) + 0.5, torch.randn(copies, copies)
    write, read, weight = torch.randn(copies), torch.randn(copies), torch.randn(width)
    y = (delta[0] + delta[1]).double() * 0.3 * scale.double()
    new = torch.einsum("sr,tsw->trw", mix.double(), x.double()) + write.double()[None, :, None] * y[:, None, :]
    u = torch.einsum("r,trw->tw", read.double(), new)
    want = u / torch.sqrt(u.pow(2).mean(-1, keepdim=True) + 1e-5) * weight.double()
    device_x = x.view(rows, -1).cuda()
    got = torch.empty(rows, width, device="cuda")
    ops.streams_update_rmsnorm(device_x, copies, delta.cuda(), scale.cuda(), 0.3, mix.cuda(), write.cuda(), read.cuda(),
                               weight.cuda(), 1e-5, got)
    assert float((got.cpu() - want).abs().max()) <= 1e-5 * float(want.abs().max())
    assert float((device_x.cpu().view(rows, copies, width) - new).abs().max()) <= 1e-5 * float(new.abs().max())
    # chosen rows only, nothing written back, the copies summed
    picked = torch.tensor([7, 2], dtype=torch.int32)
    before = device_x.clone()
    got = torch.empty(2, width, device="cuda")
    ops.streams_update_rmsnorm(device_x, copies, None, None, 1.0, None, None, None, weight.cuda(), 1e-5, got,
                               rows=picked.cuda(), write_back=False)
    total = new[picked.long()].sum(1)
    want = total / torch.sqrt(total.pow(2).mean(-1, keepdim=True) + 1e-5) * weight.double()
    assert float((got.cpu() - want).abs().max()) <= 1e-5 * float(want.abs().max())
    assert torch.equal(before, device_x)


def test_rotation_with_scaled_frequencies_reaches_the_cache():
    """The rotated shared key part as the prepare kernel writes it, at positions in the thousands, against the plain
    rotation with the same scaled frequencies."""
    from llm_serving_engine_b200.kernels import ops
    from llm_serving_engine_b200.parts.latent_attention import rotary_frequencies

    torch.manual_seed(7)
    rank, rot = 24, 12
    freq, factor = rotary_frequencies(ROT_SCALED)
    plain_freq, plain_factor = plain.rotary_frequencies(ROT_SCALED)
    assert factor == plain_factor and float((freq - plain_freq).abs().max()) == 0.0
    assert float((freq / plain.rotary_frequencies({"base": 50000.0, "dims": 12})[0]).min()) < 0.3    # the scaling acts
    positions = torch.tensor([0, 1, 63, 64, 1000, 4097, 9999], dtype=torch.int32)
    proj = torch.randn(len(positions), rank + rot)
    norm = torch.rand(rank) + 0.5
    cache = torch.zeros(2, 8, rank + rot, device="cuda")
    slots = torch.tensor([3, 9, 0, 15, 7, 8, 12], dtype=torch.int32)
    ops.latent_prepare(proj.cuda(), positions.cuda(), slots.cuda(), 1e-5, kv_off=0, rank=rank, kv_norm=norm.cuda(),
                       rot=rot, rot_dims=12, freq=freq.cuda(), rot_factor=factor, cache=cache)
    want_latent = plain.plain_norm(proj[:, :rank].double(), norm.double(), 1e-5)
    want_shared = plain.rotate(proj[:, rank:].double(), positions, ROT_SCALED)
    got = cache.view(16, -1).cpu()[slots.long()]
    assert float((got[:, :rank] - want_latent).abs().max()) <= 1e-5
    assert float((got[:, rank:] - want_shared).abs().max()) <= 1e-5
