"""The product on pairs of SMs (``csrc/gemm_pairs.cu``): gated, and over groups of rows, at the edges of its tiles, against
float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def ops():
    from llm_serving_engine_b200.kernels import ops
    return ops


def _act(kind, g, u, limit):
    if kind == "silu":
        return g * torch.sigmoid(g) * u
    if kind == "relu":
        return g.clamp(min=0) * u
    if kind == "gelu_tanh":
        return 0.5 * g * (1 + torch.tanh(0.7978845608028654 * (g + 0.044715 * g ** 3))) * u
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1)


def _check(got, want, x, w):
    """Rounded once to bfloat16 (2^-9 of the value; 2^-8 allows for a neighbour), and float32 sums of k terms: k 2^-24 of the
    magnitudes, times what the activation and the other factor make of it (all factors here are below 16)."""
    sums = x.shape[1] * 2.0 ** -24 * float((x.abs().double() @ w.abs().double().t()).max())
    assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 16 * sums + 1e-6).all())


def _random(rows, k, scale=1.0):
    return (torch.randn(rows, k, device=DEV) * scale).bfloat16()


@pytest.mark.parametrize("rows,k,inter,kind", [(1, 64, 128, "silu"), (31, 72, 8, "silu"), (33, 64, 136, "relu"), (96, 200, 320, "gelu_tanh"),
                                               (256, 128, 1000, "silu"), (257, 448, 64, "clamped_swish"), (300, 512, 264, "silu"),
                                               (522, 64, 9480, "clamped_swish"), (1349, 96, 2000, "silu")])
def test_gated_product(rows, k, inter, kind):
    torch.manual_seed(rows + k)
    x, w = _random(rows, k), _random(2 * inter, k, k ** -0.5)
    out = torch.full((rows, inter + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    ops().gated_product(x, w, out[:, :inter], kind, 1.5)
    sums = x.double() @ w.double().t()
    _check(out[:, :inter], _act(kind, sums[:, :inter], sums[:, inter:], 1.5), x, w)
    assert bool((out[:, inter:] == 7.0).all())             # nothing beside the results is written
    from llm_serving_engine_b200.kernels import library
    assert library.load().lse_gemm_pairs_status() == 0


@pytest.mark.parametrize("counts,k,columns,whole,whole_columns,kind", [
    ([64], 64, 64, 0, 0, "silu"), ([0, 1, 33, 0, 300], 128, 192, 40, 72, "clamped_swish"), ([256, 522, 5], 192, 128, 257, 200, "silu"),
    ([2, 0, 3] + [1] * 60, 72, 64, 1, 8, "silu"), ([0, 0], 64, 64, 70, 136, "clamped_swish"),
    ([0, 5, 300, 0] * 8 + [0] * 32 + [7, 0, 258] + [0, 1, 40] * 60 + [3], 64, 64, 33, 64, "silu"), ([1] * 31 + [0] * 224 + [520], 64, 128, 0, 0, "silu")])
def test_groups_of_rows_with_weights_of_their_own(counts, k, columns, whole, whole_columns, kind):
    """Both products of a mixture of experts: rows behind the last group stay as they are, a group may have none."""
    torch.manual_seed(sum(counts) + k)
    used, groups = sum(counts), len(counts)
    x, everyone = _random(used + 3, k), _random(whole, k) if whole else None
    offsets = torch.tensor(counts, device=DEV).cumsum(0).int()
    w = _random(2 * (groups * columns + whole_columns), k, k ** -0.5)
    act = torch.full((used + 3, columns), 7.0, device=DEV, dtype=torch.bfloat16)
    scale = torch.rand(whole, device=DEV) if whole else None
    if whole:
        scale[0] = 0.0
        w[2 * groups * columns] = float("nan")             # a row whose factor is zero takes nothing from anywhere
    shared = torch.empty(whole, whole_columns, device=DEV, dtype=torch.bfloat16) if whole else None
    ops().gated_product_groups(x, offsets, act, 1.5, everyone, shared, scale, 2.0, w, kind)
    assert bool((act[used:] == 7.0).all())
    start = 0
    for group, count in enumerate(counts):
        if count:
            piece = w[2 * group * columns:2 * (group + 1) * columns]
            sums = x[start:start + count].double() @ piece.double().t()
            _check(act[start:start + count], _act(kind, sums[:, :columns], sums[:, columns:], 1.5), x[start:start + count], piece)
        start += count
    if whole:
        assert bool((shared[0] == 0).all())
        piece = w[2 * groups * columns:].clone()
        piece[0] = 0
        sums = everyone.double() @ piece.double().t()
        want = _act(kind, sums[:, :whole_columns], sums[:, whole_columns:], 2.0) * scale.double()[:, None]
        _check(shared[1:, 1:], want[1:, 1:], everyone, piece)
        assert kind == "clamped_swish" or bool(torch.isnan(shared[1:, 0]).all())      # a clamp takes the number beside a NaN

    width = 328
    down_w = _random(width, groups * columns + whole_columns, columns ** -0.5)
    act[used:] = 0
    if whole:
        shared = _random(whole, whole_columns)
    down = torch.full((used + 3, width), 7.0, device=DEV, dtype=torch.bfloat16)
    total = torch.empty(whole, width, device=DEV) if whole else None
    ops().product_groups(act, offsets, down, shared, total, down_w)
    assert bool((down[used:] == 7.0).all())
    start = 0
    for group, count in enumerate(counts):
        if count:
            piece = down_w[:, group * columns:(group + 1) * columns]
            _check(down[start:start + count], act[start:start + count].double() @ piece.double().t(), act[start:start + count], piece)
        start += count
    if whole:
        piece = down_w[:, groups * columns:]
        want = shared.double() @ piece.double().t()
        bound = whole_columns * 2.0 ** -24 * (shared.abs().double() @ piece.abs().double().t()) + 1e-6
        assert bool(((total.double() - want).abs() <= bound).all())


def test_what_the_product_does_not_take():
    o = ops()
    x, w = _random(40, 64), _random(128, 64)
    assert o.gemm_pairs_ok(x, w)
    assert not o.gemm_pairs_ok(x.float(), w) and not o.gemm_pairs_ok(_random(40, 60), _random(128, 60))
    assert not o.gemm_pairs_ok(torch.empty(0, 64, device=DEV, dtype=torch.bfloat16), w)
    assert not o.gemm_pairs_ok(_random(41, 64).flatten()[4:4 + 40 * 64].view(40, 64), w)
    with pytest.raises(o.KernelError):
        o.gated_product(x.float(), w, torch.empty(40, 64, device=DEV, dtype=torch.bfloat16))


@pytest.mark.parametrize("wrong", ["strided x", "strided whole", "float32 x", "float16 weight", "misaligned whole", "misaligned weight",
                                   "rows of the result", "columns apart", "float32 result", "few weights", "int64 ends", "ends apart",
                                   "factors", "float16 result"])
def test_what_the_products_over_groups_do_not_take(wrong):
    """Every operand is looked at before a launch, in both products: nothing is read as something that it is not."""
    o = ops()

    def refused(gated):
        groups, columns, k, rows, whole = 2, 64, 128, 40, 24
        x, everyone = _random(rows, k), _random(whole, k)
        offsets, scale = torch.tensor([10, 40], device=DEV, dtype=torch.int32), torch.rand(whole, device=DEV)
        weight = _random(2 * (groups + 1) * columns, k) if gated else _random(columns, (groups + 1) * k)
        out, total = (torch.empty(count, columns, device=DEV, dtype=torch.bfloat16) for count in (rows, whole))
        if wrong == "strided x": x = _random(k, rows).t()
        if wrong == "strided whole": everyone = _random(whole, 2 * k)[:, ::2]
        if wrong == "float32 x": x = x.float()
        if wrong == "float16 weight": weight = weight.half()
        if wrong == "misaligned whole": everyone = _random(whole + 1, k).flatten()[4:4 + whole * k].view(whole, k)
        if wrong == "misaligned weight": weight = _random(weight.shape[0] + 1, weight.shape[1]).flatten()[1:1 + weight.numel()].view(weight.shape)
        if wrong == "rows of the result": out = out[1:]
        if wrong == "columns apart": total = torch.empty(columns, whole, device=DEV, dtype=torch.bfloat16).t()
        if wrong == "float32 result": out = out.float()
        if wrong == "float16 result": out = out.half()
        if wrong == "few weights": weight = weight[:, :-64] if not gated else weight[:-64]
        if wrong == "int64 ends": offsets = offsets.long()
        if wrong == "ends apart": offsets = torch.zeros(4, device=DEV, dtype=torch.int32)[::2]
        if wrong == "factors": scale = scale.half()
        if not gated and wrong in ("float32 result", "factors"):      # this product's results may be float32, and it has no factors
            return
        with pytest.raises(o.KernelError):
            if gated:
                o.gated_product_groups(x, offsets, out, 0.0, everyone, total, scale, 0.0, weight, "silu")
            else:
                o.product_groups(x, offsets, out, everyone, total, weight)
    refused(True)
    refused(False)


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("rows", [40, 4000])
def test_a_wait_that_runs_out_is_reported_and_the_kernel_returns(gated, rows):
    """Half of x's rows do not come, and the wait for them gives up (after some tenths of a second); the other waits of both blocks of the pair
    see it, for pairs of one tile and of several.  The launch ends, the status word reaches
    the host as the sampler reads it, and after a reset the product is right.  Nothing faults: a load is simply not started."""
    from llm_serving_engine_b200.kernels import library
    from llm_serving_engine_b200.sampling.sampler import GenerationConfig, Sampler

    o = ops()
    torch.manual_seed(rows)
    k, columns = 448, 2560
    x, offsets = _random(rows, k), torch.tensor([rows], device=DEV, dtype=torch.int32)
    weight = _random(2 * columns if gated else columns, k, k ** -0.5)
    out = torch.empty(rows, columns, device=DEV, dtype=torch.bfloat16)

    def product():
        if gated:
            o.gated_product(x, weight, out)
        else:
            o.product_groups(x, offsets, out, None, None, weight)
        torch.cuda.synchronize()

    sampler = Sampler(16, 1, torch.device(DEV))
    product()
    assert library.load().lse_gemm_pairs_status() == 0
    o.gemm_pairs_test_hook(withhold=True)
    try:
        product()
        assert library.load().lse_gemm_pairs_status() == 1
        ticket = sampler.launch(torch.zeros(1, 16, device=DEV), [GenerationConfig()], [0])
        with pytest.raises(o.KernelError, match="the product on pairs of SMs"):
            sampler.collect(ticket)
    finally:
        o.gemm_pairs_test_hook()
        o.kernel_status_reset()
    product()
    sums = x.double() @ weight.double().t()
    _check(out, _act("silu", sums[:, :columns], sums[:, columns:], 0.0) if gated else sums, x, weight)
    assert library.load().lse_gemm_pairs_status() == 0


@pytest.mark.parametrize("width,rows,pairs", [(2048, 401, True), (2560, 400, True), (2560, 401, False), (2560, 1000, False)])
def test_which_experts_take_the_products_over_groups(width, rows, pairs, monkeypatch):
    """Two experts of which each row chooses one: up to 200 rows an expert on average, or up to 2,048 columns.  Either way a value is
    rounded at most five times to bfloat16 (2^-9 each) on its way to the result: 2^-6 of the whole between the two, in the 2-norm."""
    from llm_serving_engine_b200.parts import FEED_FORWARDS
    from llm_serving_engine_b200.parts.base import BuildContext

    o = ops()
    torch.manual_seed(rows + width)
    ff = 64
    weights = {"router": _random(2, width, width ** -0.5)}
    for index in range(2):
        weights.update({f"e{index}.gate": _random(ff, width, width ** -0.5), f"e{index}.up": _random(ff, width, width ** -0.5),
                        f"e{index}.down": _random(width, ff, ff ** -0.5)})
    params = {"experts": 2, "top": 1, "ff": ff, "activation": "silu", "correction": False}
    part = FEED_FORWARDS.get("clamped_moe")(params, weights, BuildContext(torch.bfloat16, torch.device(DEV), width, 0, 64))
    calls = []
    product = o.product_groups
    monkeypatch.setattr(o, "product_groups", lambda *given: calls.append(1) or product(*given))
    x = _random(rows, width)
    got = part.forward(x)
    assert len(calls) == pairs
    monkeypatch.setattr(part, "_pairs_wanted", lambda tokens: not pairs)
    other = part.forward(x)
    assert len(calls) == 1
    assert float((got - other).norm() / other.norm()) <= 2.0 ** -6


@pytest.mark.parametrize("rows,in_the_product", [(1235, False), (1236, True), (1300, False), (2048, True)])
def test_which_rows_of_a_feed_forward_take_the_product_with_its_gate(rows, in_the_product, monkeypatch):
    """The dense feed-forward around the rows from which the gate goes into the product (1.7e10 multiplications and additions), and where
    the last tiles would leave the GPU idle, against float64.  A value of the gated product carries up to three roundings to bfloat16 (2^-9 of it each; one where the gate
    is inside), the result one more: 2^-7 of the whole in the 2-norm."""
    from llm_serving_engine_b200.parts import FEED_FORWARDS
    from llm_serving_engine_b200.parts.base import BuildContext

    o = ops()
    if o.sm_count() != 148:
        pytest.skip("the rows are those of 148 SMs")
    torch.manual_seed(rows)
    hidden, inter = 1536, 8960
    weights = {name: _random(*shape, scale=shape[1] ** -0.5) for name, shape in (
        ("gate_proj.weight", (inter, hidden)), ("up_proj.weight", (inter, hidden)), ("down_proj.weight", (hidden, inter)))}
    part = FEED_FORWARDS.get("swiglu")({"intermediate_size": inter}, weights, BuildContext(torch.bfloat16, torch.device(DEV), hidden, 0, 64))
    calls = []
    product = o.gated_product
    monkeypatch.setattr(o, "gated_product", lambda *given: calls.append(1) or product(*given))
    x = _random(rows, hidden)
    got = part.forward(x).double()
    assert bool(calls) == in_the_product
    gate, up, down = (weights[name + "_proj.weight"].double() for name in ("gate", "up", "down"))
    want = _act("silu", x.double() @ gate.t(), x.double() @ up.t(), 0.0) @ down.t()
    assert float((got - want).norm() / want.norm()) <= 2.0 ** -7
