"""The delta memory's front end from partial sums, and its chunked scan with one block an SM and with several."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def _step(lengths, slots):
    as_int = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    start = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    return SimpleNamespace(segment_of_token=as_int([i for i, count in enumerate(lengths) for _ in range(count)]),
                           segment_start=as_int(start), segment_state_slot=as_int(slots), decode_only=all(c == 1 for c in lengths))


@pytest.mark.parametrize("tokens", [1, 5, 256, 259, 1025])
@pytest.mark.parametrize("dim,taps", [(128, 4), (24, 3), (150, 4), (9, 4)])
def test_the_front_end_of_partial_sums_and_of_whole_rows(tokens, dim, taps):
    """Halves add up without rounding, so both forms see the same numbers and have to give the same ones; the rows end inside
    the four that are fetched together, and a request begins there."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(31)
    groups, heads, vdim, rank = 2, 2, 20, 6
    channels = 2 * groups * dim + heads * vdim
    rows = torch.randn(tokens, -(-(channels + heads + rank) // 4) * 4, device="cuda")
    conv = torch.randn(channels, taps, device="cuda")
    windows = torch.randn(2, taps - 1, channels, device="cuda")
    portions = [tokens] if tokens < 3 else [tokens - 2, 2]
    got = []
    for given in (rows, torch.stack([0.5 * rows, 0.5 * rows]), torch.stack([0.25 * rows] * 2 + [0.5 * rows] + [0 * rows] * 2)):
        state, low = windows.clone(), torch.empty(tokens, 16, device="cuda")
        parts = ops.delta_prepare(given, conv, state, _step(portions, slots=list(range(len(portions)))), low, groups, heads, dim, vdim,
                                  rank, dim ** -0.5)
        got.append((*parts, low, state))
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))


@pytest.mark.parametrize("heads,dim", [(10, 128), (11, 60), (10, 200)])
def test_a_scan_of_more_blocks_than_sms_is_the_scans_of_its_requests(heads, dim):
    """Two requests together are 160 or more blocks (several an SM), each alone at most 88 (an SM each): the same numbers."""
    from llm_serving_engine_b200.kernels import ops

    torch.manual_seed(32)
    lengths, vdim = (33, 100), 128
    total = sum(lengths)
    q, k = (torch.nn.functional.normalize(torch.randn(total, heads, dim, device="cuda"), dim=-1).view(total, -1) for _ in range(2))
    v, beta = torch.randn(total, heads * vdim, device="cuda"), torch.rand(total, heads, device="cuda")
    z, dt_bias, a_log = (torch.randn(*shape, device="cuda") for shape in ((total, heads * dim), (heads * dim,), (heads,)))
    before = torch.randn(2, heads, dim, vdim, device="cuda")

    def scan(rows, state, counts):
        step, out = _step(list(counts), slots=list(range(len(counts)))), torch.empty(sum(counts), heads * vdim, device="cuda")
        ops.delta_scan(q[rows], k[rows], v[rows], beta[rows], z[rows], dt_bias, a_log, state, step.segment_start,
                       step.segment_state_slot, out, heads, heads, dim, vdim)
        return out
    together = before.clone()
    out = scan(slice(0, total), together, lengths)
    at = 0
    for index, count in enumerate(lengths):
        alone = before[index:index + 1].clone()
        assert torch.equal(out[at:at + count], scan(slice(at, at + count), alone, (count,)))
        assert torch.equal(together[index], alone[0])
        at += count
