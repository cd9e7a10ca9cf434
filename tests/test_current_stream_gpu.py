"""Launches go to the current stream of the current device, as torch names it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_the_launch_stream_is_the_current_one():
    from llm_serving_engine_b200.kernels import ops

    torch.empty(1, device="cuda")
    assert ops._stream() == torch.cuda.current_stream().cuda_stream
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        assert ops._stream() == other.cuda_stream == torch.cuda.current_stream().cuda_stream
    assert ops._stream() == torch.cuda.current_stream().cuda_stream
