"""Launches go to the caller's current stream."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_handle_is_the_current_stream():
    from glide_b200 import _native as N
    assert N.stream_handle() == torch.cuda.current_stream().cuda_stream
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        assert N.stream_handle() == s.cuda_stream != 0
    assert N.stream_handle() == torch.cuda.current_stream().cuda_stream
    assert N.stream_handle(s) == s.cuda_stream
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        assert N.stream_handle() == torch.cuda.current_stream().cuda_stream
        torch.zeros(1, device="cuda")
