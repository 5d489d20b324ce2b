"""The stream that launches go to follows torch's current stream, per thread and device."""
import threading

import pytest
import torch

from metrale_inference_alpha_b200 import ops

pytestmark = pytest.mark.gpu


def test_launches_follow_the_current_stream():
    torch.zeros(1, device="cuda")
    current = lambda: torch.cuda.current_stream().cuda_stream
    side, seen = torch.cuda.Stream(), []
    assert ops._stream() == current()
    with torch.cuda.stream(side):
        assert ops._stream() == current() == side.cuda_stream
        t = threading.Thread(target=lambda: seen.append((ops._stream(), current())))
        t.start(), t.join()
    assert ops._stream() == current() != side.cuda_stream
    assert seen[0][0] == seen[0][1] != side.cuda_stream
