"""The autotuner's times are those of the steps that the batch then runs."""
import pytest
import torch

from uq_b200 import workloads as W
from uq_b200.solver import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_autotuned_time_is_that_of_a_step(cuda_device, prec):
    """A small solve, where a step taken phase by phase (every part a launch of
    its own, none overlapped) is more than twice as long as one from a graph."""
    b = Batch([W.couette(nx=64, ny=128, seed=1)], prec)
    stream = torch.cuda.ExternalStream(b.stream)
    times = []
    for _ in range(6):
        a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        b.step(64)
        e.record(stream)
        e.synchronize()
        times.append(a.elapsed_time(e) / 64)
    tuned = min(b.autotune([(32, 8)], steps=64)[1][32, 8] for _ in range(3))
    assert min(times) / 1.5 < tuned < 1.5 * min(times), (tuned, times)
    b.close()
