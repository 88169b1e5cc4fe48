"""The number of device allocations of a mixed context's set-up, which are most of a small context's set-up time.

It does not depend on the size: the padded copy of the inverse (N not a multiple of four) takes no allocation of
its own.
"""
import pytest

from bem_b200 import mesh
from bem_b200.sim import ColocSim

pytestmark = pytest.mark.gpu


def allocations(nu):
    from torch.profiler import ProfilerActivity, profile

    v, f = mesh.bubble(nu, 1.0, (2.0, 0.0, 0.0))
    with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as p:
        ColocSim(v, f, solver="mixed").close()
    n = sum(e.count for e in p.key_averages() if e.key == "cudaMalloc")
    if not n:
        pytest.skip("no runtime calls in the trace")
    return n


def test_allocations_do_not_depend_on_the_size():
    counts = [allocations(nu) for nu in (13, 10, 12)]  # N = 1692, 1002, 1442
    assert counts == counts[:1] * 3
