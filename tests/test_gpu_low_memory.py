"""A mixed context whose padded inverse does not fit in the GPU's memory.

The copy serves the resident refinement only, so without it the solves run as separate launches.  The rest of
the memory is taken by one tensor, sized from what an equal context held, so that everything but the copy fits.
"""
import numpy as np
import pytest

from bem_b200.sim import ColocSim

from test_gpu_bicgstab import system, uv_sphere

pytestmark = pytest.mark.gpu


def test_without_the_padded_inverse():
    import gc

    import torch

    gc.collect()
    n = 4098  # not a multiple of four: the copy takes 4 n (n + 2) bytes, 67 MB
    v, f = uv_sphere(n)
    G, b = system(n, n)
    ref = np.linalg.solve(G, b)
    sim = ColocSim(v, f, solver="mixed")
    x = sim.solve_system(G, b)  # also loads every kernel of the solve
    torch.cuda.synchronize()
    with_sim = torch.cuda.mem_get_info()[0]
    sim.close()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    rest = free - with_sim - 4 * n * (n + 2) // 2  # half of the copy short
    held = torch.empty(free - rest, dtype=torch.uint8, device="cuda")
    try:
        sim = ColocSim(v, f, solver="mixed")
        sim.solve_system(G, b)
        sim.reset_profile()
        y = sim.solve_system(G, 2.0 * b) / 2.0
        assert sim.profile().kernel_launches > 1
        assert sim.stats().fp64_fallbacks == 0
        sim.close()
    finally:
        del held
        torch.cuda.empty_cache()
    for got in (x, y):
        assert np.linalg.norm(got - ref) <= 1e-11 * np.linalg.norm(ref)
