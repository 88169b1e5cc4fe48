"""Which form of the BiCGSTAB serves a size."""
import numpy as np
import pytest

from bem_b200.sim import ColocSim

from test_gpu_bicgstab import system, uv_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 1024, 1537, 2027, 2028, 2029, 2048, 2049, 4097, 6144])
def test_a_solve_is_one_launch_up_to_6144(n):
    # the matrix on the SMs while it fits (N = 2028), streamed above; LAPACK's solution to 1e-12 as in
    # test_gpu_bicgstab
    sim = ColocSim(*uv_sphere(n), solver="bicgstab")
    G, b = system(n, n)
    sim.reset_profile()
    x = sim.solve_system(G, b)
    assert sim.profile().kernel_launches == 1
    ref = np.linalg.solve(G, b)
    assert np.linalg.norm(x - ref) <= 1e-12 * np.linalg.norm(ref)
    sim.close()
