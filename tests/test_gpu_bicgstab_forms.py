"""Which form of the BiCGSTAB serves a size, and right-hand sides of very small and large magnitude."""
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


@pytest.mark.parametrize("n", [42, 700, 1500, 2345, 4097])
@pytest.mark.parametrize("k", [-498, -440, 488])
def test_a_scaled_right_hand_side(n, k):
    # b 2^k, whose squared norm is near the ends of the FP64 range; at 2^-498 (1e-150) the dot products of the last
    # iterations fall below 1e-308.  Their rounding is then that of denormals, so the solution is met to 1e-10.
    G, b = system(n, n)
    sim = ColocSim(*uv_sphere(n), solver="bicgstab")
    ref = np.linalg.solve(G, b)
    x = sim.solve_system(G, b * 2.0**k) * 2.0**-k
    assert np.linalg.norm(x - ref) <= 1e-10 * np.linalg.norm(ref)
    sim.close()
