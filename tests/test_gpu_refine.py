"""The resident refinement of the mixed solver (one cooperative launch per round) at the edges of its size
classes, alone and over a batch's blocks.

solve_system takes any dense matrix, so the sizes are picked freely: fewer rows than a CTA holds, one more than a
multiple of the rows per CTA, the steps of the elements per thread (512, 1024, 2048, 4096), sizes with n % 4 = 1, 2,
3 (padded inverse; odd ones a copy of the matrix with an even stride), and above 6144 the separate launches.  The
solve ends at a relative residual of at most 1e-12; the matrices' condition number is below 4, so the solution is
within 4e-12 of LAPACK's (tolerance 1e-11).
"""
import numpy as np
import pytest

from bem_b200 import _lib as L
from bem_b200 import mesh
from bem_b200.batch import BubbleBatch
from bem_b200.sim import ColocSim

from test_gpu_bicgstab import system, uv_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "n", [5, 15, 16, 17, 130, 511, 512, 513, 1024, 1025, 1026, 2047, 2048, 2050, 2372, 4096, 4097, 4098, 6143, 6144, 6146]
)
def test_matches_lapack_at_size_edges(n):
    v, f = uv_sphere(n)
    sim = ColocSim(v, f, solver="mixed")
    for seed in (n, n + 1):  # the second matrix is refined with the first one's inverse, or that is renewed
        G, b = system(n, seed)
        x = sim.solve_system(G, b)
        ref = np.linalg.solve(G, b)
        assert np.linalg.norm(x - ref) <= 1e-11 * np.linalg.norm(ref)
    assert sim.stats().wait_expired == 0
    assert np.array_equal(sim.solve_system(G, np.zeros(n)), np.zeros(n))
    sim.close()


@pytest.mark.parametrize("n", [162, 1025, 2372])
def test_an_expired_wait_goes_on_with_separate_launches(n):
    v, f = uv_sphere(n)
    sim = ColocSim(v, f, solver="mixed")
    G, b = system(n, n)
    sim.solve_system(G, b)
    assert sim._L.bem_set_wait_limit(sim._h, 1) == L.BEM_OK
    ref = np.linalg.solve(G, b)
    for _ in range(2):
        assert np.linalg.norm(sim.solve_system(G, b) - ref) <= 1e-11 * np.linalg.norm(ref)
    assert sim.stats().wait_expired == 1
    sim.close()


PHYS = dict(p_inf=1.0, epsilon=1.0, sigma=0.0, gamma=1.4)


@pytest.mark.parametrize("limit", [None, 1])
@pytest.mark.parametrize(
    "nus",
    [
        [1, 2],  # 12 and 42 unknowns: far more CTAs than rows
        [4, 2, 8, 5, 11, 3, 6, 10],  # several classes (12 ... 1212), n % 4 = 0 and 2
        [2, 3] * 30,  # several blocks per team, padded and plain inverses in turn
        [0, 4],  # an odd block (47 unknowns): the separate launches
    ],
)
def test_batch_follows_single_simulations(nus, limit):
    # Both sides solve to a relative residual of 1e-12; one step of four stages keeps the states within 1e-10 and
    # the potentials within 1e-9.
    meshes = [mesh.bubble(nu, 0.7 + 0.02 * k, (2.5, 0.0, 0.0)) if nu else uv_sphere(47) for k, nu in enumerate(nus)]
    phi = np.concatenate([0.05 * np.sin(2 * v[:, 2]) for v, _ in meshes])
    bb = BubbleBatch(meshes, **PHYS)
    bb.set_block_params(amp=[0.5] * len(nus), omega=[2.0] * len(nus))
    bb.set_phi(phi)
    if limit:
        assert bb._L.bem_set_wait_limit(bb._h, limit) == L.BEM_OK
    bb.evolve_graph(2e-3, 2)
    assert bb.stats().wait_expired == (1 if limit and 0 not in nus else 0)
    X, P, S = bb.get_vertices(), bb.get_phi(), bb.get_psi()
    for b in range(0, len(nus), max(1, len(nus) // 8)):
        sl = bb.block(b)
        s = ColocSim(*meshes[b], pressurefield=(0.5, 2.0, 0.0), solver="lu", **PHYS)
        s.set_phi(phi[sl])
        for _ in range(2):
            s.evolve_system_RK4(2e-3, fixdt=True)
        for got, want, tol in ((X, s.get_vertices(), 1e-10), (P, s.get_phi(), 1e-9), (S, s.get_psi(), 1e-9)):
            assert np.max(np.abs(got[sl] - want)) <= tol * np.max(np.abs(want))
        s.close()
    bb.close()
