"""A single velocity evaluation of a batch (position_t outside a step) against the single simulations.

The evaluation solves every block itself, so it has to look at the solve's status before it hands anything
out: the resident refinement's exchange waits may run out (status read, counted once, the solve repeated
with the separate launches), and a batch that has not stepped has no approximate inverses yet.  Both sides
solve to a relative residual of 1e-12; psi and the velocities are met to 1e-9 as in test_gpu_batch.
"""
import numpy as np
import pytest

from bem_b200 import _lib as L
from bem_b200 import mesh
from bem_b200.batch import BubbleBatch
from bem_b200.sim import ColocSim

from test_gpu_bicgstab import uv_sphere

pytestmark = pytest.mark.gpu

PHYS = dict(p_inf=1.0, epsilon=1.0, sigma=0.0, gamma=1.4)


def make(nus):
    meshes = [mesh.bubble(nu, 0.7 + 0.02 * k, (2.5, 0.0, 0.0)) if nu else uv_sphere(47) for k, nu in enumerate(nus)]
    phi = np.concatenate([0.05 * np.sin(2 * v[:, 2]) + 0.1 for v, _ in meshes])
    return meshes, phi, BubbleBatch(meshes, **PHYS)


def check(bb, meshes, phi, verts=None):
    vel, psi = bb.position_t(phi, verts=verts, return_psi=True)
    x = bb.get_vertices() if verts is None else verts
    for b, (v, f) in enumerate(meshes):
        sl = bb.block(b)
        s = ColocSim(v, f, solver="lu", **PHYS)
        want = s.position_t(phi[sl], verts=x[sl], return_psi=True)
        s.close()
        for got, ref in zip((vel[sl], psi[sl]), want):
            assert np.max(np.abs(got - ref)) <= 1e-9 * np.max(np.abs(ref))


@pytest.mark.parametrize("nus", [[1, 2], [4, 2, 8, 5, 3, 6], [0, 4]])
@pytest.mark.parametrize("stepped", [False, True])
def test_an_expired_wait(nus, stepped):
    meshes, phi, bb = make(nus)
    bb.set_phi(phi)
    if stepped:
        bb.evolve_graph(2e-3, 1)
    assert bb._L.bem_set_wait_limit(bb._h, 1) == L.BEM_OK
    expired = 0 if 0 in nus else 1  # an odd block: separate launches from the start, no wait
    check(bb, meshes, phi)
    assert bb.stats().wait_expired == expired
    # nothing is left over for the calls that follow
    repeated = bb.stats().gmres_fallbacks
    check(bb, meshes, 2.0 * phi)
    bb.evolve_graph(2e-3, 1)
    assert bb.stats().wait_expired == expired and bb.stats().gmres_fallbacks == repeated
    bb.close()


def test_before_the_first_step_and_at_other_positions():
    meshes, phi, bb = make([3, 5, 4])
    check(bb, meshes, phi)
    # inverses of the current surface, positions scaled by 1.4: a contraction of 0.4 per step does not meet the
    # tolerance in a solve's eight steps
    check(bb, meshes, phi, verts=np.ascontiguousarray(1.4 * bb.get_vertices()))
    check(bb, meshes, phi)
    bb.close()


def test_values_that_are_not_finite_spread_as_in_a_single_system():
    meshes, phi, bb = make([3, 4])
    bb.set_phi(phi)
    bb.evolve_graph(2e-3, 1)
    bad = phi.copy()
    bad[3] = np.nan
    vel, psi = bb.position_t(bad, return_psi=True)
    assert np.isnan(psi[bb.block(0)]).all() and np.isfinite(psi[bb.block(1)]).all()
    bb.close()
