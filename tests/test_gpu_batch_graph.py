"""Settings changed between two calls that replay a batch's captured step.

A captured step holds its launch arguments; a change of a setting that it holds has to reach the next step.
"""
import numpy as np
import pytest

from bem_b200 import _lib as L
from bem_b200 import mesh
from bem_b200.batch import BubbleBatch

pytestmark = pytest.mark.gpu

PHYS = dict(p_inf=1.0, epsilon=1.0, sigma=0.0, gamma=1.4)


def batch():
    meshes = [mesh.bubble(nu, 0.8, (2.5, 0.0, 0.0)) for nu in (4, 3, 6)]
    bb = BubbleBatch(meshes, **PHYS)
    bb.set_phi(np.concatenate([0.05 * np.sin(2 * v[:, 2]) for v, _ in meshes]))
    return bb


def test_the_wait_limit_reaches_a_captured_step():
    a, b = batch(), batch()
    for bb in (a, b):
        bb.evolve_graph(2e-3, 1)
    assert b._L.bem_set_wait_limit(b._h, 1) == L.BEM_OK
    a.evolve_graph(2e-3, 1)
    b.evolve_graph(2e-3, 1)
    assert a.stats().wait_expired == 0 and b.stats().wait_expired == 1
    # the separate launches solve to the same relative residual of 1e-12
    assert np.max(np.abs(a.get_vertices() - b.get_vertices())) <= 1e-11
    assert np.max(np.abs(a.get_phi() - b.get_phi())) <= 1e-10
    a.close()
    b.close()


def test_parameters_reach_a_captured_step():
    a, b = batch(), batch()
    a.evolve_graph(2e-3, 1)
    b.evolve_rk4_steps(2e-3, 1)
    for bb in (a, b):
        bb._update(p_inf=2.0, gamma=1.1)
    a.evolve_graph(2e-3, 2)
    b.evolve_rk4_steps(2e-3, 2)
    assert np.array_equal(a.get_vertices(), b.get_vertices())
    assert np.array_equal(a.get_phi(), b.get_phi())
    a.close()
    b.close()
