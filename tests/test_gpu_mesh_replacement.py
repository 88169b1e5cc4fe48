"""One context that holds a single mesh, then a batch, then a single mesh again, against fresh contexts.

Every buffer of a mesh is freed or handed on when another replaces it, and a batch has none of the single
system's solver buffers; nothing that a context kept from its last mesh may reach the next one.  The
kernels sum in a fixed order, so the results are those of fresh contexts bit for bit.
"""
import numpy as np
import pytest

from bem_b200 import _lib as L
from bem_b200 import mesh
from bem_b200.batch import BubbleBatch
from bem_b200.sim import ColocSim

pytestmark = pytest.mark.gpu

PHYS = dict(p_inf=1.0, epsilon=1.0, sigma=0.0, gamma=1.4)


def set_mesh(sim, v, f):
    v, f = np.ascontiguousarray(v), np.ascontiguousarray(f, dtype=np.int64)
    sim._check(sim._L.bem_set_mesh(sim._h, len(v), v.ctypes.data_as(L._D), len(f), f.ctypes.data_as(L._I64)))
    sim.N, sim.M = len(v), len(f)


def set_blocks(sim, meshes):
    v, f = mesh.join([(np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.int64)) for a, b in meshes])
    v, f = np.ascontiguousarray(v), np.ascontiguousarray(f, dtype=np.int64)
    off = np.concatenate([[0], np.cumsum([len(a) for a, _ in meshes])]).astype(np.int64)
    sim._check(sim._L.bem_set_mesh_blocks(sim._h, len(v), v.ctypes.data_as(L._D), len(f), f.ctypes.data_as(L._I64),
                                          len(meshes), off.ctypes.data_as(L._I64)))
    sim.N, sim.M = len(v), len(f)


# the batch's unknowns in all: more than the single mesh's, fewer, and past the resident solvers' sizes
@pytest.mark.parametrize("solver", ["lu", "bicgstab", "mixed"])
@pytest.mark.parametrize("nu,nus", [(2, [4, 3, 5]), (9, [2, 3]), (3, [8] * 12)])
def test_single_blocks_single(solver, nu, nus):
    first, second = mesh.bubble(nu, 1.0, (2.0, 0.0, 0.0)), mesh.bubble(nu + 1, 0.9, (2.2, 0.0, 0.0))
    meshes = [mesh.bubble(k, 0.8 + 0.05 * i, (2.5, 0.0, 0.0)) for i, k in enumerate(nus)]
    phi = np.concatenate([0.05 * np.sin(2 * v[:, 2]) for v, _ in meshes])

    def single(sim, v):
        return sim.position_t(0.1 + 0.05 * v[:, 2], return_psi=True)

    def steps(sim):
        sim.set_phi(phi)
        sim._check(sim._L.bem_evolve_rk4_graph(sim._h, 2e-3, 2))
        return sim.get_vertices(), sim.get_phi(), sim.get_psi()

    sim = ColocSim(*first, solver=solver, **PHYS)
    single(sim, first[0])
    set_blocks(sim, meshes)
    got = steps(sim)
    set_mesh(sim, *second)
    back = single(sim, second[0])
    assert sim.stats().wait_expired == 0
    fresh = BubbleBatch(meshes, **PHYS)
    for a, b in zip(got, steps(fresh)):
        assert np.array_equal(a, b)
    alone = ColocSim(*second, solver=solver, **PHYS)
    for a, b in zip(back, single(alone, second[0])):
        assert np.array_equal(a, b)
    for s in (sim, fresh, alone):
        s.close()
