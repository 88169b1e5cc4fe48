"""The adjoint's transposed solve with a stale approximate inverse.

The inverse is built on first use and kept; a later trajectory of other positions refines with it and renews
it while the contraction is too weak.  G scales with the surface, so positions scaled by s leave the error
matrix I - G X = (1 - s) I: the contraction per step is |1 - s|, squared by every renewal.  A context that
never had another state builds its own inverse; both solve to a relative residual of 1e-12, and the gradients
agree to 1e-9.
"""
import numpy as np
import pytest

from bem_b200 import _lib as L
from bem_b200 import mesh
from bem_b200.sim import ColocSim

pytestmark = pytest.mark.gpu


def gradient(sim, x, phi, w):
    def d(a):
        return a.ctypes.data_as(L._D)

    sim.set_state(x, phi, np.zeros(sim.N), 0.0)
    sim._check(sim._L.bem_adjoint_record(sim._h, 1e-3, 1))
    gx, gp = np.empty((sim.N, 3)), np.empty(sim.N)
    xb = np.ascontiguousarray(np.outer(w, [1.0, 0.5, -0.3]))
    sim._check(sim._L.bem_adjoint_backward(sim._h, d(xb), d(w), d(gx), d(gp)))
    return gx, gp


@pytest.mark.parametrize("nu", [4, 9])
@pytest.mark.parametrize("scale", [0.35, 0.9, 1.3, 1.6, 1.7])
def test_gradient_with_a_stale_inverse(nu, scale):
    v, f = mesh.bubble(nu, 1.0, (3.0, 0.0, 0.0))
    phi, w = 0.2 + 0.05 * v[:, 2], np.random.default_rng(nu).standard_normal(len(v))
    used, fresh = (ColocSim(v, f, solver="lu", epsilon=0.0) for _ in range(2))
    gradient(used, v, phi, w)
    for got, want in zip(gradient(used, scale * v, phi, w), gradient(fresh, scale * v, phi, w)):
        assert np.max(np.abs(got - want)) <= 1e-9 * np.max(np.abs(want))
    used.close()
    fresh.close()
