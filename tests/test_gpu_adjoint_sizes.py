"""The adjoint at the edges of its kernels' sizes, against central differences of the FP64 forward path.

The pair pass takes 128 triangles by a chunk of rows per CTA (fewer rows than a warp has lanes, one chunk, several
CTAs, several sub-chunks of 128 rows), the transposed solve is resident with padded copies (n % 4 = 0, 2 and odd)
and goes on with separate launches after an expired wait.  Tolerance 1e-5 relative to the directional derivative
as in test_gpu_adjoint: the central difference at h = 1e-6 has a truncation error of (h / edge)^2 < 1e-9 and a
rounding error of 1e-13 / h.
"""
import numpy as np
import pytest

from bem_b200 import mesh
from bem_b200.sim import ColocSim

from test_gpu_adjoint import PHYS, adjoint_grad, check, directions, fd_gpu
from test_gpu_bicgstab import uv_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12, 42, 47, 162, 253, 812, 4002])
def test_gradient_at_size_edges(n):
    nu = {12: 1, 42: 2, 162: 4, 812: 9, 4002: 20}.get(n)
    v, f = mesh.bubble(nu, 1.0, (2.0, 0.0, 0.0)) if nu else uv_sphere(n)
    assert len(v) == n
    rng = np.random.default_rng(n)
    phi = 0.3 + 0.02 * rng.standard_normal(n)
    w = rng.standard_normal(n)
    dt, steps = 1e-3, 2
    _, gx, gp = adjoint_grad(v, f, phi, w, dt, steps, **PHYS)
    dirs = directions(n, 2, seed=n)
    check(gx, gp, fd_gpu(v, f, phi, w, dt, steps, dirs, **PHYS), dirs)


@pytest.mark.parametrize("nu", [4, 9])
def test_an_expired_wait_in_the_transposed_solve(nu, monkeypatch):
    v, f = mesh.bubble(nu, 1.0, (2.0, 0.0, 0.0))
    n = len(v)
    rng = np.random.default_rng(nu)
    phi, w = 0.3 + 0.02 * rng.standard_normal(n), rng.standard_normal(n)
    _, gx, gp = adjoint_grad(v, f, phi, w, 1e-3, 2, **PHYS)
    sims = []

    class Short(ColocSim):
        def __init__(self, *a, **k):
            super().__init__(*a, **k)
            self._check(self._L.bem_set_wait_limit(self._h, 1))
            sims.append(self)

    monkeypatch.setattr("test_gpu_adjoint.ColocSim", Short)
    _, hx, hp = adjoint_grad(v, f, phi, w, 1e-3, 2, **PHYS)
    assert sims[0].stats().wait_expired >= 1
    # both sides solve to a relative residual of 1e-12
    assert np.max(np.abs(hx - gx)) <= 1e-9 * np.max(np.abs(gx))
    assert np.max(np.abs(hp - gp)) <= 1e-9 * np.max(np.abs(gp))
