"""The LU's cluster panel at the edges of its layout: panels of one to several CTAs, of 255 to 257 and 4096 to
4098 rows (256 and 512 threads per CTA), last panels narrower than a block of 8 columns, and columns without
a valid candidate.  Partial pivoting on Gaussian matrices interchanges rows at almost every column; the
solution is compared with LAPACK's at 1e-10 (as tests/test_gpu_lu.py), the residual at 1e-14.
"""
import numpy as np
import pytest

from bem_b200 import _lib as L
from bem_b200.sim import ColocSim
from test_gpu_bicgstab import uv_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 63, 64, 65, 72, 127, 255, 256, 257, 513, 1031, 4097])
def test_panel_edges_against_lapack(n):
    sim = ColocSim(*uv_sphere(n), solver="lu")
    r = np.random.default_rng(n)
    A, b = np.asfortranarray(r.standard_normal((n, n))), r.standard_normal(n)
    x, ref = sim.solve_system(A, b), np.linalg.solve(A, b)
    assert np.max(np.abs(x - ref)) <= 1e-10 * np.max(np.abs(ref))
    assert np.linalg.norm(A @ x - b) <= 1e-14 * np.linalg.norm(A, 1) * np.linalg.norm(x)
    assert sim.stats().wait_expired == 0
    sim.close()


def test_ties_take_the_first_row():
    # every entry of a column is +-1: the pivot is the first row of each step's order, as in LAPACK
    n = 300
    r = np.random.default_rng(9)
    A = np.asfortranarray(np.sign(r.standard_normal((n, n))))
    b = r.standard_normal(n)
    sim = ColocSim(*uv_sphere(n), solver="lu")
    ref = np.linalg.solve(A, b)
    assert np.max(np.abs(sim.solve_system(A, b) - ref)) <= 1e-10 * np.max(np.abs(ref))
    sim.close()


def test_nan_and_zero_columns():
    # a NaN spreads into the solution and nothing else happens; a zero column is a zero pivot
    n = 200
    r = np.random.default_rng(4)
    A, b = np.asfortranarray(r.standard_normal((n, n))), r.standard_normal(n)
    sim = ColocSim(*uv_sphere(n), solver="lu")
    bad = A.copy(order="F")
    bad[:, 70] = np.nan
    assert np.isnan(sim.solve_system(bad, b)).any()
    bad[:, 70] = 0.0
    with pytest.raises(L.BemError) as e:
        sim.solve_system(bad, b)
    assert e.value.code == L.BEM_ERR_SINGULAR
    ref = np.linalg.solve(A, b)
    assert np.max(np.abs(sim.solve_system(A, b) - ref)) <= 1e-10 * np.max(np.abs(ref))
    sim.close()
