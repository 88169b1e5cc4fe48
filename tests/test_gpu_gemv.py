"""The refinement GEMVs of matrices larger than L2 (two rows per thread, no L2 policy), through the mixed solve.

Sizes: the first even one past the rule (its last CTA has 94 of 512 rows, its second row block none), an odd
number of 256-row blocks, all rows of the last CTA in use, and the odd size that keeps one row per thread.  The
mixed solve's relative residual is 1e-12 and the matrix's condition about 2, so LAPACK's solution is met to
1e-11; the residual norms steer the refinement, so a wrong row-block sum would end it early or never.
"""
import numpy as np
import pytest

from bem_b200.sim import ColocSim
from test_gpu_bicgstab import system, uv_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4701, 4702, 5376, 5632])
def test_mixed_solve_with_streaming_gemvs(n):
    sim = ColocSim(*uv_sphere(n), solver="mixed")
    G, b = system(n, n)
    x, ref = sim.solve_system(G, b), np.linalg.solve(G, b)
    assert np.linalg.norm(x - ref) <= 1e-11 * np.linalg.norm(ref)
    st = sim.stats()
    assert st.last_rel_residual <= 1e-12 and st.gmres_fallbacks == 0 and st.fp64_fallbacks == 0
    assert abs(np.linalg.norm(b - G @ x) / np.linalg.norm(b) - st.last_rel_residual) <= 1e-13
    sim.close()
