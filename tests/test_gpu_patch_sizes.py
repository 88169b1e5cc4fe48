"""The triangle patches of small systems, whose size follows the number of tiles, against the oracle.

From five triangles per patch (the smallest systems) over every size between to the largest of 32, without and
with singular pairs in a tile's rows (more than 256 rows), with the wall image and without.  Tolerances as in
test_gpu_assembly_g: G entry-wise 1e-13 relative to max|G|, b 1e-12 relative to max|b|.
"""
import numpy as np
import pytest

from bem_b200 import mesh

from test_gpu_assembly_g import check_against_oracle
from test_gpu_bicgstab import uv_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mirror", [False, True])
@pytest.mark.parametrize("n", [5, 42, 162, 257, 362, 642, 1002, 1442])
def test_small_systems(n, mirror):
    nu = {42: 2, 162: 4, 362: 6, 642: 8, 1002: 10, 1442: 12}.get(n)
    v, f = mesh.bubble(nu, 1.0, (2.0, 0.0, 0.0)) if nu else uv_sphere(n)
    check_against_oracle(v, f, 0.1 * np.sin(2 * v[:, 2]) + 0.05 * v[:, 1], mirror)
