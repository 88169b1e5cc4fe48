"""The resident BiCGSTAB (one cooperative launch) at the edges of its size classes.

solve_system takes any dense matrix, so the sizes are picked freely: fewer rows than a CTA holds, one more
than a multiple of the rows per CTA, the steps of the elements per thread (512, 1024, 1536, 2048, 4096, 6144) and of
the entries kept in registers (columns beyond them sit in shared memory); above 2048 the matrix is streamed
(odd sizes from a copy with an even stride), above 6144 the older persistent form takes over.  BiCGSTAB stops at a recursive
residual of DBL_EPSILON; with a matrix of condition about 2 the solution is then within a few hundred
roundings of LAPACK's (tolerance 1e-12).
"""
import numpy as np
import pytest

from bem_b200 import _lib as L
from bem_b200.sim import ColocSim

pytestmark = pytest.mark.gpu


def uv_sphere(n):
    """A closed triangulated sphere of exactly n >= 5 vertices: two poles and rings of equal length, or one
    ring (n - 2 a prime)."""
    m = n - 2
    ring = next((r for r in range(3, m + 1) if m % r == 0 and r >= m // r), m)
    rings = m // ring
    th = np.pi * (np.arange(rings) + 1) / (rings + 1)
    ph = 2 * np.pi * np.arange(ring) / ring
    v = [[0, 0, 1.0]]
    v += [[np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t)] for t in th for p in ph]
    v.append([0, 0, -1.0])
    f = []
    for k in range(ring):
        q = (k + 1) % ring
        f.append([0, 1 + k, 1 + q])
        f.append([n - 1, 1 + (rings - 1) * ring + q, 1 + (rings - 1) * ring + k])
        for r in range(rings - 1):
            a, b = 1 + r * ring + k, 1 + r * ring + q
            f += [[a, a + ring, b], [b, a + ring, b + ring]]
    return np.array(v) + np.array([2.0, 0, 0]), np.array(f)


def system(n, seed):
    r = np.random.default_rng(seed)
    return np.asfortranarray(np.eye(n) + 0.3 * r.standard_normal((n, n)) / np.sqrt(n)), r.standard_normal(n)


@pytest.mark.parametrize("n", [5, 15, 16, 17, 257, 512, 513, 897, 1024, 1025, 1536, 1537, 2047, 2048, 2049, 2050, 3333, 4096, 4097, 6143, 6144, 6145])
def test_matches_lapack_at_size_edges(n):
    v, f = uv_sphere(n)
    assert len(v) == n
    sim = ColocSim(v, f, solver="bicgstab")
    for seed in (n, n + 1):
        G, b = system(n, seed)
        x = sim.solve_system(G, b)
        ref = np.linalg.solve(G, b)
        assert np.linalg.norm(x - ref) <= 1e-12 * np.linalg.norm(ref)
    assert np.array_equal(sim.solve_system(G, b), x)  # fixed summation order
    assert sim.stats().wait_expired == 0
    assert np.array_equal(sim.solve_system(G, np.zeros(n)), np.zeros(n))
    sim.close()


@pytest.mark.parametrize("n", [42, 700, 2345])
def test_iterates_match_the_multikernel_form(n):
    # the first iterates, cut off by max_iters, are those of the separate kernels up to rounding (the
    # recurrence amplifies it little in three iterations: 1e-12)
    v, f = uv_sphere(n)
    G, b = system(n, 3)
    for iters in (1, 2, 3):
        got = []
        for flags in (0, L.FLAG_BICGSTAB_MULTIKERNEL):
            sim = ColocSim(v, f, solver="bicgstab")
            sim._update(max_iters=iters, flags=flags)
            got.append(sim.solve_system(G, b))
            assert sim.stats().last_iters == iters
            sim.close()
        assert np.linalg.norm(got[0] - got[1]) <= 1e-12 * np.linalg.norm(got[1])


def test_restarts_on_a_stagnating_system():
    # condition 1e5: the recursive residual stagnates above the tolerance, the shadow residual loses the
    # residual and the iteration restarts; the residual still falls to 1e-9 of b
    n = 300
    r = np.random.default_rng(5)
    q, _ = np.linalg.qr(r.standard_normal((n, n)))
    G = np.asfortranarray(q @ np.diag(np.logspace(0, -5, n)) @ q.T)
    b = G @ r.standard_normal(n)
    v, f = uv_sphere(n)
    sim = ColocSim(v, f, solver="bicgstab")
    sim._update(max_iters=8000)
    x = sim.solve_system(G, b)
    assert np.linalg.norm(G @ x - b) <= 1e-9 * np.linalg.norm(b)
    assert sim.stats().wait_expired == 0
    sim.close()
