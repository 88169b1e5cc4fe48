"""Performance cases of the boundary-element bubble simulation.

Each case is one call, or a few calls in sequence, that a user's program makes on a simulation it holds:
a velocity evaluation, RK4 or Euler steps (state in, steps, state out, as a driver with its own output
loop does), a batched sweep's steps, or a differentiated trajectory.  The sizes are those of the
repository's own workloads and tests: the two nu = 7 bubbles, the nu = 20 bubble in an oscillating
field, the 256-bubble sweep, the nu = 10 adjoint, the nu = 40 pair, and the small and medium meshes that
remeshing drivers work on.

  listed()           the fixed cases
  draw(rng)          one more case of the same ranges
  prepare(case, seed), run(state)   the inputs and simulation, and one pass
  work(case)         bytes and floating-point operations that a pass cannot do without
  exact(case, seed)  the pass's outputs from a plain FP64 torch restatement of the method
"""
from __future__ import annotations

import functools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bem-bubbles_b200"))

from bem_b200 import mesh  # noqa: E402
from bem_b200.adjoint import rk4_flow, volume  # noqa: E402
from bem_b200.batch import BubbleBatch  # noqa: E402
from bem_b200.sim import ColocSim, ColocSimPin  # noqa: E402

BATCH_DT = 2e-3


# ------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # one velocity field of a coarse bubble with the default solver: latency and launches only
        {"name": "velocity_162", "kind": "velocity", "nu": 4, "solver": "bicgstab", "mirror": False},
        # a bubble near a wall, adaptive steps, default solver: the wall driver on a remeshed-size surface
        {"name": "wall_rk4_812", "kind": "rk4", "nu": 9, "solver": "bicgstab", "mirror": True, "adaptive": True,
         "steps": 1, "dt": 0.02},
        # the two-bubble driver: nu = 7 each, dense LU, fixed steps
        {"name": "pair_lu_984", "kind": "rk4", "nu": 7, "nu2": 7, "solver": "lu", "mirror": False,
         "adaptive": False, "steps": 2, "dt": 1e-3},
        # a bubble whose contact line is pinned to the wall (an odd number of unknowns), dense LU
        {"name": "pinned_rk4_761", "kind": "pinned", "nu": 19, "solver": "lu", "steps": 1, "dt": 1e-3},
        # the oscillation driver's inner loop: Euler step, wall image, surface tension, default solver
        {"name": "euler_wall_1442", "kind": "euler", "nu": 12, "solver": "bicgstab", "mirror": True,
         "sigma": 0.02, "dt": 1e-3},
        # the bubble in an oscillating field, mixed precision, four steps between two outputs
        {"name": "oscillation_mixed_4002", "kind": "rk4", "nu": 20, "solver": "mixed", "mirror": False,
         "adaptive": False, "steps": 4, "dt": 5e-3},
        # the same bubble through the default FP64 solver
        {"name": "oscillation_fp64_4002", "kind": "rk4", "nu": 20, "solver": "bicgstab", "mirror": False,
         "adaptive": False, "steps": 1, "dt": 5e-3},
        # and one velocity field of it through the dense FP64 LU
        {"name": "velocity_lu_4002", "kind": "velocity", "nu": 20, "solver": "lu", "mirror": False},
        # a small parameter study: 24 uneven bubbles, two steps of the captured step graph
        {"name": "sweep_24", "kind": "sweep", "bubbles": 24, "nu_min": 4, "nu_max": 12, "mix": 1, "steps": 2},
        # the radius x pressure sweep: 256 uneven bubbles
        {"name": "sweep_256", "kind": "sweep", "bubbles": 256, "nu_min": 4, "nu_max": 16, "mix": 0, "steps": 1},
        # gradient of the volume through RK4 steps (forward with checkpoints, then backward)
        {"name": "adjoint_1002", "kind": "adjoint", "nu": 10, "steps": 4},
        # the large pair, mixed precision: one step of 32004 unknowns
        {"name": "pair_mixed_32004", "kind": "rk4", "nu": 40, "nu2": 40, "solver": "mixed", "mirror": False,
         "adaptive": False, "steps": 1, "dt": 1e-3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["velocity", "rk4", "rk4", "mixed", "pinned", "euler", "sweep", "adjoint"])
    if kind == "velocity":
        return {"kind": kind, "nu": _log_int(rng, 2, 24), "solver": rng.choice(["bicgstab", "bicgstab", "lu"]),
                "mirror": rng.random() < 0.4}
    if kind == "rk4":
        if rng.random() < 0.35:
            return {"kind": kind, "nu": rng.randint(3, 11), "nu2": rng.randint(3, 11),
                    "solver": rng.choice(["lu", "bicgstab"]), "mirror": False, "adaptive": rng.random() < 0.3,
                    "steps": rng.randint(1, 3), "dt": rng.uniform(5e-4, 2e-3)}
        adaptive = rng.random() < 0.5
        return {"kind": kind, "nu": _log_int(rng, 3, 22), "solver": "bicgstab", "mirror": rng.random() < 0.5,
                "adaptive": adaptive, "steps": rng.randint(1, 2),
                "dt": rng.uniform(0.005, 0.03) if adaptive else rng.uniform(1e-3, 5e-3)}
    if kind == "mixed":
        c = {"kind": "rk4", "nu": _log_int(rng, 5, 30), "solver": "mixed", "mirror": rng.random() < 0.25,
             "adaptive": rng.random() < 0.25, "steps": rng.randint(1, 5), "dt": rng.uniform(1e-3, 5e-3)}
        if rng.random() < 0.3:
            c |= {"nu": _log_int(rng, 4, 20), "nu2": _log_int(rng, 4, 20), "mirror": False}
        return c
    if kind == "pinned":
        return {"kind": kind, "nu": rng.randint(5, 26), "solver": "lu", "steps": rng.randint(1, 2),
                "dt": rng.uniform(2e-4, 1e-3)}
    if kind == "euler":
        return {"kind": kind, "nu": _log_int(rng, 4, 20), "solver": "bicgstab", "mirror": rng.random() < 0.7,
                "sigma": rng.uniform(0.005, 0.05), "dt": rng.uniform(5e-4, 2e-3)}
    if kind == "sweep":
        lo = rng.randint(3, 8)
        return {"kind": kind, "bubbles": _log_int(rng, 2, 96), "nu_min": lo, "nu_max": lo + rng.randint(0, 8),
                "mix": rng.randint(2, 10 ** 6), "steps": rng.randint(1, 3)}
    return {"kind": kind, "nu": rng.randint(4, 12), "steps": rng.randint(1, 6)}


# ------------------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _unit(nu):
    return mesh.icosphere(nu)


@functools.lru_cache(maxsize=None)
def _cap(nu):
    return mesh.wall_cap(nu)


def _surface_potential(d, rdot, r):
    """-R Rdot with a smooth low-order disturbance; d: unit directions."""
    c = r.uniform(-0.06, 0.06, 4)
    return lambda R: -R * rdot + c[0] * d[:, 0] + c[1] * d[:, 1] + c[2] * d[:, 2] + c[3] * d[:, 0] * d[:, 1]


def _bubble(nu, radius, center, noise, rdot, r):
    v, f = _unit(nu)
    scale = radius * (1.0 + noise * r.standard_normal(len(v)))
    return v * scale[:, None] + np.asarray(center)[None, :], f, _surface_potential(v, rdot, r)(radius)


def _sweep_nus(case):
    g = random.Random(case["mix"])
    return [g.randint(case["nu_min"], case["nu_max"]) for _ in range(case["bubbles"])]


def _inputs(case, seed):
    """Host arrays of a case: meshes, potential, physical constants."""
    r = np.random.RandomState(seed % (1 << 32))
    kind = case["kind"]
    phys = dict(p_inf=1.0, epsilon=1.0, sigma=0.0, gamma=1.4)
    field = None
    if kind == "pinned":
        v, f = _cap(case["nu"])
        scale = 1.0 + 0.02 * r.uniform(-1, 1)
        v = v * scale
        phi = 0.05 * r.uniform(-1, 1) + 0.03 * r.uniform(-1, 1) * v[:, 0]
        phys["epsilon"] = 1.4
        return dict(v=v, f=f, phi=phi, phys=phys, field=(-0.3, 0.7, r.uniform(0, 1), 0.2))
    if kind == "sweep":
        parts, phi = [], []
        for nu in _sweep_nus(case):
            R = math.exp(r.uniform(math.log(0.5), math.log(2.0)))
            parts.append(_bubble(nu, R, (1.5 + R, 0.0, 0.0), 0.0, 0.0, r))
            phi.append(parts[-1][2])
        n = len(parts)
        return dict(parts=[p[:2] for p in parts], phi=np.concatenate(phi), phys=phys,
                    amp=-r.uniform(0.1, 1.5, n), omega=2 * np.pi / r.uniform(2.0, 10.0, n))
    if kind == "adjoint":
        v, f, phi = _bubble(case["nu"], 1.0, (2.0, 0.0, 0.0), 0.0, r.uniform(-0.4, -0.2), r)
        return dict(v=v, f=f, phi=phi, phys=phys, field=None)
    if case.get("nu2"):  # vapour cavities of a pair (they would share one gas volume)
        a = _bubble(case["nu"], 1.0, (2.0, 0.0, 0.0), 0.0, r.uniform(-0.5, 0.5), r)
        b = _bubble(case["nu2"], 0.8, (4.6, 0.0, 0.0), 0.0, r.uniform(-0.5, 0.5), r)
        phys.update(epsilon=0.0, gamma=1.0)
        return dict(v=np.concatenate([a[0], b[0]]), f=np.concatenate([a[1], b[1] + len(a[0])]),
                    phi=np.concatenate([a[2], b[2]]), phys=phys, field=None, split=(len(a[0]), len(a[1])))
    # per-vertex radial disturbance of 1%, less where the edges are shorter than the nu = 20 mesh's
    noise = 0.01 * min(1.0, (20.0 / case["nu"]) ** 2)
    v, f, phi = _bubble(case["nu"], 1.0, (2.0, 0.0, 0.0), noise, r.uniform(-0.3, 0.3), r)
    phys["sigma"] = float(case.get("sigma", 0.0))
    return dict(v=v, f=f, phi=phi, phys=phys, field=(-0.8, 2 * np.pi / 5.0, r.uniform(0, 1)))


# ---------------------------------------------------------------------------------------------- the passes
def prepare(case, seed):
    c, d = case, _inputs(case, seed)
    s = {"case": c}
    if c["kind"] == "sweep":
        s["sim"] = BubbleBatch(d["parts"], **d["phys"])
        s["sim"].set_block_params(amp=d["amp"], omega=d["omega"])
        s["v"], s["phi"] = np.concatenate([v for v, _ in d["parts"]]), d["phi"]
    elif c["kind"] == "pinned":
        s["sim"] = ColocSimPin(d["v"], d["f"], pressurefield=d["field"], solver=c["solver"], phi_init=d["phi"], **d["phys"])
        s["v"], s["phi"] = s["sim"].get_vertices(), s["sim"].get_phi()
    elif c["kind"] == "adjoint":
        s["sim"] = ColocSim(d["v"], d["f"], solver="mixed", **d["phys"])
        s["x"] = torch.tensor(d["v"], dtype=torch.float64, device="cuda")
        s["p"] = torch.tensor(d["phi"], dtype=torch.float64, device="cuda")
        s["f"] = torch.tensor(d["f"], dtype=torch.int64, device="cuda")
    else:
        s["sim"] = ColocSim(d["v"], d["f"], pressurefield=d["field"], solver=c["solver"], mirror=c["mirror"], **d["phys"])
        s["v"], s["phi"] = d["v"], d["phi"]
    if "v" in s:
        s["v"], s["phi"], s["psi"] = np.ascontiguousarray(s["v"]), np.ascontiguousarray(s["phi"]), np.zeros(len(s["phi"]))
    return s


def run(s):
    c, sim = s["case"], s["sim"]
    if c["kind"] == "adjoint":
        x, p = s["x"].detach().requires_grad_(), s["p"].detach().requires_grad_()
        xk, pk = rk4_flow(sim, x, p, BATCH_DT, c["steps"])
        volume(xk, s["f"]).backward()
        return {"x": xk.detach(), "phi": pk.detach(), "grad_x": x.grad, "grad_phi": p.grad}
    if c["kind"] == "velocity":
        vel, psi = sim.position_t(s["phi"], verts=s["v"], return_psi=True)
        return {"vel": vel, "psi": psi}
    sim.set_state(s["v"], s["phi"], s["psi"], 0.0)
    if c["kind"] == "sweep":
        sim.evolve_graph(BATCH_DT, c["steps"])
    elif c["kind"] == "euler":
        sim.evolve_system(c["dt"], fixdt=True)
    elif c.get("adaptive"):
        for _ in range(c["steps"]):
            sim.evolve_system_RK4(c["dt"])
    else:
        sim.evolve_rk4_steps(c["dt"], c["steps"])
    x, phi, psi, t = sim.get_state()
    return {"x": x, "phi": phi, "psi": psi, "t": t}


def _counts(case):
    """[(vertices, triangles)] of the systems of a case."""
    if case["kind"] == "sweep":
        return [(10 * nu * nu + 2, 20 * nu * nu) for nu in _sweep_nus(case)]
    if case["kind"] == "pinned":
        return [(2 * case["nu"] ** 2 + 2 * case["nu"] + 1, 4 * case["nu"] ** 2)]
    nus = [case["nu"]] + ([case["nu2"]] if case.get("nu2") else [])
    return [(sum(10 * nu * nu + 2 for nu in nus), sum(20 * nu * nu for nu in nus))]


def work(case):
    """The 7-point rule over all regular (vertex, triangle) pairs (32 operations per kernel evaluation, 52
    with the wall image) and the solve: 2/3 N^3 for the dense LU, one product with the matrix for an
    iterative solver.  Backward of a step: its stages again, the transposed solve and the derivative of
    the assembly (counted as one more assembly).  Bytes: the state in and out."""
    image = case.get("mirror") or case["kind"] == "pinned"
    stages = {"velocity": 1, "euler": 1}.get(case["kind"], 4 * case.get("steps", 1))
    flops = bytes_ = 0.0
    for n, m in _counts(case):
        per = 7.0 * (n * m - 3 * m) * (52 if image else 32)
        per += 2.0 / 3.0 * n ** 3 if case.get("solver") == "lu" else 2.0 * n * n
        flops += per * stages * (3 if case["kind"] == "adjoint" else 1)
        bytes_ += 8.0 * (3 * n + 2 * n) * 2 + 12.0 * m
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------------ plain FP64 restatement of a pass
_S15 = math.sqrt(15.0)


@functools.lru_cache(maxsize=None)
def _triangle_rule():
    """Radon's seven-point rule of degree 5: barycentric weights of the corners (7, 3), weights (7,)."""
    a, b = (6 - _S15) / 21, (6 + _S15) / 21
    wa, wb = (155 - _S15) / 2400, (155 + _S15) / 2400
    pts, w = [[1 / 3, 1 / 3, 1 / 3]], [9 / 80]
    for t, wt in ((a, wa), (b, wb)):
        for k in range(3):
            p = [t, t, t]
            p[k] = 1 - 2 * t
            pts.append(p)
            w.append(wt)
    return np.array(pts), np.array(w)


def _corners(x, tri):
    return x[tri[:, 0]], x[tri[:, 1]], x[tri[:, 2]]


def _self_terms(x, tri):
    """Single-layer integrals over a triangle seen from each of its corners: (M, corner, column)."""
    t, w = np.polynomial.legendre.leggauss(7)
    th = torch.tensor((t + 1) * math.pi / 8, dtype=x.dtype, device=x.device)
    w = torch.tensor(w / 2, dtype=x.dtype, device=x.device)
    cs, sn = torch.cos(th), torch.sin(th)
    out = []
    for k in range(3):
        a, b, c = (x[tri[:, (k + s) % 3]] for s in range(3))
        ab, bc = b - a, c - b
        area = torch.linalg.cross(ab, bc).norm(dim=1)
        dist = (ab[:, None] * cs[:, None] + bc[:, None] * sn[:, None]).norm(dim=2)
        f = (math.pi / 8) * area[:, None] * w / (dist * cs * cs)
        loc = torch.stack([(f * cs).sum(1), (f * (cs - sn)).sum(1), (f * sn).sum(1)], 1)
        out.append(torch.stack([loc[:, (j - k) % 3] for j in range(3)], 1))
    return torch.stack(out, 1)


def _layers(xr, x, tri, image):
    """Regular rule for the rows xr: single- and double-layer integrals (R, M, 3) and, with the wall, those
    of the image."""
    lam, w = _triangle_rule()
    lam, w = torch.tensor(lam, dtype=x.dtype, device=x.device), torch.tensor(w, dtype=x.dtype, device=x.device)
    got = []
    for mirrored in ((False, True) if image else (False,)):
        y = x * torch.tensor([-1.0, 1.0, 1.0], dtype=x.dtype, device=x.device) if mirrored else x
        a, b, c = _corners(y, tri)
        n = torch.linalg.cross(b - a, c - b)
        area = n.norm(dim=1)
        n = n / area[:, None]
        if mirrored:
            n = -n  # the mirrored normal, not the normal of the mirrored corners
        q = lam[:, 0, None, None] * a + lam[:, 1, None, None] * b + lam[:, 2, None, None] * c  # (7, M, 3)
        dn = (a * n).sum(1)[None] - xr @ n.T
        g = h = None
        for k in range(7):
            inv = 1.0 / sum((q[k, :, e][None] - xr[:, e, None]) ** 2 for e in range(3)).sqrt()
            gk = (w[k] * inv)[..., None] * lam[k]
            hk = (-w[k] * dn * inv ** 3)[..., None] * lam[k]
            g, h = (gk, hk) if g is None else (g + gk, h + hk)
        got.append((g * area[:, None], h * area[:, None]))
    return got


def _system(x, tri, pot, image, pinned=0, psi=None):
    """G and b = H pot (after the 4 pi rule; with the pinned columns exchanged)."""
    n, m = len(x), len(tri)
    sing = _self_terms(x, tri)
    rows_g, rows_b = [], []
    step = n if x.requires_grad else max(1, min(n, int(6e6) // m))
    for r0 in range(0, n, step):
        r1 = min(n, r0 + step)
        terms = _layers(x[r0:r1], x, tri, image)
        own = (tri >= r0) & (tri < r1)  # (M, corner)
        t, k = own.nonzero(as_tuple=True)
        keep = torch.ones((r1 - r0, m, 1), dtype=x.dtype, device=x.device)
        keep[tri[t, k] - r0, t] = 0.0
        g, h = terms[0][0] * keep, terms[0][1] * keep
        if image:
            g, h = g + terms[1][0], h + terms[1][1]
        G = torch.zeros((r1 - r0, n), dtype=x.dtype, device=x.device)
        for j in range(3):
            G = G.index_add(1, tri[:, j], g[..., j])
            G = G.index_put((tri[t, k] - r0, tri[t, j]), sing[t, k, j], accumulate=True)
        if pinned:
            H = torch.zeros_like(G)
            for j in range(3):
                H = H.index_add(1, tri[:, j], h[..., j])
            i = torch.arange(r0, r1, device=x.device)
            H[i - r0, i] -= 4 * math.pi + H.sum(1)
            G, H = torch.cat([G[:, : n - pinned], -H[:, n - pinned:]], 1), torch.cat([H[:, : n - pinned], -G[:, n - pinned:]], 1)
            b = H @ torch.cat([pot[: n - pinned], psi[n - pinned:]])
        else:
            b = sum((h[..., j] * (pot[tri[:, j]][None] - pot[r0:r1, None])).sum(1) for j in range(3)) - 4 * math.pi * pot[r0:r1]
        rows_g.append(G)
        rows_b.append(b)
    if len(rows_g) == 1:
        return rows_g[0], rows_b[0]
    G = torch.empty((n, n), dtype=x.dtype, device=x.device)
    for r0 in range(0, n, step):
        G[r0:r0 + step] = rows_g.pop(0)
    return G, torch.cat(rows_b)


def _fan_mean(per_corner, tri, n):
    s = torch.zeros((n,) + per_corner.shape[1:], dtype=per_corner.dtype, device=per_corner.device)
    for k in range(3):
        s = s.index_add(0, tri[:, k], per_corner)
    c = torch.bincount(tri.reshape(-1), minlength=n).to(s.dtype)
    return s / (c if s.dim() == 1 else c[:, None])


def _vertex_normals(x, tri):
    acc = torch.zeros_like(x)
    for k in range(3):
        a, b, c = (x[tri[:, (k + s) % 3]] for s in range(3))
        u, v = b - a, c - a
        acc = acc.index_add(0, tri[:, k], torch.linalg.cross(u, v) / ((u * u).sum(1) * (v * v).sum(1))[:, None])
    return acc / acc.norm(dim=1, keepdim=True)


def _velocity(x, tri, pot, P, psi):
    """(velocity, solved unknowns, potential)."""
    n, pinned = len(x), P.get("pinned", 0)
    G, b = _system(x, tri, pot, P["image"], pinned, psi)
    sol = torch.linalg.solve(G, b)
    a, bb, c = _corners(x, tri)
    ab, bc = bb - a, c - bb
    nn = torch.linalg.cross(ab, bc)
    nrm = nn / nn.norm(dim=1, keepdim=True)
    dual = nn / (nn * nn).sum(1, keepdim=True)
    pa, pb, pc = (pot[tri[:, k]] for k in range(3))
    grad = torch.linalg.cross(dual, ab) * (pc - pb)[:, None] + torch.linalg.cross(dual, bc) * (pa - pb)[:, None]
    vel = _fan_mean(grad, tri, n) + sol[:, None] * _fan_mean(nrm, tri, n)
    if pinned:
        vn = _vertex_normals(x, tri)[n - pinned:]
        beta, ceq, cnl = 0.2, math.cos(130.0 / 180.0 * math.pi), 0.01
        cth = vn[:, 0]
        wall = torch.cat([torch.zeros_like(vn[:, :1]), vn[:, 1:] / vn[:, 1:].norm(dim=1, keepdim=True)], 1)
        drift = beta * (ceq - cth) + cnl * cth ** 3 / (cth ** 2 - 1)
        vel = torch.cat([vel[: n - pinned], wall * drift[:, None]])
        pot = torch.cat([pot[: n - pinned], sol[n - pinned:]])
    return vel, sol, pot


def _enclosed(x, tri):
    a, b, c = _corners(x, tri)
    return (torch.linalg.cross(a, b) * c).sum() / 6.0


def _bernoulli(x, vel, P, t):
    amp, omega, phase, kx = (tuple(P["field"]) + (0.0,))[:4] if P["field"] else (0.0, 0.0, 0.0, 0.0)
    gas = torch.cat([(P["eps"] * (P["V0"] / _enclosed(x, f)) ** P["gamma"]).expand(cnt) for f, cnt in P["parts"]])
    return 0.5 * (vel * vel).sum(1) + P["p_inf"] - gas + amp * torch.sin(kx * x[:, 0] + omega * t + phase)


def _stage(x, tri, pot, P, psi, t):
    vel, _, pot = _velocity(x, tri, pot, P, psi)
    return vel, _bernoulli(x, vel, P, t), pot


def _rk4(x, phi, psi, t, tri, P, dp, adaptive, stage=_stage):
    k1, q1, p1 = stage(x, tri, phi, P, psi, t)
    dt = float(dp / (q1.abs().max() + 3.0 * (k1 * k1).sum(1).max().sqrt())) if adaptive else dp
    k2, q2, _ = stage(x + 0.5 * dt * k1, tri, p1 + 0.5 * dt * q1, P, psi, t)
    k3, q3, _ = stage(x + 0.5 * dt * k2, tri, p1 + 0.5 * dt * q2, P, psi, t)
    k4, q4, _ = stage(x + dt * k3, tri, p1 + dt * q3, P, psi, t)
    avg = (k1 + 2 * k2 + 2 * k3 + k4) / 6
    x = x + dt * avg
    phi = p1 + (dt / 6) * (q1 + 2 * q2 + 2 * q3 + q4)
    return x, phi, (avg * _vertex_normals(x, tri)).sum(1), t + dt


def _wall_order(v, f, phi):
    """Wall vertices at the end of the list, in the order in which the simulation's constructor puts them."""
    v, phi, at, k, i = v.copy(), phi.copy(), np.arange(len(v)), len(v), 0
    while i < k:
        if abs(v[i, 0]) >= 1e-5:
            i += 1
            continue
        v[i, 0] = 0.0
        k -= 1
        v[[i, k]], phi[[i, k]], at[[i, k]] = v[[k, i]], phi[[k, i]], at[[k, i]]
    to = np.empty(len(v), dtype=np.int64)
    to[at] = np.arange(len(v))
    return v, to[f], phi, len(v) - k


def exact(case, seed):
    d, dev = _inputs(case, seed), "cuda" if torch.cuda.is_available() else "cpu"

    def put(a):
        return torch.tensor(np.ascontiguousarray(a), device=dev)

    ph, kind = d["phys"], case["kind"]
    P = dict(eps=ph["epsilon"], gamma=ph["gamma"], p_inf=ph["p_inf"], image=bool(case.get("mirror")), field=d.get("field"))
    if kind == "sweep":
        outs, at = [], 0
        for b, (v, f) in enumerate(d["parts"]):
            x, tri, phi = put(v), put(f), put(d["phi"][at:at + len(v)])
            at += len(v)
            Q = dict(P, V0=_enclosed(x, tri), parts=[(tri, len(v))], field=(d["amp"][b], d["omega"][b], 0.0))
            psi, t = None, 0.0
            for _ in range(case["steps"]):
                x, phi, psi, t = _rk4(x, phi, psi, t, tri, Q, BATCH_DT, False)
            outs.append((x, phi, psi))
        return {"x": torch.cat([o[0] for o in outs]), "phi": torch.cat([o[1] for o in outs]),
                "psi": torch.cat([o[2] for o in outs]), "t": BATCH_DT * case["steps"]}
    v, f, phi0 = d["v"], d["f"], d["phi"]
    if kind == "pinned":
        v, f, phi0, P["pinned"] = _wall_order(v, f, phi0)
        P["image"] = True
    x, tri, phi = put(v), put(f), put(phi0)
    P["V0"] = _enclosed(x, tri)
    nv, nf = d.get("split", (len(v), len(f)))
    P["parts"] = [(tri[:nf], nv)] + ([(tri[nf:], len(v) - nv)] if nf < len(f) else [])
    if kind == "velocity":
        vel, sol, _ = _velocity(x, tri, phi, P, None)
        return {"vel": vel, "psi": sol}
    if kind == "euler":  # the curvature's pivoted least squares is not restated: phi has no value here
        vel, _, _ = _velocity(x, tri, phi, P, None)
        return {"x": x + case["dt"] * vel, "phi": None, "psi": torch.zeros_like(phi), "t": case["dt"]}
    if kind == "adjoint":
        from torch.utils.checkpoint import checkpoint

        x0, p0 = x.clone().requires_grad_(), phi.clone().requires_grad_()

        def stage(xs, tri, ps, P, psi, t):
            return checkpoint(lambda a, b: _stage(a, tri, b, P, None, t), xs, ps, use_reentrant=False)

        xk, pk, psi, t = x0, p0, None, 0.0
        for _ in range(case["steps"]):
            xk, pk, psi, t = _rk4(xk, pk, psi, t, tri, P, BATCH_DT, False, stage)
        _enclosed(xk, tri).backward()
        return {"x": xk.detach(), "phi": pk.detach(), "grad_x": x0.grad, "grad_phi": p0.grad}
    psi, t = torch.zeros_like(phi), 0.0
    for _ in range(case["steps"]):
        x, phi, psi, t = _rk4(x, phi, psi, t, tri, P, case["dt"], case.get("adaptive", False))
    return {"x": x, "phi": phi, "psi": psi, "t": t}
