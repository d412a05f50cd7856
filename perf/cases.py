"""Timing cases of the IPM time step and closure: the calls that a program using
this package makes, at the sizes of the repository's workloads.

A case is a dict of plain values:

  kind       what one pass is
               "steps"    a solver's initial state, then `steps` time steps
                          (Solver.init_state, Solver.step)
               "solve"    the same to the end time or step limit in one call,
                          then mean and variance (Solver.run, Solver.mean_var)
               "host"     one time step from host state to host state
                          (Solver.step_host), for a program that keeps the
                          moments and duals in its own memory
               "closure"  the dual Newton solve of a batch of cells in host
                          arrays (Solver.closure_solve_host), for a program that
                          only replaces its closure
  problem    "burgers" (1-D, one state), "sw" (1-D shallow water, two states,
             adaptive moment order), "euler" (2-D, four states, 2 or 3 uncertainties)
  cells, or nx and ny (2 nx ny triangles); degree, nquad per uncertainty;
  dim_xi; steps; precision ("fp64" or "mixed")

The seed moves the uncertain shock or interface and draws the mesh jitter (the
batch of states of a "closure" case). `exact` recomputes the outputs with plain
torch operations in 64 bits: its own tables, mesh, Newton solve and time loop.
"""
import functools
import math

import numpy as np
import torch

from uqcreator_b200 import workloads
from uqcreator_b200.solver import Settings, Solver

GAMMA, CFL, GRAV = 1.4, 0.5, 9.81
BB_LO, BB_HI = 2.5, 12.5


def listed():
    return [
        # a single cell's closure through the C ABI: what an adapter that calls
        # SolveClosure cell by cell pays, nothing but latency
        dict(name="closure_1_cell", kind="closure", problem="burgers", cells=1, degree=4, nquad=20, dim_xi=1, steps=0, precision="fp64"),
        # a batch of cells through the same call, 84 duals each: an adapter that
        # hands over a whole mesh's closure
        dict(name="closure_5k_euler", kind="closure", problem="euler", cells=5001, degree=5, nquad=10, dim_xi=2, steps=0, precision="fp64"),
        # the plain Burgers workload, whole solve: 500 cells, 5 moments, about
        # 460 steps of a few tens of microseconds (launches and latency)
        dict(name="solve_500_burgers", kind="solve", problem="burgers", cells=500, degree=4, nquad=20, dim_xi=1, steps=0, precision="fp64"),
        # the largest Burgers request of the serving stream, 10 moments
        dict(name="steps_20k_burgers", kind="steps", problem="burgers", cells=19997, degree=9, nquad=40, dim_xi=1, steps=64, precision="fp64"),
        # the smallest 2-D Euler request of the serving stream: 6 moments, 24 duals
        dict(name="steps_10k_euler", kind="steps", problem="euler", nx=89, ny=57, degree=2, nquad=4, dim_xi=2, steps=32, precision="fp64"),
        # adaptive shallow water, ordinary and large mesh: cells of 2-10 moments
        dict(name="steps_50k_sw", kind="steps", problem="sw", cells=49999, degree=9, nquad=30, dim_xi=1, steps=24, precision="fp64"),
        dict(name="steps_1m_sw", kind="steps", problem="sw", cells=1000000, degree=9, nquad=30, dim_xi=1, steps=12, precision="fp64"),
        # the flagship 2-D Euler mesh, both precisions (84 duals, 100 nodes)
        dict(name="steps_200k_euler", kind="steps", problem="euler", nx=400, ny=250, degree=5, nquad=10, dim_xi=2, steps=16, precision="fp64"),
        dict(name="steps_200k_euler_mixed", kind="steps", problem="euler", nx=400, ny=250, degree=5, nquad=10, dim_xi=2, steps=32,
             precision="mixed"),
        # the same step for a program that keeps its state in host memory
        dict(name="host_200k_euler_mixed", kind="host", problem="euler", nx=400, ny=250, degree=5, nquad=10, dim_xi=2, steps=3,
             precision="mixed"),
        # three uncertainties: 140 duals, 512 nodes, both precisions; the largest
        dict(name="steps_262k_euler3_mixed", kind="steps", problem="euler", nx=512, ny=256, degree=4, nquad=8, dim_xi=3, steps=8,
             precision="mixed"),
        dict(name="steps_262k_euler3", kind="steps", problem="euler", nx=512, ny=256, degree=4, nquad=8, dim_xi=3, steps=8, precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges (the serving stream's sizes where it has them)."""
    what = rng.choice(["closure", "burgers", "sw", "euler", "euler", "euler", "host", "euler3"])
    precision = rng.choice(["fp64", "mixed"])
    if what == "closure":
        if rng.random() < 0.5:
            deg = rng.randint(2, 9)
            return dict(kind="closure", problem="burgers", cells=_log_int(rng, 1, 20000), degree=deg, nquad=4 * deg + 4, dim_xi=1, steps=0,
                        precision="fp64")
        deg = rng.randint(2, 5)
        return dict(kind="closure", problem="euler", cells=_log_int(rng, 1, 6000), degree=deg, nquad=2 * deg, dim_xi=2, steps=0,
                    precision="fp64")
    if what == "burgers":
        deg = rng.randint(2, 9)
        return dict(kind=rng.choice(["steps", "solve"]), problem="burgers", cells=_log_int(rng, 200, 20000), degree=deg, nquad=4 * deg + 4,
                    dim_xi=1, steps=rng.randint(16, 200), precision="fp64")
    if what == "sw":
        return dict(kind="steps", problem="sw", cells=_log_int(rng, 1000, 1000000), degree=rng.randint(2, 9), nquad=rng.randint(20, 30),
                    dim_xi=1, steps=rng.randint(6, 24), precision="fp64")
    if what == "euler3":
        deg = rng.randint(2, 4)
        nx, ny = rng.randint(60, 250), rng.randint(40, 120)
        return dict(kind="steps", problem="euler", nx=nx, ny=ny, degree=deg, nquad=2 * deg, dim_xi=3, steps=rng.randint(4, 8), precision=precision)
    cells, deg = _log_int(rng, 10000, 200000), rng.randint(2, 5)
    nx = max(4, round(math.sqrt(cells / 2 * 1.6)))
    ny = max(4, cells // (2 * nx))
    if what == "host":
        return dict(kind="host", problem="euler", nx=nx, ny=ny, degree=deg, nquad=2 * deg, dim_xi=2, steps=rng.randint(2, 5),
                    precision=precision)
    return dict(kind="steps", problem="euler", nx=nx, ny=ny, degree=deg, nquad=2 * deg, dim_xi=2, steps=rng.randint(8, 24),
                precision=precision)


def _cells(case):
    return case["cells"] if "cells" in case else 2 * case["nx"] * case["ny"]


def _offset(seed):
    """The shock / interface offset of a seed, in [0.05, 0.3] as in the serving stream."""
    return 0.05 + 0.25 * np.random.default_rng(1000 + seed).random()


# ---------------------------------------------------------------- the framework's side


def _toml(case, seed):
    p, off = case["problem"], _offset(seed)
    steps = case["steps"] if case["kind"] == "solve" else 0
    if p == "burgers":
        tend = 10.0 if steps else 0.11
        return workloads.burgers1d(ncells=max(case["cells"], 3), degree=case["degree"], nquad=case["nquad"], x0=0.5 + off, tend=tend,
                                   steps=steps, precision=case["precision"])
    if p == "sw":
        kw = dict(ncells=case["cells"], max_degree=case["degree"], nquad=case["nquad"], tend=10.0, precision=case["precision"])
        return workloads.shallow_water1d(**kw).replace("ic = [0.5,", "ic = [%r," % (0.5 + off / 2))
    nx, ny = case.get("nx", 4), case.get("ny", 4)
    return workloads.euler2d(nx=nx, ny=ny, degree=case["degree"], nquad=case["nquad"], dim_xi=case["dim_xi"], tend=10.0, seed=seed % 1000,
                             xs=0.5 - off, steps=steps, precision=case["precision"])


class _DeviceArray:
    """The resident state for torch (no copy); a tensor made of it keeps this object, and with it the solver, alive."""

    def __init__(self, solver, ptr, shape):
        self.solver = solver
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=2)


def _batch(case, seed, phi, phi_wf, xi):
    """Duals and moments of a "closure" case: smooth uncertain states, one per
    cell, and the duals of their means (the rule of the initial state)."""
    r = np.random.default_rng(seed)
    n, d = case["cells"], xi.shape[1]
    if case["problem"] == "burgers":
        mid, amp = r.uniform(5.0, 10.0, (n, 1)), r.uniform(-2.0, 2.0, (n, 2))
        u = (mid + amp[:, :1] * xi[:, 0] + 0.2 * amp[:, 1:] * xi[:, 0] ** 2)[:, None, :]
        lam = np.zeros((n, 1, phi.shape[1]))
    else:
        a = r.uniform(-0.15, 0.15, (4, n, d)) @ xi.T
        rho = r.uniform(0.2, 1.2, (n, 1)) * (1 + a[0])
        p = r.uniform(0.2, 1.2, (n, 1)) * (1 + a[1])
        v1, v2 = r.uniform(-0.6, 0.6, (n, 1)) + a[2], r.uniform(-0.6, 0.6, (n, 1)) + a[3]
        u = np.stack([rho, rho * v1, rho * v2, p / (GAMMA - 1) + 0.5 * rho * (v1 ** 2 + v2 ** 2)], 1)
        lam = np.zeros((n, 4, phi.shape[1]))
    u = u @ phi_wf
    if case["problem"] != "burgers":
        lam[:, :, 0] = _euler_ds(torch.from_numpy(u[:, :, 0])).numpy()
    return np.ascontiguousarray(lam), np.ascontiguousarray(u)


def prepare(case, seed):
    s = Solver(Settings(_toml(case, seed)))
    if case["kind"] == "closure":
        phi, phi_wf, xi, _ = s.tables()
        lam, u = _batch(case, seed, phi, phi_wf, xi)
        return dict(case=case, solver=s, lam=lam, u=u)
    s.init_state()
    shape = (s.n_cells, s.n_states, s.n_total)
    if case["kind"] == "host":
        s.step(case["steps"] - 1)
        pinned = [torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy() for _ in range(4)]
        level = np.zeros(s.n_cells, dtype=np.uint32)
        s.download_state(out=(pinned[0], pinned[1], level))
        return dict(case=case, solver=s, u=pinned[0], lam=pinned[1], out=(pinned[2], pinned[3], level))
    views = [torch.as_tensor(_DeviceArray(s, p, shape), device="cuda") for p in s.device_state()]
    return dict(case=case, solver=s, views=views)


def run(state):
    case, s = state["case"], state["solver"]
    if case["kind"] == "closure":
        lam, status = s.closure_solve_host(state["lam"], state["u"])
        return dict(lam=lam, status=status)
    if case["kind"] == "host":
        u, lam, _, info = s.step_host(state["u"], state["lam"], out=state["out"])
        return dict(u=u, lam=lam, dt=info["dt"])
    s.init_state()
    if case["kind"] == "solve":
        info = s.run()
        return dict(u=state["views"][0], lam=state["views"][1], mean_var=s.mean_var(), t=info["t"])
    info = s.step(case["steps"])
    return dict(u=state["views"][0], lam=state["views"][1], t=info["t"], dt=info["dt"])


def work(case):
    """Bytes: per step the moments and duals once in and once out, and the
    geometry once. Flops: per cell and step the nodal duals and the projections
    of the ansatz and of the fluxes (2 n nQ each, n = duals per cell), the fluxes;
    and Newton (symmetric Hessian, Cholesky, trial gradient) for the eighth of the
    cells that the benchmark's steps find unconverged, two iterations each (all
    cells, four iterations, in a closure call)."""
    ns = dict(burgers=1, sw=2, euler=4)[case["problem"]]
    d, deg = case["dim_xi"], case["degree"]
    nt = math.comb(deg + d, d)
    if case["problem"] == "sw":
        nt = (nt + 2) / 2  # adaptive: 2 .. degree + 1 moments, about half in the mean
    n, nq, cells = ns * nt, case["nquad"] ** d, _cells(case)
    newton = nq * nt * (nt + 1) / 2 * ns * (ns + 1) + n ** 3 / 3 + 2 * n * n + 4 * nq * n
    if case["kind"] == "closure":
        return dict(bytes=cells * 8 * 3 * n, flops=cells * 4 * newton)
    faces, fl = (3, 90) if case["problem"] == "euler" else (2, 12)
    # a solve to the end time 0.11 takes dt = CFL dx / 12 steps
    steps = 1 if case["kind"] == "host" else case["steps"] or round(0.11 * 12 / CFL * case["cells"] / 3)
    step = cells * (6 * nq * n + faces / 2 * nq * fl) + cells / 8 * 2 * newton
    return dict(bytes=steps * cells * 8 * (4 * n + 5 * faces + 3), flops=steps * step)


# ---------------------------------------------------------------- 64-bit recomputation


def _tables(case, device):
    """Orthonormal Legendre basis of total degree <= degree (functions ordered by
    their degrees, first dimension fastest; in one dimension by degree), tensor
    Gauss nodes (first dimension fastest) and phi times weight / 2^d."""
    d, deg, nq = case["dim_xi"], case["degree"], case["nquad"]
    x, w = np.polynomial.legendre.leggauss(nq)
    idx = [i for i in (np.arange((deg + 1) ** d)[:, None] // (deg + 1) ** np.arange(d)) % (deg + 1) if i.sum() <= deg]
    k = (np.arange(nq ** d)[:, None] // nq ** np.arange(d)) % nq
    one = np.stack([np.polynomial.legendre.legval(x, np.eye(deg + 1)[m]) * math.sqrt(2 * m + 1) for m in range(deg + 1)], 1)
    phi = np.ones((nq ** d, len(idx)))
    for c, i in enumerate(idx):
        for l in range(d):
            phi[:, c] *= one[k[:, l], i[l]]
    wt = np.prod(w[k] / 2, axis=1)
    return [torch.from_numpy(np.ascontiguousarray(a)).to(device) for a in (phi, phi * wt[:, None], x[k], wt)]


def _line(case, device):
    n = case["cells"]
    a, b = (0.0, 3.0) if case["problem"] == "burgers" else (0.0, 1.0)
    x = a + np.arange(n + 1) * (b - a) / n
    j = np.arange(n)
    end = (j == 0) | (j == n - 1)
    nbr = np.stack([np.where(end, j, j - 1), np.where(end, j, j + 1)], 1)
    unit = np.tile(np.array([[-1.0, 0.0], [1.0, 0.0]]), (n, 1, 1))
    m = dict(center=np.stack([x[:-1], 0 * x[:-1]], 1), area=np.abs(np.diff(x)), frozen=end, nbr=nbr, unit=unit, length=np.ones((n, 2)))
    m["dx"] = m["area"]
    return {k: torch.from_numpy(np.ascontiguousarray(v)).to(device) for k, v in m.items()}


def _triangles(case, seed, device):
    m = _jittered_grid(case["nx"], case["ny"], seed % 1000)
    xy, tri, bnd = m
    p = xy[tri]
    n = len(tri)
    area = np.abs(p[:, 0, 0] * (p[:, 1, 1] - p[:, 2, 1]) + p[:, 1, 0] * (p[:, 2, 1] - p[:, 0, 1]) + p[:, 2, 0] * (p[:, 0, 1] - p[:, 1, 1])) / 2
    cen = p.mean(1)
    e = p[:, [1, 2, 0]] - p
    length = np.sqrt((e ** 2).sum(-1))
    nrm = np.stack([e[..., 1], -e[..., 0]], -1)
    nrm *= np.where((nrm * (cen[:, None] - p)).sum(-1, keepdims=True) > 0, -1.0, 1.0)
    unit = nrm / np.linalg.norm(nrm, axis=-1, keepdims=True)
    a, b = np.minimum(tri, tri[:, [1, 2, 0]]).astype(np.int64), np.maximum(tri, tri[:, [1, 2, 0]])
    key = (a * (len(xy) + 1) + b).reshape(-1)
    order = np.argsort(key, kind="stable")
    same = np.nonzero(key[order][1:] == key[order][:-1])[0]
    nbr = np.repeat(np.arange(n), 3)
    nbr[order[same]], nbr[order[same + 1]] = order[same + 1] // 3, order[same] // 3
    m = dict(center=cen, area=area, frozen=bnd[tri].sum(1) == 2, nbr=nbr.reshape(n, 3), unit=unit, length=length, dx=length.max(1) / area)
    return {k: torch.from_numpy(np.ascontiguousarray(v)).to(device) for k, v in m.items()}


def _jittered_grid(nx, ny, seed, jitter=0.2):
    """Nodes, triangles and boundary marks of the jittered grid: interior node
    `id` moves by jitter (2 r - 1) of a grid spacing, r the SplitMix64 stream of
    seed 2^32 + 2 id + c in 53 bits; every rectangle is cut in two."""
    i, j = np.arange((nx + 1) * (ny + 1)) % (nx + 1), np.arange((nx + 1) * (ny + 1)) // (nx + 1)
    bnd = (i == 0) | (i == nx) | (j == 0) | (j == ny)
    with np.errstate(over="ignore"):
        z = np.uint64(seed) * np.uint64(1 << 32) + np.arange(2 * len(i), dtype=np.uint64) + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    r = ((z ^ (z >> np.uint64(31))) >> np.uint64(11)).astype(np.float64).reshape(-1, 2) * 2.0 ** -53
    g = np.stack([i, j], 1).astype(np.float64)
    xy = np.where(bnd[:, None], g, g + jitter * (2.0 * r - 1.0)) / np.array([nx, ny], dtype=np.float64)
    ri, rj = np.arange(nx * ny) % nx, np.arange(nx * ny) // nx
    a = rj * (nx + 1) + ri
    b, c, d = a + 1, a + nx + 2, a + nx + 1
    flip = (((ri == 0) & (rj == ny - 1)) | ((ri == nx - 1) & (rj == 0)))[:, None]
    t0, t1 = np.where(flip, np.stack([a, b, d], 1), np.stack([a, b, c], 1)), np.where(flip, np.stack([b, c, d], 1), np.stack([a, c, d], 1))
    return xy, np.stack([t0, t1], 1).reshape(-1, 3), bnd


def _euler_ds(u):
    rho, m1, m2, e = u.unbind(1)
    k = m1 * m1 + m2 * m2
    p = e - k / (2 * rho)
    return torch.stack([(k - GAMMA * (2 * rho * e - k)) / (k - 2 * rho * e) - torch.log(rho ** -GAMMA * p), -2 * rho * m1 / (k - 2 * rho * e),
                        -2 * rho * m2 / (k - 2 * rho * e), -rho / p], 1)


def _ansatz(problem, L):
    """U(Lambda) and the blocks (a, b), a <= b, of its Jacobian at every node (L: cells x states x nodes)."""
    if problem == "burgers":
        s = torch.sigmoid(L[:, 0])
        return ((BB_LO + (BB_HI - BB_LO) * s)[:, None], {(0, 0): (BB_HI - BB_LO) * s * torch.sigmoid(-L[:, 0])})
    if problem == "sw":
        a, b = L.unbind(1)
        h = (a + b * b / 2) / GRAV
        return torch.stack([h, h * b], 1), {(0, 0): torch.full_like(a, 1 / GRAV), (0, 1): b / GRAV, (1, 1): (a + 1.5 * b * b) / GRAV}
    v1, v2, v3, v4 = L.unbind(1)
    A, k = 1 / (1 - GAMMA), v2 * v2 + v3 * v3
    rho = torch.exp(A * ((k - 2 * v1 * v4 + 2 * GAMMA * v4) / (2 * v4) + torch.log(-v4)))
    ux, uy, en = -v2 / v4, -v3 / v4, (k - 2 * v4) / (2 * v4 * v4)  # momentum and energy per mass
    U = torch.stack([rho, rho * ux, rho * uy, rho * en], 1)
    # d log rho / d Lambda; the Jacobian is the symmetric one of an entropy ansatz
    r1, r2, r3 = -A, A * v2 / v4, A * v3 / v4
    r4 = A * (1 / v4 - k / (2 * v4 * v4))
    du = {(0, 0): rho * r1, (0, 1): rho * r2, (0, 2): rho * r3, (0, 3): rho * r4}
    du[1, 1] = rho * (ux * r2 - 1 / v4)
    du[1, 2] = rho * ux * r3
    du[1, 3] = rho * (ux * r4 + v2 / (v4 * v4))
    du[2, 2] = rho * (uy * r3 - 1 / v4)
    du[2, 3] = rho * (uy * r4 + v3 / (v4 * v4))
    du[3, 3] = rho * (en * r4 - k / v4 ** 3 + 1 / (v4 * v4))
    return U, du


def _newton(problem, lam, u, phi, pwf, wt):
    """The duals of the moments u: damped Newton on every cell until the gradient stops falling."""
    S, T = lam.shape[1:]
    lam = lam.clone()

    def grad(x, v):
        return _ansatz(problem, x @ phi.T)[0] @ pwf - v

    g = grad(lam, u)
    tol = 1e-14 * (1 + u.flatten(1).norm(dim=1))
    todo = torch.nonzero(g.flatten(1).norm(dim=1) > tol)[:, 0]
    for _ in range(80):
        if not len(todo):
            break
        keep = []
        for c in todo.split(max(64, int(2e9 / (8 * T * (phi.shape[0] + S * S * T))))):
            x, v, gc = lam[c], u[c], g[c]
            _, du = _ansatz(problem, x @ phi.T)
            H = x.new_empty(len(c), S, T, S, T)
            for (a, b), y in du.items():
                blk = (phi.T * (y * wt)[:, None, :]) @ phi
                H[:, a, :, b, :] = blk
                H[:, b, :, a, :] = blk
            d = torch.linalg.solve(H.reshape(len(c), S * T, S * T), gc.reshape(len(c), -1, 1)).reshape(x.shape)
            old, step = gc.flatten(1).norm(dim=1), torch.ones(len(c), 1, 1, dtype=x.dtype, device=x.device)
            best = torch.zeros(len(c), dtype=torch.bool, device=x.device)
            for _ in range(50):
                xn = x - step * d
                gn = grad(xn, v)
                now = gn.flatten(1).norm(dim=1)
                good = ~best & torch.isfinite(now) & (now < old)
                lam[c[good]], g[c[good]] = xn[good], gn[good]
                best |= good
                # near rounding a full step that does not help is the end
                if bool((best | (old < 1e-11)).all()):
                    break
                step = torch.where(best[:, None, None], step, step / 2)
            keep.append(c[best & (g[c].flatten(1).norm(dim=1) > tol[c])])
        todo = torch.cat(keep)
    return lam, g


def _pressure(u):
    rho, m1, m2, e = u.unbind(1)
    ux, uy = m1 / rho, m2 / rho
    return ux, uy, (GAMMA - 1) * (e - 0.5 * rho * (ux * ux + uy * uy))


def _flux(problem, a, b, n, length):
    """Numerical flux through a face with unit normal n at every node (a, b: cells x states x nodes)."""
    n0, n1, ln = n[:, 0, None], n[:, 1, None], length[:, None]
    if problem == "burgers":
        beta = torch.maximum(a.abs(), b.abs())
        return 0.25 * (a * a + b * b) * n0[:, None] - 0.5 * beta * (b - a)
    if problem == "sw":
        fa, fb = (torch.stack([u[:, 1], u[:, 1] ** 2 / u[:, 0] + 0.5 * GRAV * u[:, 0] ** 2], 1) for u in (a, b))
        return 0.5 * (fa + fb) * n0[:, None] - 6 / CFL * (b - a)

    def normal(u):
        ux, uy, p = _pressure(u)
        vn = (ux * n0 + uy * n1) * ln
        return torch.stack([u[:, 0] * vn, u[:, 1] * vn + p * n0 * ln, u[:, 2] * vn + p * n1 * ln, (u[:, 3] + p) * vn], 1)

    (ua, va, pa), (ub, vb, pb) = _pressure(a), _pressure(b)
    lo = (n0 * ua + n1 * va - torch.sqrt(GAMMA * pa / a[:, 0]))[:, None]
    hi = (n0 * ub + n1 * vb + torch.sqrt(GAMMA * pb / b[:, 0]))[:, None]
    fa, fb = normal(a), normal(b)
    mid = (hi * fa - lo * fb + hi * lo * (b - a) * ln[:, None]) / (hi - lo)
    return torch.where(lo >= 0, fa, torch.where(hi <= 0, fb, mid))


def _initial(case, seed, mesh, xi):
    """Nodal initial states (cells x states x nodes) and the duals' first guess from their means."""
    x, off = mesh["center"][:, :1], _offset(seed)
    if case["problem"] == "burgers":
        x0 = 0.5 + off
        x1 = x0 + 0.1
        z = 0.2 * xi[None, :, 0]
        ramp = 12.0 + (3.0 - 12.0) * (x0 + z - x) / (x0 - x1)
        return torch.where(x < x0 + z, 12.0, torch.where(x < x1 + z, ramp, 3.0))[:, None]
    if case["problem"] == "sw":
        h = torch.where(x < 0.5 + off / 2, 1 + 0.2 * xi[None, :, 0], 0.5)
        return torch.stack([h, 0 * h], 1)
    left = x < 0.5 - off + 0.05 * xi[None, :, 0]
    rho = torch.where(left, 1 + 0.1 * xi[None, :, 1], 0.125)
    p = torch.where(left, 1 + 0.1 * xi[None, :, 2] if xi.shape[1] > 2 else torch.ones_like(rho), 0.1)
    return torch.stack([rho, 0 * rho, 0 * rho, p / (GAMMA - 1)], 1)


def _first_duals(problem, u):
    lam = torch.zeros_like(u)
    if problem == "sw":
        h, q = u[:, 0, 0], u[:, 1, 0]
        lam[:, 0, 0], lam[:, 1, 0] = GRAV * h - 0.5 * (q / h) ** 2, q / h
    if problem == "euler":
        lam[:, :, 0] = _euler_ds(u[:, :, 0])
    return lam


def _nodal(problem, lam, phi):
    return torch.cat([_ansatz(problem, x @ phi.T)[0] for x in lam.split(65536)])


def _advance(case, mesh, phi, pwf, wt, u, lam, level, t, t_end):
    """One time step; level: each cell's moment count (adaptive shallow water) or None."""
    p = case["problem"]
    if level is None:
        lam, _ = _newton(p, lam, u, phi, pwf, wt)
        uq = _nodal(p, lam, phi)
        uq_moments = torch.cat([x @ pwf for x in uq.split(65536)])
    else:
        new, uq, uq_moments = level.clone(), u.new_empty(*u.shape[:2], phi.shape[0]), torch.zeros_like(u)
        top = u.shape[2]
        for nt in range(2, top + 1):
            c = torch.nonzero(level == nt)[:, 0]
            if not len(c):
                continue
            x, _ = _newton(p, lam[c][:, :, :nt].contiguous(), u[c][:, :, :nt].contiguous(), phi[:, :nt].contiguous(),
                           pwf[:, :nt].contiguous(), wt)
            y = lam[c]
            y[:, :, :nt] = x
            lam[c] = y
            uq[c] = _nodal(p, x, phi[:, :nt])
            ind = u[c, 0, nt - 1].abs() + u[c, 0, nt - 2].abs()
            new[c] = torch.where((ind > 0.02) & (nt < top), nt + 1, torch.where((ind < 0.004) & (nt > 2), nt - 1, nt))
        level = new
        uq_moments = (uq @ pwf) * (torch.arange(top, device=u.device) < level[:, None])[:, None]
    dx = mesh["dx"]
    if p == "burgers":
        dt = float((CFL * dx / uq.abs().amax((1, 2))).min())
    elif p == "sw":
        dt = float(mesh["area"][0]) * CFL / 12
    else:
        dt = math.inf
        for q, h in zip(uq.split(65536), dx.split(65536)):
            ux, uy, pr = _pressure(q)
            a = torch.sqrt(GAMMA * pr / q[:, 0])
            dt = min(dt, float((CFL / (h * (torch.maximum(ux.abs(), uy.abs()) + a).amax(1))).min()))
    out = uq_moments.clone()
    cut = (lambda x, c: x) if level is None else (lambda x, c: x * (torch.arange(u.shape[2], device=u.device) < level[c, None])[:, None])
    for c in torch.nonzero(~mesh["frozen"])[:, 0].split(32768):
        total = 0
        for f in range(mesh["nbr"].shape[1]):
            total = total + _flux(p, uq[c], uq[mesh["nbr"][c, f]], mesh["unit"][c, f], mesh["length"][c, f])
        out[c] -= cut(total @ pwf, c) * (dt / mesh["area"][c])[:, None, None]
    return out, lam, level, t + dt, dt


@functools.lru_cache(maxsize=1)
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def exact(case, seed):
    dev, p = _device(), case["problem"]
    phi, pwf, xi, wt = _tables(case, dev)
    if case["kind"] == "closure":
        lam, u = _batch(case, seed, *(x.cpu().numpy() for x in (phi, pwf, xi)))
        lam, _ = _newton(p, torch.from_numpy(lam).to(dev), torch.from_numpy(u).to(dev), phi, pwf, wt)
        return dict(lam=lam, status=None)
    mesh = _triangles(case, seed, dev) if p == "euler" else _line(case, dev)
    u = torch.cat([_initial(case, seed, {"center": x}, xi) @ pwf for x in mesh["center"].split(65536)])
    lam = _first_duals(p, u)
    level = torch.full((len(u),), u.shape[2], device=dev) if p == "sw" else None
    t, dt, taken = 0.0, 0.0, 0
    t_end = 0.11 if case["kind"] == "solve" and not case["steps"] else math.inf
    while (t < t_end) if t_end < math.inf else (taken < case["steps"]):
        u, lam, level, t, dt = _advance(case, mesh, phi, pwf, wt, u, lam, level, t, t_end)
        taken += 1
    if case["kind"] == "host":
        return dict(u=u, lam=lam, dt=dt)
    if case["kind"] == "solve":
        uq = _nodal(p, lam, phi)
        mean = uq @ pwf[:, 0]
        var = ((uq - mean[:, :, None]) ** 2) @ pwf[:, 0]
        return dict(u=u, lam=lam, mean_var=torch.cat([mean, var], 1), t=t)
    # above its level a shallow-water cell's duals are what its last solve at a finer level left
    return dict(u=u, lam=None if p == "sw" else lam, t=t, dt=dt)
