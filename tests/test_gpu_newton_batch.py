"""k_newton, the FP64 closure whose cells iterate together: every launch shape and the remainders of its tiles (basis pairs in eights, duals in
eights, nodes in fours), against the FP64 oracle."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from uqcreator_b200 import workloads as W
from uqcreator_b200.solver import Solver

pytestmark = pytest.mark.gpu

EPS = 1e-10
# (degree, nodes per dimension, uncertainties): duals, basis pairs, nodes
SHAPES = [
    (1, 2, 2),    # 12 duals, 6 pairs, 4 nodes
    (1, 20, 2),   # 400 nodes for 12 duals
    (2, 3, 2),    # 24 duals, 9 nodes (not a multiple of 4)
    (3, 5, 2),    # 40 duals, 55 pairs, 25 nodes
    (4, 7, 2),    # 60 duals, 120 pairs (15 tiles exactly), 49 nodes
    (5, 10, 2),   # 84 duals
    (6, 9, 2),    # 112 duals, 406 pairs
    (7, 8, 2),    # 144 duals, 666 pairs: more row tiles than the largest shape holds
    (2, 3, 3),    # 40 duals, 27 nodes
    (4, 5, 3),    # 140 duals, 125 nodes (basis table in chunks)
]


def _oracle(toml):
    return Oracle(toml, W.mesh_for(toml))


def _residual(o, lam, u):
    """||g|| per cell at the duals lam (closure.cpp:234-253) from the oracle's tables and ansatz."""
    phi, phi_wf = o.tables()[:2]
    out = []
    for x, v in zip(lam, u):
        uk = np.stack([o.ansatz(x @ phi[k])[0] for k in range(phi.shape[0])], 1)
        out.append(np.linalg.norm(uk @ phi_wf - v))
    return np.array(out)


@pytest.mark.parametrize("degree,nquad,dim_xi", SHAPES)
@pytest.mark.parametrize("n", [1, 37])
def test_closure_of_a_batch(degree, nquad, dim_xi, n):
    """Cold closure of n cells (fewer than, and not a multiple of, a CTA's):
    same statuses as the oracle, and every solved cell meets the convergence
    test ||g|| < eps (plus the rounding of its own evaluation, nQ ulps of the
    moments' size)."""
    toml = W.euler2d(nx=12, ny=4, degree=degree, nquad=nquad, dim_xi=dim_xi, eps=EPS)
    o, s = _oracle(toml), Solver(toml)
    o.init_state()
    u, lam0, _ = o.get_state()
    pick = np.linspace(0, len(u) - 1, n).astype(int)
    u, lam0 = np.ascontiguousarray(u[pick]), np.ascontiguousarray(lam0[pick])
    lam, status = s.closure_solve_host(lam0, u)
    expect, expect_status = o.solve_closure(lam0.copy(), u)[:2]
    np.testing.assert_array_equal(status, expect_status)
    ok = status == 0
    rounding = 8 * nquad ** dim_xi * np.finfo(float).eps * np.linalg.norm(u.reshape(n, -1), axis=1)
    assert np.all(_residual(o, lam[ok], u[ok]) < EPS + rounding[ok])


@pytest.mark.parametrize("toml", [
    W.burgers1d(ncells=90, degree=6, nquad=9, eps=EPS),      # 7 duals
    W.burgers1d(ncells=90, degree=9, nquad=40, eps=EPS),     # 55 pairs, 7 row tiles
    W.burgers1d(ncells=90, degree=10, nquad=21, eps=EPS),    # 66 pairs: the second shape
    W.burgers1d(ncells=90, degree=14, nquad=30, eps=EPS),    # 120 pairs, its largest
    W.shallow_water1d(ncells=90, max_degree=3, nquad=7, eps=EPS),
    W.shallow_water1d(ncells=90, max_degree=9, nquad=30, eps=EPS),
], ids=["burgers_7", "burgers_10", "burgers_11", "burgers_15", "sw_8", "sw_20"])
@pytest.mark.parametrize("tiny", [-1, 0])
def test_closure_of_small_systems(toml, tiny):
    """One and two states, odd numbers of blocks: statuses and the convergence
    test as above, with different moment counts per cell where there are levels;
    up to 10 duals with the kernel of tiny systems and without it."""
    o, s = Oracle(toml), Solver(toml)
    s.set_option("closure_tiny", tiny)
    o.init_state()
    u, lam0, _ = o.get_state()
    nt = np.array(s.n_total_levels, dtype=np.uint32)[np.arange(len(u)) % s.n_levels]
    for j, t in enumerate(nt):
        u[j, :, t:] = 0.0
    lam, status = s.closure_solve_host(lam0, u, nt)
    _, expect_status = o.solve_closure(lam0.copy(), u, nt)[:2]
    np.testing.assert_array_equal(status, expect_status)
    phi, phi_wf = o.tables()[:2]
    for j in np.nonzero(status == 0)[0]:
        t = nt[j]
        uk = np.stack([o.ansatz(lam[j, :, :t] @ phi[k, :t])[0] for k in range(phi.shape[0])], 1)
        rounding = 8 * phi.shape[0] * np.finfo(float).eps * np.linalg.norm(u[j])
        assert np.linalg.norm(uk @ phi_wf[:, :t] - u[j, :, :t]) < EPS + rounding
    assert np.count_nonzero(status == 0) > len(u) // 2


@pytest.mark.parametrize("degree,nquad,dim_xi", [(1, 2, 2), (3, 5, 2), (4, 7, 2), (4, 5, 3)])
def test_steps_match_oracle(degree, nquad, dim_xi):
    """The fused epilogue: time steps against the oracle (E and Var of each state within 1e-10, relative L1)."""
    toml = W.euler2d(nx=16, ny=4, degree=degree, nquad=nquad, dim_xi=dim_xi, eps=EPS)
    o, s = _oracle(toml), Solver(toml)
    o.init_state()
    s.init_state()
    o.step(4)
    s.step(4)
    a, b = o.mean_var(), s.mean_var()
    scale = np.abs(a).sum(0)
    big = scale > 1e-8 * scale.max()
    assert np.all((np.abs(a - b).sum(0) / scale)[big] <= 1e-10)


def test_cells_of_different_levels():
    """Moment counts per cell (the scatter by level): each cell as if solved alone."""
    toml = W.euler2d(nx=12, ny=4, degree=3, nquad=6, eps=EPS).replace("[[\"totalDegree\"],[3]]", "[[\"totalDegree\"],[1,2,3]]")
    toml = toml.replace("[[\"tensorizedGrid\"],[6]]", "[[\"tensorizedGrid\"],[6,6,6]]")
    o, s = _oracle(toml), Solver(toml)
    assert s.n_total_levels == [3, 6, 10]
    o.init_state()
    u, lam0, _ = o.get_state()
    nt = np.array([3, 6, 10], dtype=np.uint32)[np.arange(len(u)) % 3]
    for j, t in enumerate(nt):
        u[j, :, t:] = 0.0
    lam, status = s.closure_solve_host(lam0, u, nt)
    expect, expect_status = o.solve_closure(lam0.copy(), u, nt)[:2]
    np.testing.assert_array_equal(status, expect_status)
    for j, t in enumerate(nt):
        np.testing.assert_array_equal(lam[j, :, t:], lam0[j, :, t:])
        if j % 7 == 0:
            alone, _ = s.closure_solve_host(lam0[j:j + 1], u[j:j + 1], nt[j:j + 1])
            np.testing.assert_array_equal(alone[0], lam[j])
    # the solved part meets the convergence test on its own moments
    phi, phi_wf = o.tables()[:2]
    for j in np.nonzero(status == 0)[0]:
        t = nt[j]
        uk = np.stack([o.ansatz(lam[j, :, :t] @ phi[k, :t])[0] for k in range(phi.shape[0])], 1)
        assert np.linalg.norm(uk @ phi_wf[:, :t] - u[j, :, :t]) < EPS + 8 * 36 * np.finfo(float).eps * np.linalg.norm(u[j])
