"""Cells whose Hessian is not positive definite, found at a diagonal tile after
the first, among cells that converge: the warps of a cell leave the
factorisation together, and the others' results do not change."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from uqcreator_b200 import workloads as W
from uqcreator_b200.solver import Solver

pytestmark = pytest.mark.gpu

NOT_PD = 3    # UQC_CELL_NOT_PD


def _batch(toml, n):
    """n cells of the initial state, every third with duals whose Hessian fails
    after the first basis functions of the first state: a negative depth
    (shallow water; the second state's block is negative) or an overflowing
    derivative of the momentum (Euler)."""
    o = Oracle(toml, W.mesh_for(toml))
    o.init_state()
    u, lam, _ = o.get_state()
    # away from the uncertain interface, where Newton converges from the first guess
    pick = np.r_[np.arange(n // 2), np.arange(len(u) - n + n // 2, len(u))]
    u, lam = np.ascontiguousarray(u[pick]), np.ascontiguousarray(lam[pick])
    bad = np.arange(n) % 3 == 1
    lam[bad] = 0.0
    if lam.shape[1] == 2:
        lam[bad, 0, 0] = -5.0
    else:
        lam[bad, 3, 0] = -1e-160
        lam[bad, 0, 0] = 1.4 + np.log(1e-160)
    return o, u, lam, bad


CASES = {
    "sw_24": W.shallow_water1d(ncells=200, max_degree=11, nquad=24),    # 78 basis pairs
    "sw_30": W.shallow_water1d(ncells=200, max_degree=14, nquad=30),
    "euler_60": W.euler2d(nx=40, ny=4, degree=4, nquad=8),
    "euler_84": W.euler2d(nx=40, ny=4),
    "euler_140": W.euler2d(nx=40, ny=4, degree=4, nquad=6, dim_xi=3),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_statuses_and_neighbours(name):
    o, u, lam, bad = _batch(CASES[name], 46)
    _, expect, _ = o.solve_closure(lam, u)
    np.testing.assert_array_equal(expect, np.where(bad, NOT_PD, 0))
    s = Solver(CASES[name])
    got, status = s.closure_solve_host(lam, u)
    np.testing.assert_array_equal(status, expect)
    np.testing.assert_array_equal(got[bad], lam[bad])
    alone, status = s.closure_solve_host(lam[~bad], u[~bad])
    assert not status.any()
    np.testing.assert_array_equal(got[~bad], alone)


@pytest.mark.parametrize("newton,group", [("reference", 256), ("guarded", 256), ("safe", 64), ("safe", 256)])
@pytest.mark.parametrize("name", ["sw_24", "euler_84"])
def test_general_kernel(name, newton, group):
    """The same through the general kernel's Cholesky, two and eight warps a cell."""
    toml = CASES[name]
    toml = toml.replace('newton = "guarded"', 'newton = "reference"').replace('newton = "reference"', f'newton = "{newton}"')
    o, u, lam, bad = _batch(toml, 46)
    _, expect, _ = o.solve_closure(lam, u)
    np.testing.assert_array_equal(expect, np.where(bad, NOT_PD, 0))
    s = Solver(toml)
    s.set_option("closure_group", group)
    got, status = s.closure_solve_host(lam, u)
    np.testing.assert_array_equal(status, expect)
    np.testing.assert_array_equal(got[bad], lam[bad])
    alone, status = s.closure_solve_host(lam[~bad], u[~bad])
    assert not status.any()
    np.testing.assert_array_equal(got[~bad], alone)
