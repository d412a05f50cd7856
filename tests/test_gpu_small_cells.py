"""The check and update kernels of cells with few moments (several lanes per
cell; instances of 6, 10 and 16 moments) and the 2-D Euler update on the tensor
cores: cell counts that leave a warp partly empty, node counts that leave lanes
idle, with and without the next step's test, against the FP64 oracle."""
import functools

import numpy as np
import pytest

from oracle.oracle import Oracle
from uqcreator_b200 import workloads as W
from uqcreator_b200.solver import Solver

pytestmark = pytest.mark.gpu

CASES = {
    "burgers_3_cells": W.burgers1d(ncells=3, degree=4, nquad=20, tend=10.0),
    "burgers_2_moments": W.burgers1d(ncells=37, degree=1, nquad=3, tend=10.0),
    "burgers_6_moments": W.burgers1d(ncells=65, degree=5, nquad=17, tend=10.0),
    "burgers_7_moments": W.burgers1d(ncells=41, degree=6, nquad=9, tend=10.0),
    "burgers_16_moments": W.burgers1d(ncells=43, degree=15, nquad=33, tend=10.0),
    "burgers_17_moments": W.burgers1d(ncells=43, degree=16, nquad=35, tend=10.0),    # the warp-per-cell kernels
    "sw_levels": W.shallow_water1d(ncells=131, max_degree=9, nquad=30, tend=10.0),
    "sw_16_moments": W.shallow_water1d(ncells=70, max_degree=15, nquad=32, tend=10.0),
    "sw_many_cells": W.shallow_water1d(ncells=250001, max_degree=2, nquad=5, tend=10.0),    # the next cell prefetched
    "euler_3_moments": W.euler2d(nx=7, ny=3, degree=1, nquad=3, tend=10.0),
    "euler_6_moments": W.euler2d(nx=16, ny=5, degree=2, nquad=5, tend=10.0),
    # k_update_mma: two cells a warp (odd counts of cells per warp and mesh), its three
    # widths, node counts that are not multiples of 4, the table in chunks
    "euler_10_moments": W.euler2d(nx=9, ny=5, degree=3, nquad=5, tend=10.0),
    "euler_15_moments": W.euler2d(nx=11, ny=3, degree=4, nquad=7, tend=10.0),
    "euler_28_moments": W.euler2d(nx=7, ny=4, degree=6, nquad=9, tend=10.0),
    "euler_45_moments": W.euler2d(nx=6, ny=3, degree=8, nquad=10, tend=10.0),
    "euler_35_moments_chunks": W.euler2d(nx=6, ny=4, degree=4, nquad=7, dim_xi=3, tend=10.0),
}


@pytest.mark.parametrize("update_test", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_steps_match_oracle(name, update_test):
    """Moments within 1e-9 of their largest, equal levels, dt, residual and failed
    cells. (Not the relative error of E and Var: three cells keep a state
    without variance, whose relative error compares rounding with rounding.)"""
    toml = CASES[name]
    s, o = Solver(toml), Oracle(toml, W.mesh_for(toml))
    s.set_option("update_test", update_test)
    s.init_state()
    o.init_state()
    a, b = s.step(9), o.step(9)
    assert a["steps"] == 9 and a["failed_cells"] == b["failures"]
    assert a["dt"] == pytest.approx(b["dt"], rel=1e-12) and a["residual"] == pytest.approx(b["residual"], rel=1e-9, abs=1e-15)
    us, _, vs = s.download_state()
    uo, _, vo = o.get_state()
    np.testing.assert_array_equal(vs, vo)
    np.testing.assert_allclose(us, uo, rtol=0, atol=1e-9 * np.abs(uo).max())


def _levels(toml, degrees, nquad):
    top = degrees[-1]
    toml = toml.replace(f'[["totalDegree"],[{top}]]', f'[["totalDegree"],{degrees}]')
    return toml.replace(f'[["tensorizedGrid"],[{nquad}]]', f'[["tensorizedGrid"],{[nquad] * len(degrees)}]')


# meshes that a warp per cell covers in several rounds, where the lanes take more moments
# and nodes than on the meshes above; and the other side of those rules
LARGE = {
    "burgers_16_moments": W.burgers1d(ncells=10007, degree=15, nquad=33, tend=10.0),
    "burgers_10_moments_warps": W.burgers1d(ncells=61, degree=9, nquad=70, tend=10.0),
    "sw_16_moments": W.shallow_water1d(ncells=5003, max_degree=15, nquad=32, tend=10.0),
    "sw_10_moments_warps": W.shallow_water1d(ncells=77, max_degree=9, nquad=80, tend=10.0),
    "euler_3_moments": W.euler2d(nx=41, ny=31, degree=1, nquad=3, tend=10.0),
    "euler_3_moments_4_nodes": W.euler2d(nx=7, ny=5, degree=1, nquad=2, tend=10.0),
    "euler_6_moments": W.euler2d(nx=41, ny=31, degree=2, nquad=4, tend=10.0),
    "euler_levels": _levels(W.euler2d(nx=41, ny=31, degree=2, nquad=4, tend=10.0), [1, 2], 4),
    # two cells a warp: beyond a CTA an SM, with 25 nodes of 6 moments, and 100 (k_update in one round)
    "euler_6_moments_25_nodes": W.euler2d(nx=41, ny=31, degree=2, nquad=5, tend=10.0),
    "euler_6_moments_100_nodes": W.euler2d(nx=35, ny=20, degree=2, nquad=10, tend=10.0),
    "euler_15_moments": W.euler2d(nx=35, ny=20, degree=4, nquad=7, tend=10.0),
    "euler_28_moments": W.euler2d(nx=31, ny=20, degree=27, nquad=30, dim_xi=1, tend=10.0),
    "euler_41_moments": W.euler2d(nx=31, ny=20, degree=40, nquad=43, dim_xi=1, tend=10.0),
    "euler_25_moments_chunks": W.euler2d(nx=31, ny=20, degree=24, nquad=203, dim_xi=1, tend=10.0),
}


@functools.lru_cache(maxsize=1)
def _four_steps(name):
    o = Oracle(LARGE[name], W.mesh_for(LARGE[name]))
    o.init_state()
    return o.step(4), o.get_state()


@pytest.mark.parametrize("name,update_test", [(n, t) for n in sorted(LARGE) for t in (0, 1)])
def test_steps_match_oracle_by_rounds(name, update_test):
    """The same comparison (fewer steps: the initial closure counts most)."""
    b, (uo, _, vo) = _four_steps(name)
    s = Solver(LARGE[name])
    s.set_option("update_test", update_test)
    s.init_state()
    a = s.step(4)
    assert a["steps"] == 4 and a["failed_cells"] == b["failures"]
    assert a["dt"] == pytest.approx(b["dt"], rel=1e-12) and a["residual"] == pytest.approx(b["residual"], rel=1e-9, abs=1e-15)
    us, _, vs = s.download_state()
    np.testing.assert_array_equal(vs, vo)
    np.testing.assert_allclose(us, uo, rtol=0, atol=1e-9 * np.abs(uo).max())
