"""Pivot blocks of two where the product of their entries leaves the format's
range although the entries do not (a state's unit is the user's)."""
import numpy as np
import pytest

from uqcreator_b200 import workloads as W
from uqcreator_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [4, 11], ids=["5_duals", "12_duals"])
@pytest.mark.parametrize("newton", ["reference", "guarded"])
def test_batched_newton(degree, newton):
    """Bounds, moments and tolerance times 2^512: every operation scales by a
    power of two, so the duals are the unscaled ones, bit for bit. (The norm of
    the gradient, a sum of squares, still fits: it starts below half a unit.)"""
    def solver(scale):
        toml = W.burgers1d(ncells=20, degree=degree, nquad=24, eps=1e-10 * scale, newton=newton)
        s = Solver(toml.replace("bounds = [2.5,12.5]", "bounds = [%r,%r]" % (2.5 * scale, 12.5 * scale)))
        s.set_option("closure_tiny", 0)
        return s

    s = solver(1.0)
    _, phi_wf, xi, _ = s.tables()
    r = np.random.default_rng(3)
    u = (7.5 + 0.2 * r.uniform(-1, 1, (33, 1)) + 0.2 * r.uniform(-1, 1, (33, 1)) * xi[:, 0])[:, None, :] @ phi_wf
    lam, status = s.closure_solve_host(np.zeros_like(u), u)
    assert not status.any()
    big, status = solver(2.0 ** 512).closure_solve_host(np.zeros_like(u), u * 2.0 ** 512)
    assert not status.any()
    np.testing.assert_array_equal(big, lam)
