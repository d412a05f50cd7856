"""Pivot blocks of two where the product of their entries leaves the format's
range although the entries do not (a state's unit is the user's)."""
import numpy as np
import pytest

from uqcreator_b200 import MIXED, workloads as W
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


def test_mixed_inverse():
    """Pressure in a unit that takes the energy block beyond 1e19, whose square
    FP32 does not hold: the inverse is not formed, and the cells take the FP64
    form's iterations, no others."""
    unit, text = 2.0 ** 40, W.euler2d(nx=12, ny=4)
    s = Solver(text)
    s.init_state()
    s.step(2)
    u, lam, level = s.download_state()
    r = np.sqrt(unit)
    u = u * np.array([1.0, r, r, unit])[:, None]
    lam = lam / np.array([1.0, r, r, unit])[:, None]
    lam[:, 0, 0] -= np.log(unit)
    info = []
    for precision in (0, MIXED):
        s = Solver(W.euler2d(nx=12, ny=4, eps=1e-10 * unit))
        s.set_precision(precision)
        s.upload_state(u, lam, level)
        info.append(s.step(1))
        assert info[-1]["failed_cells"] == 0
    assert info[0]["newton_iterations"] > 0
    assert info[1]["newton_iterations"] == info[0]["newton_iterations"]
    assert info[1]["fallback_cells"] > 0
