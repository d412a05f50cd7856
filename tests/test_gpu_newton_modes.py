"""A live handle whose Newton settings change (uqc_set_newton): the launch plan
follows, whatever mode the handle was set up in. Against the FP64 oracle."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from uqcreator_b200 import MIXED, workloads as W
from uqcreator_b200.solver import Solver

pytestmark = pytest.mark.gpu

MODES = {"reference": 0, "guarded": 1, "safe": 2}
STEPS = 5
# one per update kernel: several lanes per cell, a warp per cell, tensor cores
CASES = {
    "burgers_5_moments": lambda **kw: W.burgers1d(ncells=120, tend=10.0, **kw),
    "burgers_17_moments": lambda **kw: W.burgers1d(ncells=40, degree=16, nquad=35, tend=10.0, **kw),
    "sw_levels": lambda **kw: W.shallow_water1d(ncells=90, max_degree=4, nquad=12, tend=10.0, **kw),
    "euler_6_moments": lambda **kw: W.euler2d(nx=9, ny=4, degree=2, nquad=5, tend=10.0, **kw),
    "euler_21_moments": lambda **kw: W.euler2d(nx=9, ny=4, tend=10.0, **kw),
}


@pytest.mark.parametrize("before", [0, 2], ids=["at_once", "after_steps"])
@pytest.mark.parametrize("modes", [("safe", "first"), ("first", "safe")], ids=["leaving_safe", "to_safe"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_mode_of_a_live_handle(name, modes, before):
    """Steps after a change of mode, through uqc_step and through uqc_run's
    graphs, as an oracle in that mode takes them from the same state (moments
    within 1e-9 of their largest, as in the step tests)."""
    first = "guarded" if name.startswith("euler") else "reference"
    a, b = (first if m == "first" else m for m in modes)
    text = {m: CASES[name](newton=m, steps=before + STEPS) for m in (a, b)}
    o = Oracle(text[a], W.mesh_for(text[a]))
    o.init_state()
    if before:
        o.step(before)
    late = Oracle(text[b], W.mesh_for(text[b]))
    late.init_state()
    late.set_state(*o.get_state())
    late.step(STEPS)
    expect = late.get_state()[0]
    for graphs in (False, True):
        s = Solver(text[a])
        if name == "sw_levels":
            s.set_option("update_test", 1)    # automatic: off with refinement levels
        s.init_state()
        s.step(before)
        s.set_newton(1000, 1e-10, MODES[b])
        info = s.run() if graphs else s.step(STEPS)
        assert info["steps"] == STEPS and info["failed_cells"] == 0 and np.isfinite(info["dt"])
        np.testing.assert_allclose(s.download_state()[0], expect, rtol=0, atol=1e-9 * np.abs(expect).max())


def test_mixed_form_follows_the_mode():
    """UQC_MIXED set up in safe mode has no rounds; after the change it has, and
    their held factors start empty (the mixed bound of the step tests)."""
    safe, guarded = (W.euler2d(nx=12, ny=4, tend=10.0, newton=m) for m in ("safe", "guarded"))
    o = Oracle(guarded, W.mesh_for(guarded))
    o.init_state()
    o.step(STEPS)
    s = Solver(safe)
    s.set_precision(MIXED)
    s.init_state()
    s.step(1)
    s.set_newton(1000, 1e-10, 1)
    assert s.form()["mixed_form"] == 2
    s.init_state()
    assert s.step(STEPS)["failed_cells"] == 0
    expect = o.get_state()[0]
    np.testing.assert_allclose(s.download_state()[0], expect, rtol=0, atol=1e-6 * np.abs(expect).max())
    s.set_newton(1000, 1e-10, 2)
    assert s.form()["mixed_form"] == 0
    s.init_state()
    assert s.step(STEPS)["failed_cells"] == 0
    np.testing.assert_allclose(s.download_state()[0], expect, rtol=0, atol=1e-6 * np.abs(expect).max())


def test_rounds_that_appear_between_steps():
    """mixed_chord 0 and 1 again on a live handle: the rounds start from gradients
    that the single kernel's steps did not store, so every cell is tested anew.
    The same state uploaded again, where every cell is, gives the same steps."""
    s = Solver(W.euler2d(nx=24, ny=5, tend=10.0))
    s.set_precision(MIXED)
    s.init_state()
    s.set_option("mixed_chord", 0)
    s.step(2)
    state, t = s.download_state(), s.step(0)["t"]
    s.set_option("mixed_chord", 1)
    assert s.form()["mixed_form"] == 2
    a = s.step(STEPS)
    ua, la, _ = s.download_state()
    s.upload_state(*state, t=t)
    b = s.step(STEPS)
    ub, lb, _ = s.download_state()
    assert a["failed_cells"] == b["failed_cells"] == 0
    assert a["fallback_cells"] == b["fallback_cells"] and a["newton_iterations"] == b["newton_iterations"]
    np.testing.assert_array_equal(ua, ub)
    np.testing.assert_array_equal(la, lb)
