"""The autotuner's saved tunings (host code)."""
import json

import pytest

from uqcreator_b200 import Solver, UqcError, workloads as W
from uqcreator_b200.autotune import autotune


def test_tunings_of_earlier_kernels_are_not_applied(tmp_path):
    """closure_group 32 and 256 exclude the batched Newton kernel, so a tuning
    that was saved when they were launch shapes of one kernel is stale: the
    configuration is tuned again (here it has no state to be tuned on)."""
    cache = tmp_path / "tune.json"
    saved = {"best": {"closure_group": 32}, "ms_per_step": {}}
    cache.write_text(json.dumps({"v4_s1_t15_q32_l1_d1_p0_m0": saved}))
    s = Solver(W.burgers1d(ncells=30, degree=14, nquad=32))
    assert (s.n_states, s.n_total, s.n_quad, s.n_levels, s.dim_xi) == (1, 15, 32, 1, 1)
    with pytest.raises(UqcError):
        autotune(s, cache=cache)
