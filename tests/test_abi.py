"""The C ABI library loads without a GPU, exports every symbol include/uqc.h
declares, and its host-side parts (configuration, footprint, admission
limits) work on the CPU."""
import ctypes as C
import re
from pathlib import Path

import pytest

import uqcreator_b200._lib as L
from uqcreator_b200 import Solver, UqcError, workloads as W
from uqcreator_b200.serve import Server

HEADER = Path(__file__).resolve().parents[1] / "include" / "uqc.h"


def declared_functions():
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return sorted(set(re.findall(r"\b(uqc_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_function():
    lib = L.lib()
    names = declared_functions()
    assert len(names) >= 30
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing, missing
    assert sorted(L.EXPORTS) == names


def test_config_errors_are_reported_not_fatal():
    with pytest.raises(UqcError) as e:
        Solver(W.burgers1d().replace('closure = "BoundedBarrier"', 'closure = "NoSuchClosure"'))
    assert e.value.code == -2


def test_device_footprint_is_host_side_and_grows_with_cells():
    a = Solver(W.burgers1d(ncells=200)).device_bytes()
    b = Solver(W.burgers1d(ncells=2000)).device_bytes()
    assert 0 < a < b


def test_server_rejects_request_beyond_budget_without_gpu_work():
    toml = W.burgers1d(ncells=2000)
    need = Solver(toml).device_bytes()
    srv = Server(budget_bytes=need // 2, max_active=2, steps_per_slice=1)
    rid = srv.submit(toml)
    q, r, d = srv.progress()
    assert (q, r, d) == (0, 0, 1)
    info = srv.result(rid)
    assert info["state"] == "failed" and info["status"] == -7
    srv.release(rid)
    with pytest.raises(UqcError):
        srv.info(rid)


def test_device_footprint_counts_every_table():
    """What does not grow with the cells, 140 duals on 512 nodes: phi, phi wt, phi
    node-contiguous and in FP32, the update's padded phi wt (40 columns and 4),
    the places of the pairs' ten blocks, the nodes and their weights."""
    nt, nq = 35, 512
    few, more = (Solver(W.euler2d(nx=3, ny=n, degree=4, nquad=8, dim_xi=3)) for n in (2, 3))
    cell = (more.device_bytes() - few.device_bytes()) / (more.n_cells - few.n_cells)
    tables = nq * nt * (8 + 8 + 8 + 4) + nq * 44 * 8 + nt * (nt + 1) // 2 * 10 * 4 + nq * (3 + 1) * 8
    ghost = 8 * 4 * nq
    other = 40 * 1024    # the control block, the residual's partial sums, row padding
    assert tables + ghost <= few.device_bytes() - cell * few.n_cells <= tables + ghost + other


def test_device_footprint_counts_the_tiny_kernel_table():
    """20 nodes, 5 duals: 32 columns of Hessian and gradient weights. The other
    tables and a cell's share, then 10 duals with 96 columns."""
    def table(degree):
        few, more = (Solver(W.burgers1d(ncells=n, degree=degree, nquad=20)).device_bytes() for n in (3, 4))
        return few - 3 * (more - few)    # what does not grow with the cells
    # 5 -> 10 duals: five more columns of phi, phi wt, phi^T (8 bytes each) and FP32 phi
    # (row strides 5 and 11), 64 more columns of the tiny kernel's table
    assert table(9) - table(4) >= 20 * (6 * (8 + 8 + 4) + 5 * 8 + 64 * 8)
