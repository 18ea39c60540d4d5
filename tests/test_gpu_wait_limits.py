"""Waits of the cell-per-thread PCG and of the block walks that nothing ends: the
kernel returns after its limit with the fault word set and an invalid result,
and the context stays usable.  The walks are given a schedule that leaves a
cell out, so that the cell after it never finds its value; all indices are in
range."""

import ctypes

import numpy as np
import pytest
import torch

from pyopenfoam_gb300 import LduMatrix, PCGSolver, _lib
from pyopenfoam_gb300.solvers.preconditioners import factor_dic
from pyopenfoam_gb300.solvers.smoothers import gs_sweep

pytestmark = pytest.mark.gpu


def chain(n=40):
    own = torch.arange(n - 1)
    m = LduMatrix(n, own, own + 1, device="cuda")
    one = torch.ones(n, dtype=torch.float64)
    m.diag, m.lower, m.upper = 3.0 * one, -one[1:], -one[1:]
    return m


def test_resident_pcg_gives_up():
    out = (ctypes.c_int32 * 2)()
    _lib.check(_lib.lib().gbf_selftest_pcg_resident_fault(out))
    assert list(out) == [1, 1]
    m, b = chain(), torch.ones(40, dtype=torch.float64)
    s = PCGSolver(tolerance=0.0, rel_tol=1e-12, max_iter=100)
    x, _, _ = s(m, b, torch.zeros_like(b))
    assert s.last_info.converged and torch.allclose(m.Ax(x), b.cuda(), rtol=1e-9)


def short_order(m, left_out):
    """One block of all cells in order, but for one."""
    cells = [c for c in range(m.n_cells) if c != left_out]
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")  # noqa: E731
    return i32(cells), i32([0, len(cells)])


def fault(barrier):
    out = ctypes.c_int32()
    _lib.check(_lib.lib().gbf_wavefront_fault(barrier.data_ptr(), ctypes.byref(out),
                                              _lib.stream_ptr(barrier.device)))
    return out.value


@pytest.mark.parametrize("left_out", [0, 35])
def test_dic_block_walk_gives_up(left_out):
    m = chain()
    cells, ptr = short_order(m, left_out)
    d = torch.zeros(m.n_cells, dtype=torch.float64, device="cuda")
    bar = torch.zeros(64, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib().gbf_dic_build_block_f64(
        m.topology().layout_ref, m.packed().data_ptr(), m.diag.data_ptr(), cells.data_ptr(),
        ptr.data_ptr(), 1, m.n_cells, d.data_ptr(), bar.data_ptr(), _lib.stream_ptr(m.device)))
    assert fault(bar) == 1 and torch.isnan(d).all()
    factor_dic(m.topology(), m.packed(), m.diag, d, m.device, "flow")
    assert torch.isfinite(d).all()


@pytest.mark.parametrize("left_out", [0, 35])
def test_gauss_seidel_block_walk_gives_up(left_out):
    m = chain()
    cells, ptr = short_order(m, left_out)
    b = torch.ones(m.n_cells, dtype=torch.float64, device="cuda")
    x, scratch = torch.zeros_like(b), torch.zeros_like(b)
    bar = torch.zeros(64, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib().gbf_gauss_seidel_block_f64(
        m.topology().layout_ref, m.packed().data_ptr(), m.diag.data_ptr(), b.data_ptr(),
        cells.data_ptr(), ptr.data_ptr(), 1, m.n_cells, 0, 1.0, 0, x.data_ptr(),
        scratch.data_ptr(), bar.data_ptr(), _lib.stream_ptr(m.device)))
    assert fault(bar) == 1 and torch.isnan(x).all()
    x.zero_()
    gs_sweep(m, x, b, form="flow")
    assert torch.isfinite(x).all() and np.isclose(float(x[0]), 1.0 / 3.0)
