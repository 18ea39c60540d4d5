"""The single-launch PCG with a cell per thread (hex 3+3 layouts up to two
blocks of 256 per SM) against the multi-cell kernel bit for bit: one block, a last block of one
cell, several blocks, one and two blocks per SM, the largest system it takes;
with and without preconditioner,
stopped by either tolerance, by the iteration limit, by breakdown and at the
first check."""

import numpy as np
import pytest
import torch

from pyopenfoam_gb300 import LduMatrix, PCGSolver
from pyopenfoam_gb300.mesh.poisson import hex_faces

pytestmark = pytest.mark.gpu


def system(dims, seed=2):
    n, own, nei = hex_faces(*dims)
    rng = np.random.default_rng(seed)
    c = rng.lognormal(0.0, 0.4, own.shape[0])
    diag = np.bincount(own, c, n) + np.bincount(nei, c, n) + 0.05
    m = LduMatrix(n, torch.as_tensor(own), torch.as_tensor(nei), device="cuda")
    m.diag, m.lower, m.upper = (torch.as_tensor(a) for a in (diag, -c, -c))
    return m, rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)


def bits(a):
    return np.asarray(a, np.float64).view(np.int64)


def check(m, b, x0, precond, monkeypatch, **tol):
    """The bits and decisions of the multi-cell kernel: the same system under an explicit-column
    layout runs that one, with the same cells in each partial sum."""
    out = []
    for layout in (None, m.topology().uncompressed_layout()):
        if layout is not None:
            monkeypatch.setattr(m.topology(), "layout", layout)
        s = PCGSolver(preconditioner=precond, launch="single", **tol)
        x, it, res = s(m, torch.as_tensor(b), torch.as_tensor(x0))
        out.append((x.cpu().numpy(), it, res, s.last_info))
    (x, it, res, info), (x2, it2, res2, info2) = out
    assert it2 == it and info2.converged == info.converged
    assert (bits(x) == bits(x2)).all() and bits([res]) == bits([res2])
    assert (bits(info.residual_history) == bits(info2.residual_history)).all()


@pytest.mark.parametrize("precond", ["DIC", "none"])
@pytest.mark.parametrize("dims", [(6, 5, 4), (16, 16, 1), (257, 1, 1), (19, 17, 13), (36, 33, 32),
                                  (45, 41, 37), (64, 64, 19)])
def test_resident_pcg_is_the_multi_cell_kernel(dims, precond, monkeypatch):
    m, b, x0 = system(dims)
    check(m, b, x0, precond, monkeypatch, tolerance=0.0, rel_tol=1e-9, max_iter=4000)


@pytest.mark.parametrize("tol", [
    dict(tolerance=1e-3, rel_tol=0.0, max_iter=500), dict(tolerance=1e-7, rel_tol=1e-3, max_iter=500),
    dict(tolerance=0.0, rel_tol=0.0, max_iter=7), dict(tolerance=0.0, rel_tol=2.0, max_iter=5),
    dict(tolerance=1e9, rel_tol=0.0, max_iter=5), dict(tolerance=0.0, rel_tol=1e-6, max_iter=0),
    dict(tolerance=-1.0, rel_tol=-1.0, max_iter=9)])
def test_stopping_rules(tol, monkeypatch):
    m, b, x0 = system((11, 9, 8))
    check(m, b, x0, "DIC", monkeypatch, **tol)


def test_zero_source_breaks_down(monkeypatch):
    m, b, x0 = system((9, 8, 7))
    check(m, 0 * b, 0 * x0, "DIC", monkeypatch, tolerance=0.0, rel_tol=1e-6, max_iter=20)


@pytest.mark.parametrize("scale", [1e-160, 1e160, float("nan"), float("inf")])
def test_norms_outside_the_ordinary_range(scale):
    """The rules applied as they stand: the three-kernel form takes the same decisions."""
    m, b, x0 = system((9, 8, 7))
    out = []
    for launch in ("single", "kernels"):
        s = PCGSolver(tolerance=0.0, rel_tol=1e-6, max_iter=30, launch=launch)
        x, it, res = s(m, torch.as_tensor(b * scale), torch.as_tensor(0 * x0))
        out.append((it, s.last_info.converged, np.isfinite(res)))
    assert out[0] == out[1]
