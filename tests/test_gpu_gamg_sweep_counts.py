"""Sweep counts of the GAMG cycle and the Jacobi smoother are what range()
takes: none below zero, and no fractions."""

import pytest
import torch

from pyopenfoam_gb300.solvers import GAMGSolver, JacobiSmoother
from tests.test_gpu_gamg_cycle import system

pytestmark = pytest.mark.gpu


def solve(m, b, pre, post):
    s = GAMGSolver(tolerance=0.0, rel_tol=0.0, max_iter=2, n_pre_smooth=pre, n_post_smooth=post)
    return s(m, b, torch.zeros_like(b))[0].view(torch.int64)


@pytest.mark.parametrize("use", [(-1, 2), (2, -3)])
@pytest.mark.parametrize("dims", [(6, 5, 4), (16, 16, 9)])
def test_a_negative_count_is_no_sweep(dims, use):
    m, b = system(dims)
    assert torch.equal(solve(m, b, *use), solve(m, b, *(max(k, 0) for k in use)))


@pytest.mark.parametrize("dims", [(6, 5, 4), (16, 16, 9)])
def test_a_fraction_is_refused(dims):
    m, b = system(dims)
    solve(m, b, 2, 2)
    for use in [(2.0, 2), (2, 1.5)]:
        with pytest.raises(TypeError):
            solve(m, b, *use)


def test_jacobi_counts():
    m, b = system((6, 5, 4))
    x0 = torch.ones_like(b)
    for k in (-2, 0):
        assert torch.equal(JacobiSmoother(m).smooth(x0, b, k), x0)
    with pytest.raises(TypeError):
        JacobiSmoother(m).smooth(x0, b, 2.5)
