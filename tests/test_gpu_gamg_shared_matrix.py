"""GAMG solvers with different settings on one unchanged matrix: each runs its
own V-cycle."""

import pytest
import torch

from pyopenfoam_gb300.solvers import GAMGSolver
from tests.test_gpu_gamg_cycle import cycle, system

pytestmark = pytest.mark.gpu


def solver(pre, post, use_graph=True):
    return GAMGSolver(tolerance=0.0, rel_tol=0.0, max_iter=2, n_pre_smooth=pre,
                      n_post_smooth=post, use_graph=use_graph)


def expected(s, m, b, x0, pre, post):
    x = x0.clone()
    levels, aggs = s._hierarchy(m)
    for _ in range(2):
        cycle(levels, aggs, 0, x, b, pre, post)
    return x.view(torch.int64)


@pytest.mark.parametrize("dims", [(6, 5, 4), (16, 16, 9)])
@pytest.mark.parametrize("use_graph", [True, False])
def test_each_solver_runs_its_own_cycle(dims, use_graph):
    m, b = system(dims)
    x0 = torch.linspace(-1, 1, m.n_cells, dtype=torch.float64, device="cuda")
    for pre, post in [(2, 2), (1, 3), (3, 0), (2, 2)]:
        s = solver(pre, post, use_graph)
        x, _, _ = s(m, b, x0)
        assert torch.equal(x.view(torch.int64), expected(s, m, b, x0, pre, post))


def test_a_solver_without_graph_after_one_with():
    m, b = system((16, 16, 9))
    x0 = torch.zeros(m.n_cells, dtype=torch.float64, device="cuda")
    solver(2, 2, True)(m, b, x0)
    solver(2, 2, False)(m, b, x0)
    assert [("graph" in v) for k, v in m._csr_cache.items() if k[0] == "gamg_cycle"] == [True,
                                                                                       False]
