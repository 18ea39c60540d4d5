"""The one-pass Jacobi sweep, the restriction with the zero start and the
one-launch coarse end of the GAMG V-cycle against the same V-cycle made of
one launch per operation (residual, relax, restrict, prolong), bit for bit:
systems whose levels all fit the one launch, just fit, or do not; odd sweep
counts (the sweeps end in the other buffer); a level without faces."""

import numpy as np
import pytest
import torch

from pyopenfoam_gb300 import LduMatrix, _lib
from pyopenfoam_gb300.mesh.poisson import hex_faces
from pyopenfoam_gb300.solvers import GAMGSolver, JacobiSmoother
from pyopenfoam_gb300.solvers.smoothers import relax, residual
from tests.golden.cases import random_ldu

pytestmark = pytest.mark.gpu


def system(dims, seed=5):
    n, own, nei = hex_faces(*dims)
    rng = np.random.default_rng(seed)
    c = rng.lognormal(0.0, 0.5, own.shape[0])
    diag = np.bincount(own, c, n) + np.bincount(nei, c, n) + 0.3
    m = LduMatrix(n, torch.as_tensor(own), torch.as_tensor(nei), device="cuda")
    m.diag, m.lower, m.upper = (torch.as_tensor(a) for a in (diag, -c, -0.9 * c))
    return m, torch.as_tensor(rng.uniform(-1, 1, n)).cuda()


def cycle(levels, aggs, i, x, b, pre, post):
    m, r = levels[i].matrix, torch.empty_like(x)

    def sweeps(k):
        for _ in range(k):
            residual(m, b, x, r)
            relax(x, r, 1.0, m.diag)

    if i == len(levels) - 1:
        return sweeps(50)
    sweeps(pre)
    residual(m, b, x, r)
    a, L, st = aggs[i], _lib.lib(), _lib.stream_ptr(m.device)
    rc = torch.empty(a.n_coarse, device=m.device, dtype=torch.float64)
    _lib.check(L.gbf_gamg_restrict_f64(a.n_coarse, a.agg_ptr.data_ptr(), a.agg_cells.data_ptr(),
                                       r.data_ptr(), rc.data_ptr(), st))
    ec = torch.zeros_like(rc)
    cycle(levels, aggs, i + 1, ec, rc, pre, post)
    _lib.check(L.gbf_gamg_prolong_add_f64(m.n_cells, a.f2c32.data_ptr(), ec.data_ptr(),
                                          x.data_ptr(), st))
    sweeps(post)


@pytest.mark.parametrize("dims,pre,post,max_levels", [
    ((2, 1, 1), 2, 2, 10), ((6, 5, 4), 1, 3, 10), ((16, 16, 8), 2, 2, 10), ((16, 16, 9), 3, 0, 10),
    ((29, 23, 17), 2, 2, 10), ((29, 23, 17), 1, 2, 1), ((33, 31, 30), 0, 1, 3), ((7, 1, 1), 2, 2, 10)])
def test_v_cycle_is_the_launch_per_operation_cycle(dims, pre, post, max_levels):
    m, b = system(dims)
    s = GAMGSolver(tolerance=0.0, rel_tol=0.0, max_iter=2, n_pre_smooth=pre, n_post_smooth=post,
                   max_levels=max_levels, min_cells_coarse=1 if dims[1] == 1 else 10)
    x0 = torch.linspace(-1, 1, m.n_cells, dtype=torch.float64, device="cuda")
    x, _, res = s(m, b, x0)
    want = x0.clone()
    levels, aggs = s._hierarchy(m)
    for _ in range(2):
        cycle(levels, aggs, 0, want, b, pre, post)
    assert torch.equal(x.view(torch.int64), want.view(torch.int64))
    r = residual(m, b, want)
    assert res == pytest.approx(float(torch.linalg.vector_norm(r)), rel=1e-13)


@pytest.mark.parametrize("n_sweeps", [1, 2, 5])
@pytest.mark.parametrize("kind", ["hex", "wide"])
def test_jacobi_sweep_is_residual_then_relax(kind, n_sweeps):
    if kind == "hex":
        m, b = system((31, 9, 8))
    else:
        d = random_ldu(9, seed=41, permute_faces=True)
        m = LduMatrix(d["n"], torch.as_tensor(d["owner"]), torch.as_tensor(d["neighbour"]),
                      device="cuda")
        m.diag, m.lower, m.upper = (torch.as_tensor(d[k]) for k in ("diag", "lower", "upper"))
        b = torch.as_tensor(d["r"]).cuda()
    x0 = torch.linspace(0, 1, m.n_cells, dtype=torch.float64, device="cuda")
    got = JacobiSmoother(m, omega=0.7).smooth(x0, b, n_sweeps)
    want, r = x0.clone(), torch.empty_like(x0)
    for _ in range(n_sweeps):
        residual(m, b, want, r)
        relax(want, r, 0.7, m.diag)
    assert torch.equal(got.view(torch.int64), want.view(torch.int64))
