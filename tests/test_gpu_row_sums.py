"""Residual, Jacobi sweep and the coarse end of the GAMG V-cycle against the
matrix product b - A x, which has its own gather, bit for bit: random
numberings, layouts of few and of many slices, slices of more slots than are
held at a time, and rows too many for the coarse end's shared memory."""

import numpy as np
import pytest
import torch

from pyopenfoam_gb300 import LduMatrix, _lib
from pyopenfoam_gb300.mesh.poisson import hex_faces
from pyopenfoam_gb300.solvers import GAMGSolver, JacobiSmoother
from pyopenfoam_gb300.solvers.smoothers import residual

pytestmark = pytest.mark.gpu
ROW_SLOTS, TAIL_ROWS = 32, 8192


def matrix(n, own, nei, rng):
    lo, up = -rng.lognormal(0.0, 0.5, (2, own.shape[0]))
    diag = np.bincount(own, -lo, n) + np.bincount(nei, -up, n) + rng.uniform(0.1, 1.0, n)
    m = LduMatrix(n, torch.as_tensor(own), torch.as_tensor(nei), device="cuda")
    m.diag, m.lower, m.upper = (torch.as_tensor(a) for a in (diag, lo, up))
    vec = lambda: torch.as_tensor(rng.uniform(-1, 1, n)).cuda()  # noqa: E731
    return m, vec(), vec()


def renumbered(dims, seed=6):
    rng = np.random.default_rng(seed)
    n, own, nei = hex_faces(*dims)
    p = rng.permutation(n)
    own, nei = np.minimum(p[own], p[nei]), np.maximum(p[own], p[nei])
    o = np.lexsort((nei, own))
    return matrix(n, own[o], nei[o], rng)


def graph(n, pairs, seed=7):
    """Random pairs of cells, the lower-numbered ones in more of them."""
    rng = np.random.default_rng(seed)
    a, b = (n * rng.random((2, pairs)) ** 1.3).astype(np.int64)
    keep = a != b
    own, nei = np.unique(np.stack([np.minimum(a, b), np.maximum(a, b)])[:, keep], axis=1)
    return matrix(n, own, nei, rng)


def bits(t):
    return t.view(torch.int64)


def sweep(m, b, x, omega):
    s = omega * (1.0 / m.diag.abs().clamp(min=1e-30))
    return x + s * (b - m.Ax(x))


SYSTEMS = {"few_slices": lambda: renumbered((31, 29, 27)),
           "many_slices": lambda: renumbered((48, 40, 37)),
           "cells": lambda: renumbered((60, 50, 41)),
           "cells_2d": lambda: renumbered((330, 300, 1)),
           "one_slice": lambda: graph(30, 200),
           "wide_few": lambda: graph(1003, 16000),
           "wide_many": lambda: graph(39999, 700000),
           "wide_full": lambda: graph(99999, 900000)}


def kernel(t):
    """Which of the kernels the layout takes."""
    per_sm = t.n_slices / torch.cuda.get_device_properties(0).multi_processor_count
    return "cells" if per_sm > 18 and t.max_width <= 40 else "few" if per_sm <= 8 else "many"


@pytest.mark.parametrize("kind,takes", [
    ("few_slices", "few"), ("many_slices", "many"), ("cells", "cells"), ("cells_2d", "cells"),
    ("one_slice", "few"), ("wide_few", "few"), ("wide_many", "many"), ("wide_full", "many")])
def test_residual_and_jacobi_are_the_product(kind, takes):
    m, b, x = SYSTEMS[kind]()
    t = m.topology()
    assert kernel(t) == takes and (t.max_width > ROW_SLOTS) == kind.startswith("wide")
    assert torch.equal(bits(residual(m, b, x)), bits(b - m.Ax(x)))
    want = x
    for k in range(1, 4):
        want = sweep(m, b, want, 0.7)
        assert torch.equal(bits(JacobiSmoother(m, omega=0.7).smooth(x, b, k)), bits(want))


def cycle(levels, aggs, i, x, b, pre, post):
    m = levels[i].matrix
    for _ in range(50 if i == len(levels) - 1 else pre):
        x = sweep(m, b, x, 1.0)
    if i == len(levels) - 1:
        return x
    a, r = aggs[i], b - m.Ax(x)
    rc = torch.empty(a.n_coarse, device=m.device, dtype=torch.float64)
    _lib.check(_lib.lib().gbf_gamg_restrict_f64(
        a.n_coarse, a.agg_ptr.data_ptr(), a.agg_cells.data_ptr(), r.data_ptr(), rc.data_ptr(),
        _lib.stream_ptr(m.device)), "gbf_gamg_restrict_f64")
    x = x + cycle(levels, aggs, i + 1, torch.zeros_like(rc), rc, pre, post)[a.fine_to_coarse]
    for _ in range(post):
        x = sweep(m, b, x, 1.0)
    return x


@pytest.mark.parametrize("n,pairs,staged", [(250, 4000, False), (256, 30000, False),
                                            (150, 500, True)])
def test_coarse_end_is_the_product(n, pairs, staged):
    m, b, x = graph(n, pairs)
    s = GAMGSolver(tolerance=0.0, rel_tol=0.0, max_iter=1, n_pre_smooth=1, n_post_smooth=2)
    levels, aggs = s._hierarchy(m)
    assert s._tail(levels, aggs)[0] == 0 and len(levels) > 1
    assert (m.topology().n_slots <= TAIL_ROWS) == staged
    got, _, _ = s(m, b, x)
    assert torch.equal(bits(got), bits(cycle(levels, aggs, 0, x, b, 1, 2)))
