"""Workspaces of the FP64 PCG entry point: a caller may size one for its
largest system and pass it for smaller ones, and may pass the least size (four
vectors, partial sums, state), where the multi-cell kernel runs in place of the
cell-per-thread one with the same bits."""

import ctypes

import numpy as np
import pytest
import torch

from pyopenfoam_gb300 import LduMatrix, _lib
from pyopenfoam_gb300.mesh.poisson import hex_faces
from pyopenfoam_gb300.solvers.preconditioners import DICPreconditioner

pytestmark = pytest.mark.gpu
GUARD = 0xA5


def least_bytes(n):
    up = lambda k: (k + 255) // 256 * 256  # noqa: E731
    return 4 * up(8 * n) + up(8 * 2 * 4096) + 256


def system(dims, seed=4):
    n, own, nei = hex_faces(*dims)
    rng = np.random.default_rng(seed)
    c = rng.lognormal(0.0, 0.4, own.shape[0])
    diag = np.bincount(own, c, n) + np.bincount(nei, c, n) + 0.05
    m = LduMatrix(n, torch.as_tensor(own), torch.as_tensor(nei), device="cuda")
    m.diag, m.lower, m.upper = (torch.as_tensor(a) for a in (diag, -c, -c))
    return m, torch.as_tensor(rng.uniform(-1, 1, n)).cuda()


def solve(m, b, pd, nbytes, room=None, offset=0, max_iter=40):
    """x, history and the workspace's bytes after a solve in `nbytes` of it."""
    L = _lib.lib()
    ws = torch.full((offset + (room or nbytes) + 4096,), GUARD, dtype=torch.uint8, device="cuda")
    x = torch.zeros_like(b)
    hist = torch.zeros(max_iter + 1, dtype=torch.float64, device="cuda")
    P, R = _lib.SolveParams(0.0, 1e-9, max_iter, 0, 16, 0), _lib.SolveResult()
    _lib.check(L.gbf_pcg_solve_f64(
        m.topology().layout_ref, m.packed().data_ptr(), m.diag.data_ptr(), pd.data_ptr(),
        b.data_ptr(), x.data_ptr(), hist.data_ptr(), ctypes.byref(P), ctypes.byref(R),
        ws.data_ptr() + offset, nbytes, _lib.stream_ptr(m.device)), "gbf_pcg_solve_f64")
    assert (ws[offset + nbytes:] == GUARD).all() and (ws[:offset] == GUARD).all()
    return [x.view(torch.int64), hist.view(torch.int64)], R.iterations, ws


@pytest.mark.parametrize("dims", [(32, 32, 32), (64, 64, 19), (64, 64, 32)])
def test_one_workspace_for_the_largest_system(dims):
    """A workspace sized for 200000 cells, the least one and the query's own, on 32768, 77824
    and 131072 cells."""
    m, b = system(dims)
    pd, n = DICPreconditioner(m).precond_diag, m.n_cells
    query = _lib.lib().gbf_pcg_workspace_bytes
    want, its, _ = solve(m, b, pd, least_bytes(n))
    for nbytes in (query(n), query(200000), least_bytes(200000)):
        got, it, _ = solve(m, b, pd, nbytes)
        assert it == its and all(torch.equal(g, w) for g, w in zip(got, want))
    with pytest.raises(_lib.GbfError, match="workspace too small"):
        solve(m, b, pd, least_bytes(n) - 1, room=least_bytes(n))


def test_the_cell_per_thread_kernel_runs_where_its_words_have_room():
    m, b = system((32, 32, 32))
    pd, n = DICPreconditioner(m).precond_diag, m.n_cells
    query = _lib.lib().gbf_pcg_workspace_bytes
    for nbytes, words in ((least_bytes(n), False), (query(n) - 1, False), (query(n), True),
                          (query(400000), True)):
        _, _, ws = solve(m, b, pd, nbytes)
        assert bool((ws[least_bytes(n):] != GUARD).any()) == words


def test_the_query_grows_with_the_system():
    query = _lib.lib().gbf_pcg_workspace_bytes
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    last = min(2 * sms, 512) * 256  # the largest system of the cell-per-thread kernel
    ns = sorted({0, 1, 255, 256, 257, 32768, last - 1, last, last + 1, 131072, 131073, 200000,
                 400000, 650000, 1 << 21, *range(1, 700000, 9973)})
    got = [query(n) for n in ns]
    assert all(a <= b for a, b in zip(got, got[1:]))
    assert all(least_bytes(n) <= g <= max(least_bytes(n), query(last)) for n, g in zip(ns, got)
               if n > last)


@pytest.mark.parametrize("dims", [(6, 5, 4), (32, 32, 32)])
def test_a_workspace_aligned_to_eight_bytes(dims):
    m, b = system(dims)
    pd, n = DICPreconditioner(m).precond_diag, m.n_cells
    nbytes = _lib.lib().gbf_pcg_workspace_bytes(n)
    want, its, _ = solve(m, b, pd, nbytes)
    got, it, _ = solve(m, b, pd, nbytes, offset=8)
    assert it == its and all(torch.equal(g, w) for g, w in zip(got, want))
