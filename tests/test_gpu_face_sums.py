"""Sums over a cell's faces in the pressure equation's and the upwind diagonal,
bit for bit against the sums written out in face order: at most one, three,
four (bodies of their own) and more slots a side, ragged last slices, cells
without faces."""

import numpy as np
import pytest
import torch

from pyopenfoam_gb300 import _lib
from pyopenfoam_gb300.core.topology import Topology

pytestmark = pytest.mark.gpu


def _sums(n, own, nei, of_own, of_nei):
    so, sn = np.zeros(n), np.zeros(n)
    for f in range(nei.size):
        so[own[f]] += of_own[f]
        sn[nei[f]] += of_nei[f]
    return so + sn


@pytest.mark.parametrize("n,side", [(1, 0), (33, 1), (100, 3), (257, 4), (130, 5), (64, 9)])
def test_sums_follow_the_face_order(n, side):
    rng = np.random.default_rng(7 * n + side)
    pairs = [(c, c + s) for c in range(n) for s in range(1, side + 1)
             if c + s < n and rng.random() < 0.8]
    own = np.array([a for a, _ in pairs], np.int64)
    nei = np.array([b for _, b in pairs], np.int64)
    nf, nb = own.size, 5
    at = rng.integers(0, n, nb)  # cells of the boundary faces
    bnd_face = nf + np.argsort(at, kind="stable")
    bnd_ptr = np.concatenate([[0], np.cumsum(np.bincount(at, minlength=n))])
    V, A = rng.uniform(0.5, 2, n), rng.normal(size=n)
    delta, w = rng.uniform(1, 3, nf + nb), rng.uniform(0, 1, nf + nb)
    phi = rng.normal(size=nf + nb)
    areas = np.zeros((nf + nb, 3))
    areas[:, 0] = 1.0  # |S| = 1

    dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", t)  # noqa: E731
    f64, i32 = torch.float64, torch.int32
    topo = Topology(n, dev(own, torch.int64), dev(nei, torch.int64))
    t = [dev(a, f64) for a in (areas, delta, w, A, V, phi)]
    bp, bf = dev(bnd_ptr, i32), dev(bnd_face, i32)
    lower, upper, diag, source, div = (torch.full((k,), 9.0, dtype=f64, device="cuda")
                                       for k in (nf + 1, nf + 1, n, n, n))
    s, L = _lib.stream_ptr(torch.device("cuda")), _lib.lib()
    _lib.check(L.gbf_pressure_assemble_f64(
        topo.layout_ref, nf + nb, bp.data_ptr(), bf.data_ptr(), *[a.data_ptr() for a in t],
        lower.data_ptr(), upper.data_ptr(), diag.data_ptr(), source.data_ptr(), s))

    inv = 1.0 / np.maximum(np.abs(A), 1e-30)
    c = (w[:nf] * inv[own] + (1.0 - w[:nf]) * inv[nei]) * 1.0 * delta[:nf]
    lo, up = -c / V[own], -c / V[nei]
    assert np.array_equal(lower[:nf].cpu().numpy(), lo)
    assert np.array_equal(upper[:nf].cpu().numpy(), up)
    assert np.array_equal(diag.cpu().numpy(), _sums(n, own, nei, -lo, -up))
    src = _sums(n, own, nei, -phi[:nf], phi[:nf])
    bnd = np.zeros(n)
    for f in np.sort(bnd_face):
        bnd[at[f - nf]] += -phi[f]
    assert np.array_equal(source.cpu().numpy(), (src + bnd) / V)

    _lib.check(L.gbf_div_upwind_assemble_f64(
        topo.layout_ref, t[5].data_ptr(), t[4].data_ptr(), lower.data_ptr(), upper.data_ptr(),
        div.data_ptr(), s))
    F = phi[:nf]
    pos, neg = np.where(F >= 0, F, 0.0), np.where(F < 0, F, 0.0)
    assert np.array_equal(div.cpu().numpy(),
                          _sums(n, own, nei, -pos / V[own], np.abs(neg) / V[nei]))
