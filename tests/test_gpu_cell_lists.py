"""Cell -> face lists made on the device against the host pass that defines
their order, whole numbers that have to be equal: counts at the edges of the
1024-cell scan blocks, cells without faces, no internal faces, owners and
neighbours in no order, a cell at the largest and beyond the largest number of
faces, and indices outside the mesh (refused by the host pass as before)."""

import numpy as np
import pytest
import torch

from pyopenfoam_gb300 import _lib
from pyopenfoam_gb300.mesh import FvMesh

pytestmark = pytest.mark.gpu


def _mesh(own, nei):
    """A mesh of triangles on three points: only its addressing matters here."""
    nf = own.shape[0]
    return FvMesh(np.eye(3), (np.arange(0, 3 * nf + 1, 3), np.tile(np.arange(3), nf)), own, nei,
                  validate=False, device="cuda")


@pytest.mark.parametrize("n,nf,ni", [(1, 1, 0), (1, 6, 0), (2, 11, 1), (1023, 3000, 2500),
                                     (1024, 3000, 0), (1025, 3000, 3000), (5000, 700, 650),
                                     (70001, 256 * 900 + 1, 200000), (1, 4096, 0), (3, 4100, 90)])
def test_lists_match_the_host_pass(n, nf, ni):
    rng = np.random.default_rng(n + nf)
    own = rng.integers(0, n, nf)
    own[rng.integers(nf)] = n - 1
    nei = rng.integers(0, n, ni)
    m = _mesh(own, nei)
    got, want = m._cell_faces_device(), m._cell_faces_host()
    assert got is not None
    for g, w, k in zip(got, want, (nf, ni, n + 1, nf + ni)):
        assert torch.equal(g[:k], w[:k])


def test_a_cell_of_too_many_faces_takes_the_host_pass():
    own = np.zeros(4097, np.int64)
    m = _mesh(own, np.zeros(0, np.int64))
    assert m._cell_faces_device() is None
    assert torch.equal(m._addr()["cell_faces"].cpu(), torch.arange(4097, dtype=torch.int32))


@pytest.mark.parametrize("own,nei", [([0, -1, 1], [1]), ([0, 1, 1], [2]), ([0, 0, 0], [-5, 0])])
def test_cells_outside_the_mesh_are_refused(own, nei):
    m = _mesh(np.array(own), np.array(nei))
    assert m._cell_faces_device() is None
    with pytest.raises(_lib.GbfError, match="outside"):
        m.face_centres
