"""The block walks of the DIC factorisation and the Gauss-Seidel sweep (cells
dealt to blocks that pass values through shared memory) and the walks over the
whole schedule, against one launch per level, bit for bit: one cell, a block
not full, a block just overfull, several blocks, random numberings (values
mostly cross blocks), faces in any order, holes and zero rows."""

import numpy as np
import pytest
import torch

from pyopenfoam_gb300 import LduMatrix
from pyopenfoam_gb300.core.topology import WALK_CELLS_MAX, WALK_CELLS_MIN, block_order
from pyopenfoam_gb300.mesh.poisson import hex_faces
from pyopenfoam_gb300.solvers import smoothers
from pyopenfoam_gb300.solvers.preconditioners import factor_dic

pytestmark = pytest.mark.gpu
DIMS = [(1, 1, 1), (511, 1, 1), (513, 1, 1), (33, 31, 5), (40, 30, 29), (97, 83, 61)]


def matrix(dims, kind, seed=3):
    rng = np.random.default_rng(seed)
    n, own, nei = hex_faces(*dims)
    if kind == "renumbered":
        p = rng.permutation(n)
        own, nei = np.minimum(p[own], p[nei]), np.maximum(p[own], p[nei])
        o = np.lexsort((nei, own))
        own, nei = own[o], nei[o]
    elif kind == "shuffled":  # faces in any order, some of them owner > neighbour
        o = rng.permutation(own.shape[0])
        flip = rng.random(own.shape[0]) < 0.3
        own, nei = np.where(flip, nei, own)[o], np.where(flip, own, nei)[o]
    lo, up = -rng.lognormal(0.0, 0.5, (2, own.shape[0]))
    diag = np.bincount(own, -lo, n) + np.bincount(nei, -up, n) + rng.uniform(0.1, 1.0, n)
    diag[rng.random(n) < 0.002] = 0.0
    m = LduMatrix(n, torch.as_tensor(own), torch.as_tensor(nei), device="cuda")
    m.diag, m.lower, m.upper = (torch.as_tensor(a) for a in (diag, lo, up))
    b = torch.as_tensor(rng.uniform(-1, 1, n) * (rng.random(n) < 0.9)).cuda()
    return m, b


def bits(t):
    return t.nan_to_num(nan=7.0).view(torch.int64)


@pytest.mark.parametrize("kind", ["mesh", "renumbered", "shuffled"])
@pytest.mark.parametrize("dims", DIMS)
def test_dic_walks(dims, kind, monkeypatch):
    m, _ = matrix(dims, kind)
    topo, out = m.topology(), []
    assert topo.dic_blocks() is not None
    for form in ("per_level", "flow", "whole"):
        if form == "whole":
            monkeypatch.setattr(topo, "_dic_blocks", None)
        d = torch.empty(m.n_cells, dtype=torch.float64, device="cuda")
        factor_dic(topo, m.packed(), m.diag, d, m.device, "flow" if form == "whole" else form)
        out.append(d)
    assert torch.equal(bits(out[0]), bits(out[1])) and torch.equal(bits(out[0]), bits(out[2]))


@pytest.mark.parametrize("relax", [False, True])
@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("kind", ["mesh", "renumbered", "shuffled"])
@pytest.mark.parametrize("dims", DIMS)
def test_gauss_seidel_walks(dims, kind, reverse, relax, monkeypatch):
    m, b = matrix(dims, kind)
    x0, out = torch.linspace(-1, 1, m.n_cells, dtype=torch.float64, device="cuda"), []
    for form in ("per_level", "flow", "whole"):
        if form == "whole":
            monkeypatch.setattr(smoothers._gs_schedule(m, reverse), "blocks", None)
        x = x0.clone()
        smoothers.gs_sweep(m, x, b, reverse=reverse, omega=0.8, relax=relax,
                           form="flow" if form == "whole" else form)
        out.append(x)
    assert torch.equal(bits(out[0]), bits(out[1])) and torch.equal(bits(out[0]), bits(out[2]))


@pytest.mark.parametrize("n", [1, WALK_CELLS_MIN, WALK_CELLS_MIN + 1, 200000])
def test_block_order_deals_every_cell_once_in_level_order(n):
    rng = np.random.default_rng(n)
    cells = rng.permutation(n).astype(np.int32)
    o = block_order(cells, torch.device("cuda"))
    ptr, got = o.ptr.cpu().numpy(), o.cells.cpu().numpy()
    assert sorted(got.tolist()) == list(range(n)) and ptr[0] == 0 and ptr[-1] == n
    rank = np.empty(n, np.int64)
    rank[cells] = np.arange(n)
    for k in range(o.n_blocks):
        mine = got[ptr[k]:ptr[k + 1]]
        assert (mine // o.per == k).all() and (np.diff(rank[mine]) > 0).all()


def test_block_order_refuses_more_than_a_block_keeps():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert block_order(np.zeros(sms * WALK_CELLS_MAX + 1, np.int32), torch.device("cuda")) is None
