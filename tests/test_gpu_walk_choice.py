"""The rule that takes a walk to blocks: the mean number of chunks that a level
has on its busiest block, against a count by numpy over the same levels, and
both walks, bit for bit, whichever the rule takes."""

import numpy as np
import pytest
import torch

from pyopenfoam_gb300.core.topology import WALK_CELLS_MIN, WALK_SHARE_MAX, WALK_SHARE_MAX_WIDE
from pyopenfoam_gb300.solvers import smoothers
from pyopenfoam_gb300.solvers.preconditioners import factor_dic
from tests.test_gpu_block_walk import bits, matrix

pytestmark = pytest.mark.gpu


def share_of(ptr, cells, per):
    share, every = [], max(1, min(cells.shape[0] // 65536, (ptr.shape[0] - 1) // 64))
    for a, b in list(zip(ptr[:-1], ptr[1:]))[every // 2::every]:
        share.append(np.ceil(np.bincount(cells[a:b] // per) / 32).max())
    return float(np.mean(share))


@pytest.mark.parametrize("dims,kind,pays", [
    ((1, 1, 1), "mesh", True), ((513, 1, 1), "mesh", True), ((33, 31, 5), "renumbered", True),
    ((40, 40, 40), "renumbered", True),
    ((67, 59, 53), "mesh", True), ((67, 59, 53), "renumbered", False),
    ((100, 100, 100), "mesh", True), ((100, 100, 100), "renumbered", False),
    ((128, 128, 128), "mesh", False), ((97, 83, 61), "shuffled", True)])
def test_share_and_choice(dims, kind, pays):
    m, _ = matrix(dims, kind)
    topo = m.topology()
    limit = WALK_SHARE_MAX if topo.max_width <= 8 else WALK_SHARE_MAX_WIDE
    sch, gs = topo.dic_schedule(), smoothers._gs_schedule(m, True)
    for order, ptr, cells in ((topo.dic_blocks(), sch.ptr, sch.items),
                              (gs.blocks, gs.ptr, gs.cells)):
        want = share_of(ptr.cpu().numpy(), cells.cpu().numpy(), order.per)
        assert order.per == WALK_CELLS_MIN or order.share == pytest.approx(want, rel=1e-12)
        assert order.pays == pays == (order.per == WALK_CELLS_MIN or want <= limit)


@pytest.mark.parametrize("kind", ["mesh", "renumbered", "shuffled"])
@pytest.mark.parametrize("dims", [(40, 30, 29), (97, 83, 61)])
def test_both_walks_whatever_the_rule(dims, kind):
    m, b = matrix(dims, kind)
    topo, out = m.topology(), []
    orders = [topo.dic_blocks()] + [smoothers._gs_schedule(m, r).blocks for r in (False, True)]
    for pays in (True, False):
        for o in orders:
            o.pays = pays
        d = torch.empty(m.n_cells, dtype=torch.float64, device="cuda")
        factor_dic(topo, m.packed(), m.diag, d, m.device, "flow")
        out.append([d])
        for reverse in (False, True):
            x = torch.linspace(-1, 1, m.n_cells, dtype=torch.float64, device="cuda")
            smoothers.gs_sweep(m, x, b, reverse=reverse, omega=0.9, relax=True, form="flow")
            out[-1].append(x)
    assert all(torch.equal(bits(p), bits(q)) for p, q in zip(*out))
