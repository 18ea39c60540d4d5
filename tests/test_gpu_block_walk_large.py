"""Block walks whose blocks keep more than 48 KB of cells in shared memory (the
launch then depends on the raised limit), up to nearly all that a block may
keep, against one launch per level, bit for bit."""

import pytest
import torch

from pyopenfoam_gb300.core.topology import WALK_CELLS_MAX
from pyopenfoam_gb300.solvers.preconditioners import factor_dic
from pyopenfoam_gb300.solvers.smoothers import gs_sweep
from tests.test_gpu_block_walk import bits, matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,kind", [((100, 99, 98), "mesh"), ((100, 99, 98), "renumbered"),
                                       ((155, 152, 150), "mesh")])
def test_walks_of_large_blocks(dims, kind):
    m, b = matrix(dims, kind)
    blocks = m.topology().dic_blocks()
    assert 8 * blocks.per > 48 * 1024 and blocks.per <= WALK_CELLS_MAX
    out = []
    for form in ("per_level", "flow"):
        d = torch.empty(m.n_cells, dtype=torch.float64, device="cuda")
        factor_dic(m.topology(), m.packed(), m.diag, d, m.device, form)
        out.append([d])
        for reverse in (False, True):
            x = torch.linspace(-1, 1, m.n_cells, dtype=torch.float64, device="cuda")
            gs_sweep(m, x, b, reverse=reverse, omega=0.8, relax=True, form=form)
            out[-1].append(x)
    assert all(torch.equal(bits(a), bits(c)) for a, c in zip(*out))
