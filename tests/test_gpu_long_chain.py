"""Block walks over the longest chain they take, one cell a level: every block
waits for all before it, far longer than any poll count of a short wait.  The
DIC factor and the Gauss-Seidel sweep against the same recurrences in plain
float64."""

import numpy as np
import pytest
import torch

from pyopenfoam_gb300 import LduMatrix
from pyopenfoam_gb300.solvers.preconditioners import factor_dic
from pyopenfoam_gb300.solvers.smoothers import gs_sweep

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def chain():
    n = 23000 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(8)
    c = rng.lognormal(0.0, 0.3, n - 1)
    diag = rng.uniform(0.1, 0.5, n)
    diag[:-1] += c
    diag[1:] += c
    own = torch.arange(n - 1)
    m = LduMatrix(n, own, own + 1, device="cuda")
    m.diag, m.lower, m.upper = (torch.as_tensor(a) for a in (diag, -c, -0.8 * c))
    return m, diag, -c, -0.8 * c, rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)


def test_dic_of_a_chain(chain):
    m, diag, _, up, _, _ = chain
    assert m.topology().dic_blocks() is not None
    d = torch.empty(m.n_cells, dtype=torch.float64, device="cuda")
    factor_dic(m.topology(), m.packed(), m.diag, d, m.device, "flow")
    want, last = diag.tolist(), diag[0]
    for c, (v, a) in enumerate(zip(diag[1:].tolist(), up.tolist()), 1):
        last = want[c] = v - (a * a) / last
    assert np.array_equal(d.cpu().numpy(), np.asarray(want))


def test_gauss_seidel_sweep_of_a_chain(chain):
    m, diag, lo, up, b, x0 = chain
    x = torch.as_tensor(x0).cuda()
    gs_sweep(m, x, torch.as_tensor(b).cuda(), form="flow")
    dx = (diag * x0).tolist()
    right = np.append(lo * x0[1:], 0.0).tolist()  # the last cell has no such face
    want, prev, n = [], 0.0, m.n_cells
    ups = [0.0] + up.tolist()
    for c, (d, bc) in enumerate(zip(diag.tolist(), b.tolist())):
        row = dx[c]
        if c > 0:
            row += ups[c] * prev
        if c < n - 1:
            row += right[c]
        prev = (bc - (row - dx[c])) / d
        want.append(prev)
    assert np.array_equal(x.cpu().numpy(), np.asarray(want))
