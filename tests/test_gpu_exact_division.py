"""The integer-pipe product, division and square root (csrc/exact.cuh) against numpy's IEEE
operations, bit for bit, through the operators that divide and take roots
directly: compute_HbyA (H / max(|A|, 1e-30)) and fvm.laplacian's lower
coefficient on unit volumes and deltas (-|S_f|)."""

import numpy as np
import pytest
import torch

from pyopenfoam_gb300.discretisation import fvm
from pyopenfoam_gb300.solvers.rhie_chow import compute_face_flux_HbyA, compute_HbyA

pytestmark = pytest.mark.gpu
N = 1 << 16


def bits(a):
    return np.ascontiguousarray(a, np.float64).view(np.int64)


def same(a, b):
    """Equal bits, any NaN equal to any NaN."""
    return bool(((bits(a) == bits(b)) | (np.isnan(a) & np.isnan(b))).all())


def mantissas(rng, n):
    """Doubles in [1, 2): random, and with long runs of zeros or ones at either end."""
    m = rng.integers(0, 1 << 52, n, dtype=np.int64)
    k = rng.integers(0, 6, n)
    low = (1 << rng.integers(0, 52, n)) - 1
    m = np.where(k == 1, m & low, np.where(k == 2, m | low, np.where(k == 3, m & ~low, m)))
    return (m + (1023 << 52)).view(np.float64)


def pairs(kind, rng):
    if kind == "random":
        return (mantissas(rng, N) * np.exp2(rng.integers(-90, 90, N)) * rng.choice([-1.0, 1.0], N),
                mantissas(rng, N) * np.exp2(rng.integers(-90, 90, N)))
    if kind == "near_midpoint":  # a = the doubles around (2 q + 1) b / 2, q a 53-bit quotient
        b, q = mantissas(rng, 4096), mantissas(rng, 4096)
        a = []
        for bi, qi in zip(bits(b) & ((1 << 52) - 1), bits(q) & ((1 << 52) - 1)):
            p = (2 * (int(qi) + (1 << 52)) + 1) * (int(bi) + (1 << 52))
            a.append(float((p >> (p.bit_length() - 53)) + int(rng.integers(-1, 2))))
        return np.array(a), b
    if kind == "exact_and_close":
        b = mantissas(rng, N)
        step = rng.integers(-4, 5, N)
        return np.where(rng.random(N) < 0.5, b * mantissas(rng, N).astype(np.float32),
                        (bits(b) + step).view(np.float64)), b
    a = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.2e-308, 2.3e-308, 1.8e308, 1e-300,
                  1e300, 1.0])
    b = np.array([1e-30, 1.0, 3.0, 1e300, 1.7e308, np.inf, 7e-30, 2.0 ** 600])
    return [v.ravel().copy() for v in np.meshgrid(a, b)]


@pytest.mark.parametrize("kind", ["random", "near_midpoint", "exact_and_close", "special"])
def test_division_is_ieee(kind):
    a, b = pairs(kind, np.random.default_rng(7))
    n = a.shape[0]
    H = torch.as_tensor(np.stack([a, -a, a], 1)).cuda()
    got = compute_HbyA(H, torch.as_tensor(-b).cuda()).cpu().numpy()
    with np.errstate(all="ignore"):
        want = a / np.maximum(b, 1e-30)
    assert got.shape == (n, 3)
    assert same(got[:, 0], want) and same(got[:, 1], -want) and same(got[:, 2], want)


class _Faces:
    """Mesh of unit volumes and deltas whose internal faces carry given area vectors."""

    def __init__(self, areas):
        nf = areas.shape[0]
        self.n_cells, self.n_faces, self.n_internal_faces = nf + 1, nf, nf
        self.owner = torch.arange(nf).cuda()
        self.neighbour = self.owner + 1
        self.face_areas = torch.as_tensor(areas).cuda()
        self.delta_coefficients = torch.ones(nf, dtype=torch.float64).cuda()
        self.cell_volumes = torch.ones(nf + 1, dtype=torch.float64).cuda()
        self.device, self.dtype = torch.device("cuda"), torch.float64


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("scale", [-510, -30, 0, 40, 500])
def test_square_root_is_ieee(scale, odd):
    rng = np.random.default_rng(1000 + scale + 5000 * odd)
    # x^2 is rounded once and y^2 = 4^k exactly, so numpy's x * x + y * y has the operator's bits
    x = mantissas(rng, N) * 2.0 ** scale * np.sqrt(2.0) ** odd
    y = np.exp2(scale + rng.integers(-30, 2, N)) * (rng.random(N) < 0.7)
    A = fvm.laplacian(1.0, torch.zeros(1), mesh=_Faces(np.stack([x, y, np.zeros(N)], 1)))
    with np.errstate(all="ignore"):
        want = -np.sqrt(x * x + y * y)
    assert same(A.lower.cpu().numpy(), want) and same(A.upper.cpu().numpy(), want)


@pytest.mark.parametrize("kind", ["random", "near_midpoint", "exact_and_close", "special"])
def test_product_is_ieee(kind):
    """The integer-pipe product, through compute_face_flux_HbyA: the flux of a boundary face with
    area (s, 0, 0) is h s (+ 0 + 0); of an internal one with weight 1, (1 h + 0 h') s."""
    a, b = pairs(kind, np.random.default_rng(9))
    n = a.shape[0]
    H = torch.as_tensor(np.stack([np.concatenate([a, [1.0]])] + [np.ones(n + 1)] * 2, 1)).cuda()
    S = torch.as_tensor(np.stack([b, np.zeros(n), np.zeros(n)], 1)).cuda()
    own = torch.arange(n).cuda()
    with np.errstate(all="ignore"):
        want = a * b + 0.0
        inner = (1.0 * a + 0.0 * np.concatenate([a[1:], [1.0]])) * b + 0.0
    got = compute_face_flux_HbyA(H, S, own, own + 1, n, torch.ones(n, dtype=torch.float64).cuda())
    assert same(got.cpu().numpy(), inner)
    got = compute_face_flux_HbyA(H, S, own, own[:0], 0)
    assert same(got.cpu().numpy(), want)
