"""Workloads of the linear-solve path at the sizes and options it is used with.

Twelve listed cases, one per call a flow solver makes in a time step (and the
mesh set-up before the first one), from a few thousand cells to the 256^3
headline system; ``draw`` gives more of the same with other sizes, shapes,
numberings and options.

* ``prepare(case, seed)`` -- what the program holds before the call: mesh,
  matrix object with its addressing, coefficients, fields.
* ``run(state)`` -- one call through the public entry points, all its outputs.
* ``work(case)`` -- bytes (each input read once, each output written once; the
  vectors of an iterative solve once per iteration) and operations.
* ``exact(case, seed)`` -- the outputs in 64-bit plain torch where they have a
  closed form or a known solution.

Solves set the matrix coefficients anew in every pass, as a time step does, so
packing and factorisation are part of the call.
"""

from __future__ import annotations

import math

import torch

from pyopenfoam_gb300 import (LduMatrix, MixedPrecisionPBiCGSTABSolver, MixedPrecisionPCGSolver,
                              PBiCGSTABSolver, PCGSolver)
from pyopenfoam_gb300.differentiable.unrolled import UnrolledDiffusion, UnrolledImplicitDiffusion
from pyopenfoam_gb300.discretisation import fvm
from pyopenfoam_gb300.mesh import FvMesh, HexMesh, PolyMesh
from pyopenfoam_gb300.solvers import (BatchedPCGSolver, GAMGSolver, SmoothSolver,
                                      assemble_pressure_equation, correct_face_flux,
                                      correct_velocity)
from pyopenfoam_gb300.solvers.rhie_chow import compute_face_flux

DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(op, nx, ny, nz, **kw):
    return dict(op=op, nx=nx, ny=ny, nz=nz, **kw)


def listed():
    return [
        # a residual evaluation on a small mesh: latency of one product and its transpose
        _case("amul", 23, 17, 11, name="amul_small", dtype="float64", renumber=False),
        # implicit momentum operator on an ordinary mesh: upwind convection + diffusion with a
        # per-cell (turbulent) viscosity
        _case("momentum_assembly", 96, 81, 64, name="momentum_assembly", d="cell"),
        # everything around the pressure solve of one corrector step, on a large mesh
        _case("pressure_step", 128, 128, 128, name="pressure_step"),
        # reading in a mesh: addressing and geometry of a polyhedral mesh
        _case("mesh_setup", 64, 48, 40, name="mesh_setup"),
        # FP64 PCG + DIC to 1e-6 on 32^3: the small solve of every corrector
        _case("pcg", 32, 32, 32, name="pcg_f64_32", solver="f64", rel_tol=1e-6, sigma=0.0,
              renumber=False),
        # the headline: mixed-precision PCG + DIC to 1e-10 on the 256^3 Poisson system
        _case("pcg", 256, 256, 256, name="pcg_mixed_256", solver="mixed", rel_tol=1e-10, sigma=0.0,
              renumber=False),
        # momentum solve on a mesh whose cells are numbered in no useful order
        _case("bicgstab", 72, 60, 50, name="bicgstab_f64_unordered", solver="f64", rel_tol=1e-8,
              renumber=True),
        # mixed-precision momentum solve on 128^3, cell Peclet number 10, to 1e-8
        _case("bicgstab", 128, 128, 128, name="bicgstab_mixed_128", solver="mixed", rel_tol=1e-8,
              renumber=False),
        # many independent systems of uneven size in one call (parameter sweeps, training sets)
        _case("batched", 16, 48, 24, name="batched_24", rel_tol=1e-8),
        # multigrid solve of an implicit diffusion (transient pressure) system
        _case("gamg", 64, 64, 64, name="gamg_64", rel_tol=1e-6),
        # Gauss-Seidel smoothing solve of a momentum system, odd sizes
        _case("smooth", 67, 59, 53, name="smooth_gs", smoother="GaussSeidel", rel_tol=1e-5),
        # gradient of a short unrolled diffusion with respect to every face diffusivity
        _case("adjoint", 48, 40, 36, name="adjoint_48", steps=4, every=2),
    ]


# range of cells of each call; the product also takes FP32 matrices
_CELLS = {"amul": (2e3, 1.2e7), "momentum_assembly": (8e3, 4e6), "pressure_step": (8e3, 4e6),
          "mesh_setup": (4e3, 3e5), "pcg": (8e3, 6e6), "bicgstab": (8e3, 2.1e6),
          "gamg": (4e3, 3e5), "smooth": (4e3, 5e5), "adjoint": (8e3, 2e5)}


def draw(rng):
    op = rng.choice(sorted(_CELLS) + ["batched"])
    if op == "batched":
        lo = rng.randint(8, 24)
        return _case(op, lo, rng.randint(lo + 8, 64), rng.randint(6, 40), rel_tol=1e-8)
    a, b = _CELLS[op]
    n = math.exp(rng.uniform(math.log(a), math.log(b)))
    sx, sy = math.exp(rng.uniform(-0.4, 0.4)), math.exp(rng.uniform(-0.4, 0.4))
    h = n ** (1.0 / 3.0)
    nx, ny = max(6, round(h * sx)), max(6, round(h * sy))
    nz = max(6, round(n / (nx * ny)))
    kw = {}
    if op == "amul":
        kw = dict(dtype=rng.choice(["float64", "float64", "float32"]),
                  renumber=rng.random() < 0.4)
    elif op == "momentum_assembly":
        kw = dict(d=rng.choice(["cell", "face", "constant"]))
    elif op == "pcg":
        kw = dict(solver=rng.choice(["f64", "mixed"]), rel_tol=rng.choice([1e-6, 1e-8]),
                  sigma=rng.choice([0.0, 0.5]), renumber=rng.random() < 0.3)
    elif op == "bicgstab":
        kw = dict(solver=rng.choice(["f64", "mixed"]), rel_tol=1e-8,
                  renumber=rng.random() < 0.4)
    elif op == "gamg":
        kw = dict(rel_tol=1e-6)
    elif op == "smooth":
        kw = dict(smoother=rng.choice(["GaussSeidel", "DILU"]), rel_tol=1e-5)
    elif op == "adjoint":
        kw = dict(steps=rng.randint(2, 6), every=2)
    return _case(op, nx, ny, nz, **kw)


# ---------------------------------------------------------------------------
# meshes and systems, in plain torch
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _uniform(g, n, lo=-1.0, hi=1.0):
    return torch.rand(n, generator=g, device=DEV, dtype=F64) * (hi - lo) + lo


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _hex_faces(nx, ny, nz):
    """Owner, neighbour and direction of the internal faces, per cell +x, +y, +z."""
    n = nx * ny * nz
    c = torch.arange(n, device=DEV)
    has = torch.stack([c % nx < nx - 1, (c // nx) % ny < ny - 1, c // (nx * ny) < nz - 1], 1)
    flat = has.reshape(-1).nonzero().squeeze(1)
    own, d = flat // 3, flat % 3
    return n, own, own + torch.tensor([1, nx, nx * ny], device=DEV)[d], d


class _Stencil:
    """Seven-point system on an nx * ny * nz grid: ``lo[c, d]`` multiplies the +d neighbour in
    row c, ``up[c, d]`` multiplies c in that neighbour's row.  Sums run over shifted arrays, so
    that the same seed gives the same bits."""

    def __init__(self, case):
        self.nx, self.ny, self.nz = nx, ny, nz = case["nx"], case["ny"], case["nz"]
        self.n = nx * ny * nz
        self.step = (1, nx, nx * ny)
        c = torch.arange(self.n, device=DEV)
        self.i, self.j, self.k = c % nx, (c // nx) % ny, c // (nx * ny)
        self.has = torch.stack([self.i < nx - 1, self.j < ny - 1, self.k < nz - 1], 1)

    def to_neighbour(self, v):
        out = torch.zeros(self.n, device=DEV, dtype=F64)
        for d, st in enumerate(self.step):
            if st < self.n:
                out[st:] += v[: self.n - st, d]
        return out

    def product(self, x):
        y = self.diag * x
        for d, st in enumerate(self.step):
            if st < self.n:
                y[: self.n - st] += self.lo[: self.n - st, d] * x[st:]
        return y + self.to_neighbour(self.up * x[:, None])

    def field(self, g):
        """A smooth field plus a little noise: the solution the systems are given."""
        x, y, z = (self.i + 0.5) / self.nx, (self.j + 0.5) / self.ny, (self.k + 0.5) / self.nz
        a = _normal(g, 3)
        f = (torch.sin(math.pi * x / 2) * (2.0 + a[0] * torch.cos(math.pi * y))
             + a[1] * torch.cos(2 * math.pi * z) * torch.sin(math.pi * x) + 0.3 * a[2] * y * z)
        return (f + 0.02 * _normal(g, self.n)).to(F64)


def _poisson(case, g):
    """Diffusion system per unit volume on the unit cube, fixed value on x = 0 (and, with
    ``time``, an implicit time term): face diffusivity LogNormal(0, sigma)."""
    t = _Stencil(case)
    N = torch.tensor([t.nx, t.ny, t.nz], device=DEV, dtype=F64)
    c = (N * N) * t.has
    if case.get("sigma"):
        c = c * torch.exp(case["sigma"] * _normal(g, t.n, 3))
    t.lo = t.up = -c
    t.diag = c.sum(1) + t.to_neighbour(c) + 2.0 * N[0] * N[0] * (t.i == 0)
    t.diag += case.get("time", 0.0) * (N * N).max()
    return t


def _momentum(case, g):
    """Upwind convection-diffusion system: face diffusion LogNormal(0, 1), cell Peclet number
    about 10, fixed value on x = 0, outflow on the far faces, implicit time term ``time``."""
    t = _Stencil(case)
    D = torch.exp(_normal(g, t.n, 3)) * t.has
    F = 10.0 * torch.tensor([1.0, 0.5, 0.25], device=DEV, dtype=F64) * t.has
    t.lo, t.up = -D, -D - F
    t.diag = (D + F).sum(1) + t.to_neighbour(D) + 2.0 * (t.i == 0) + 10.0 * (t.i == t.nx - 1)
    t.diag += 5.0 * (t.j == t.ny - 1) + 2.5 * (t.k == t.nz - 1) + case.get("time", 0.0)
    return t


def _arrays(case, t, g, **vectors):
    """The system's LDU arrays and cell vectors, faces in upper-triangular order; with
    ``renumber`` under a random cell numbering."""
    flat = t.has.reshape(-1).nonzero().squeeze(1)
    own, d = flat // 3, flat % 3
    nei = own + torch.tensor(t.step, device=DEV)[d]
    lo, up = t.lo.reshape(-1)[flat], t.up.reshape(-1)[flat]
    vectors = dict(vectors, diag=t.diag)
    if case.get("renumber"):
        p = torch.randperm(t.n, generator=g, device=DEV)
        a, b = p[own], p[nei]
        lo, up = torch.where(a < b, lo, up), torch.where(a < b, up, lo)
        own, nei = torch.minimum(a, b), torch.maximum(a, b)
        order = torch.argsort(own * t.n + nei)
        own, nei, lo, up = own[order], nei[order], lo[order], up[order]
        inverse = torch.argsort(p)
        vectors = {k: None if v is None else v[inverse] for k, v in vectors.items()}
    return dict(n=t.n, owner=own.contiguous(), neighbour=nei.contiguous(), lower=lo.contiguous(),
                upper=up.contiguous(), **vectors)


def _sum_faces(n, own, nei, to_own, to_nei):
    return torch.zeros(n, device=DEV, dtype=F64).index_add_(0, own, to_own).index_add_(0, nei,
                                                                                       to_nei)


def _product(s, x, transposed=False):
    lo, up = (s["upper"], s["lower"]) if transposed else (s["lower"], s["upper"])
    y = s["diag"].double() * x
    y.index_add_(0, s["owner"], lo.double() * x[s["neighbour"]])
    return y.index_add_(0, s["neighbour"], up.double() * x[s["owner"]])


def _matrix(s, dtype=F64):
    m = LduMatrix(s["n"], s["owner"], s["neighbour"], device=DEV, dtype=dtype)
    m.diag, m.lower, m.upper = s["diag"], s["lower"], s["upper"]
    m.topology()
    return m


def _system(case, seed):
    """The arrays of one solve and its known solution ``x`` (None on the headline system, whose
    right-hand side is random; elsewhere it is the product with a known field)."""
    op, g = case["op"], _gen(seed)
    if op in ("pcg", "gamg"):
        t = _poisson(dict(case, time=0.05 if op == "gamg" else 0.0), g)
    else:
        t = _momentum(dict(case, time=60.0 if op == "smooth" else 0.0), g)
    if op == "pcg" and case["rel_tol"] < 1e-9:
        return _arrays(case, t, g, x=None, b=_uniform(g, t.n))
    x = t.field(g)
    return _arrays(case, t, g, x=x, b=t.product(x))


def _polymesh(case, seed):
    """Points (interior jittered by 20 % of the spacing), face quads and owner / neighbour of a
    hex mesh of the unit cube."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = _gen(seed)
    n, own, nei, d = _hex_faces(nx, ny, nz)
    gz, gy, gx = torch.meshgrid(*(torch.linspace(0, 1, k + 1, device=DEV, dtype=F64)
                                  for k in (nz, ny, nx)), indexing="ij")
    pts = torch.stack([gx, gy, gz], 3)
    h = torch.tensor([1.0 / nx, 1.0 / ny, 1.0 / nz], device=DEV, dtype=F64)
    r = torch.rand(pts.shape, generator=g, device=DEV, dtype=F64)
    pts[1:-1, 1:-1, 1:-1] += (0.4 * (r - 0.5) * h)[1:-1, 1:-1, 1:-1]
    sx, sy, sz = 1, nx + 1, (nx + 1) * (ny + 1)

    def quads(cell, k, plane):
        """Vertices of the face of ``cell`` normal to axis k at its low (0) or high (1) side,
        counter-clockwise about +k."""
        p = cell % nx + (cell // nx) % ny * sy + cell // (nx * ny) * sz
        st = torch.tensor([[sx, sy, sz], [sy, sz, sx], [sz, sx, sy]], device=DEV)[k]
        e0, e1, e2 = st.unbind(-1)
        p = p + e0 * plane
        return torch.stack([p, p + e1, p + e1 + e2, p + e2], -1)

    faces, owner = [quads(own, d, 1)], [own]
    c = torch.arange(n, device=DEV)
    ijk = (c % nx, (c // nx) % ny, c // (nx * ny))
    for k, size in enumerate((nx, ny, nz)):
        for plane in (0, 1):
            cells = c[ijk[k] == (size - 1 if plane else 0)]
            q = quads(cells, torch.full_like(cells, k), plane)
            faces.append(q if plane else q.flip(-1))
            owner.append(cells)
    return dict(n=n, points=pts.reshape(-1, 3), faces=torch.cat(faces), owner=torch.cat(owner),
                neighbour=nei, g=g)


def _poly(pm):
    nf = pm["faces"].shape[0]
    ptr = torch.arange(0, 4 * nf + 1, 4).numpy()
    return PolyMesh(pm["points"], (ptr, pm["faces"].reshape(-1).cpu().numpy()),
                    pm["owner"].cpu().numpy(), pm["neighbour"].cpu().numpy(), device=DEV)


def _mesh_fields(case, pm, mesh_n, nf):
    """Face flux, viscosity / diffusivity, pressure, 1/A_p source and HbyA on a mesh."""
    g = pm["g"]
    op = case["op"]
    if op == "momentum_assembly":
        kind = case["d"]
        D = (0.75 if kind == "constant" else
             torch.exp(_normal(g, mesh_n if kind == "cell" else nf)))
        return dict(phi=_normal(g, nf), D=D)
    return dict(H=_normal(g, mesh_n, 3), p=_uniform(g, mesh_n), A=_uniform(g, mesh_n, 0.5, 3.0))


def _batch_sides(case):
    g = torch.Generator()
    g.manual_seed(3)
    return torch.randint(case["nx"], case["ny"] + 1, (case["nz"],), generator=g).tolist()


def _batch(case, seed):
    """nz systems with sides drawn from nx..ny, face diffusivity LogNormal(0, 0.5)."""
    return [_system(dict(op="pcg", nx=N, ny=N, nz=N, sigma=0.5, rel_tol=case["rel_tol"]),
                    64 * int(seed) + k) for k, N in enumerate(_batch_sides(case))]


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    op = case["op"]
    if op == "amul":
        dt = getattr(torch, case["dtype"])
        s = _system(case, seed)
        return dict(op=op, m=_matrix(s, dt), x=s["x"].to(dt))
    if op in ("momentum_assembly", "pressure_step", "mesh_setup"):
        pm = _polymesh(case, seed)
        poly = _poly(pm)
        if op == "mesh_setup":
            return dict(op=op, poly=poly)
        mesh = FvMesh.from_poly_mesh(poly)
        mesh.compute_geometry()
        f = _mesh_fields(case, pm, pm["n"], mesh.n_faces)
        return dict(op=op, mesh=mesh, U=torch.zeros(pm["n"], 3, device=DEV, dtype=F64), **f)
    if op == "batched":
        ss = _batch(case, seed)
        return dict(op=op, m=[_matrix(s) for s in ss], b=[s["b"] for s in ss],
                    solver=BatchedPCGSolver(tolerance=0.0, rel_tol=case["rel_tol"], max_iter=20000,
                                            form="graph", block_size=256, tile_cells=1024,
                                            wavefront="flow", threads_per_cell=1))
    if op == "adjoint":
        mesh = HexMesh(case["nx"], case["ny"], case["nz"], device=DEV)
        g = _gen(seed)
        model = UnrolledImplicitDiffusion(mesh, dt=1e-3, steps=case["steps"],
                                          checkpoint_every=case["every"])
        return dict(op=op, model=model, gamma=torch.exp(_normal(g, mesh.n_faces)),
                    x0=_uniform(g, mesh.n_cells), w=_uniform(g, mesh.n_cells))
    s = _system(case, seed)
    tol = dict(tolerance=0.0, rel_tol=case["rel_tol"])
    if op == "pcg":
        solver = (PCGSolver if case["solver"] == "f64" else MixedPrecisionPCGSolver)(
            max_iter=20000, preconditioner="DIC", **tol)
    elif op == "bicgstab":
        solver = (PBiCGSTABSolver if case["solver"] == "f64" else MixedPrecisionPBiCGSTABSolver)(
            max_iter=5000, preconditioner="DILU", omega="standard", **tol)
    elif op == "gamg":
        solver = GAMGSolver(max_iter=200, **tol)
    else:
        solver = SmoothSolver(max_iter=200, smoother=case["smoother"], n_sweeps=2, **tol)
    return dict(op=op, m=_matrix(s), diag=s["diag"], lower=s["lower"], upper=s["upper"], b=s["b"],
                x0=torch.zeros_like(s["b"]), solver=solver)


def run(s):
    op = s["op"]
    if op == "amul":
        return [s["m"].Ax(s["x"]), s["m"].Ax_T(s["x"])]
    if op == "momentum_assembly":
        conv = fvm.div(s["phi"], s["U"], "Gauss upwind", mesh=s["mesh"])
        lap = fvm.laplacian(s["D"], s["U"], mesh=s["mesh"])
        return [conv.lower, conv.upper, conv.diag, lap.lower, lap.upper, lap.diag]
    if op == "pressure_step":
        m = s["mesh"]
        phi = compute_face_flux(s["H"], s["p"], s["A"], m.face_areas, m.delta_coefficients,
                                m.owner, m.neighbour, m.n_internal_faces, m.cell_volumes,
                                m.face_weights)
        eqn = assemble_pressure_equation(phi, s["A"], m)
        phi2 = correct_face_flux(phi, s["p"], s["A"], m)
        U = correct_velocity(s["U"], s["H"], s["p"], s["A"], m)
        return [phi, eqn.lower, eqn.upper, eqn.diag, eqn.source, phi2, U]
    if op == "mesh_setup":
        m = FvMesh.from_poly_mesh(s["poly"])
        m.compute_geometry()
        return [m.face_centres, m.face_areas, m.cell_volumes, m.cell_centres, m.face_weights,
                m.delta_coefficients]
    if op == "batched":
        return [x for x, _, _ in s["solver"].solve(s["m"], s["b"])]
    if op == "adjoint":
        gamma = s["gamma"].detach().requires_grad_(True)
        x0 = s["x0"].detach().requires_grad_(True)
        xT = UnrolledDiffusion.apply(gamma, x0, s["model"])
        xT.backward(s["w"])
        return [xT.detach(), gamma.grad, x0.grad]
    m = s["m"]
    m.diag, m.lower, m.upper = s["diag"], s["lower"], s["upper"]
    x, iterations, _ = s["solver"](m, s["b"], s["x0"])
    return [x, iterations]


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _sizes(nx, ny, nz):
    n = nx * ny * nz
    ni = 3 * n - nx * ny - ny * nz - nx * nz
    return n, ni, ni + 2 * (nx * ny + ny * nz + nx * nz)


def work(case):
    op, nx, ny, nz = case["op"], case["nx"], case["ny"], case["nz"]
    if op == "batched":
        b = f = 0.0
        for N in _batch_sides(case):
            n, ni, _ = _sizes(N, N, N)
            its = 8 * N  # about what these systems take to 1e-8
            b += its * (8.0 * ni + 44.0 * n) + 24.0 * ni + 24.0 * n
            f += its * (4.0 * ni + 13.0 * n)
        return dict(bytes=b, flops=f)
    n, ni, nf = _sizes(nx, ny, nz)
    if op == "amul":
        w = 8 if case["dtype"] == "float64" else 4
        return dict(bytes=2.0 * (w * (2 * ni + 2 * n) + 8 * n), flops=2.0 * (4 * ni + n))
    if op == "momentum_assembly":
        # flux, volumes and addressing in, three coefficient arrays out; the Laplacian also
        # reads areas, deltas, weights and the diffusivity
        d = {"cell": 8 * n + 8 * ni, "face": 8 * nf, "constant": 0}[case["d"]]
        return dict(bytes=2.0 * (8 * ni + 8 * n + 16 * ni + 8 * n) + 8 * ni + 32 * nf + d,
                    flops=6.0 * ni + 16.0 * ni)
    if op == "pressure_step":
        flux = nf * (8 + 24 + 8 + 8 + 8) + n * 40
        asm = nf * (8 + 24 + 8 + 8 + 8) + 16 * ni + n * 32
        corr = nf * (8 + 24 + 8 + 8 + 16) + n * 16
        vel = nf * (8 + 24 + 8) + n * 72
        return dict(bytes=float(flux + asm + corr + vel), flops=100.0 * nf + 40.0 * n)
    if op == "mesh_setup":
        return dict(bytes=float(4 * nf * 4 + 4 * (nf + ni) + 24 * n + 48 * nf + 32 * n + 16 * nf),
                    flops=1000.0 * n + 120.0 * nf)
    size = max(nx, ny, nz)
    if op == "adjoint":
        its = case["steps"] * 2.4 * 60
        return dict(bytes=its * (16.0 * ni + 88.0 * n), flops=its * (4.0 * ni + 14.0 * n))
    digits = -math.log10(case["rel_tol"])
    if op == "pcg":
        its = 0.83 * digits * size
        v = 4 if case["solver"] == "mixed" else 8
        return dict(bytes=its * v * (2.0 * ni + 11.0 * n), flops=its * (4.0 * ni + 14.0 * n))
    if op == "bicgstab":
        its = 0.4 * digits * size
        v = 4 if case["solver"] == "mixed" else 8
        return dict(bytes=its * v * (4.0 * ni + 20.0 * n), flops=its * (8.0 * ni + 24.0 * n))
    if op == "gamg":
        its = 10.0  # V-cycles of about six products on twice the fine level's cells
        return dict(bytes=its * 12 * 8 * (2.0 * ni + 4.0 * n), flops=its * 12 * (4.0 * ni + n))
    its = 2.0 * digits  # sweeps and a residual per check
    return dict(bytes=its * 3 * 8 * (2.0 * ni + 4.0 * n), flops=its * 3 * (4.0 * ni + 2.0 * n))


# ---------------------------------------------------------------------------
# the outputs in 64-bit plain torch
# ---------------------------------------------------------------------------
def _cross(a, b):
    return torch.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1],
                        a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                        a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def _geometry(pm):
    """Face centres (vertex mean) and area vectors, cell volumes and centres (tetrahedra of the
    vertex mean, each face centre and each edge), weights and delta coefficients."""
    own, nei, n = pm["owner"], pm["neighbour"], pm["n"]
    ni = nei.shape[0]
    v = pm["points"][pm["faces"]]
    w = torch.roll(v, -1, 1)
    fc = v.mean(1)
    S = 0.5 * _cross(v, w).sum(1)
    corners = torch.zeros(n, 3, device=DEV, dtype=F64)
    for cells, fs in ((own, slice(0, None)), (nei, slice(0, ni))):
        corners.index_add_(0, cells, v[fs].sum(1))
    ref = corners / 24.0  # a hex counts each corner three times
    vol = torch.zeros(n, device=DEV, dtype=F64)
    mom = torch.zeros(n, 3, device=DEV, dtype=F64)
    for cells, fs in ((own, slice(0, None)), (nei, slice(0, ni))):
        r = ref[cells][:, None, :]
        t = ((fc[fs][:, None, :] - r) * _cross(v[fs] - r, w[fs] - r)).sum(-1).abs() / 6.0
        cen = (r + fc[fs][:, None, :] + v[fs] + w[fs]) / 4.0
        vol.index_add_(0, cells, t.sum(1))
        mom.index_add_(0, cells, (t[..., None] * cen).sum(1))
    cc = mom / vol[:, None]
    wt = torch.ones(own.shape[0], device=DEV, dtype=F64)
    dl = torch.zeros_like(wt)
    P, N = own[:ni], nei
    dP, dN = (fc[:ni] - cc[P]).norm(dim=1), (fc[:ni] - cc[N]).norm(dim=1)
    wt[:ni] = dN / (dP + dN)
    dl[:ni] = 1.0 / ((cc[N] - cc[P]) * S[:ni] / S[:ni].norm(dim=1, keepdim=True)).sum(1).abs()
    return fc, S, vol, cc, wt, dl


def _cg(A, b, tol=1e-15, most=4000):
    """Plain conjugate gradients with Jacobi scaling on the symmetric system ``A``."""
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / A["diag"]
    p, rz, stop = z.clone(), torch.dot(r, z), tol * float(b.norm())
    for _ in range(most):
        Ap = _product(A, p)
        a = rz / torch.dot(p, Ap)
        x += a * p
        r -= a * Ap
        if float(r.norm()) < stop:
            break
        z = r / A["diag"]
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return x


def _exact_adjoint(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n, own, nei, d = _hex_faces(nx, ny, nz)
    ni, nf = own.shape[0], _sizes(nx, ny, nz)[2]
    g = _gen(seed)
    gamma = torch.exp(_normal(g, nf))
    x0, w = _uniform(g, n), _uniform(g, n)
    N = torch.tensor([nx, ny, nz], device=DEV, dtype=F64)
    geo = (N * N)[d]                       # |S| delta / V of internal faces
    fixed = torch.arange(n, device=DEV)
    fixed = fixed[fixed % nx == 0]         # x = 0 faces follow the internal ones
    bnd = slice(ni, ni + fixed.shape[0])
    c, cb = gamma[:ni] * geo, 2.0 * N[0] * N[0] * gamma[bnd]
    diag = _sum_faces(n, own, nei, c, c)
    diag[fixed] += cb
    A = dict(n=n, owner=own, neighbour=nei, lower=-c, upper=-c, diag=diag + 1e3)
    xs = [x0]
    for _ in range(case["steps"]):
        xs.append(_cg(A, xs[-1] * 1e3))
    gg, lam = torch.zeros(nf, device=DEV, dtype=F64), w
    for x in reversed(xs[1:]):
        lam = _cg(A, lam)
        gg[:ni] -= geo * (x[own] - x[nei]) * (lam[own] - lam[nei])
        gg[bnd] -= 2.0 * N[0] * N[0] * lam[fixed] * x[fixed]
        lam = lam * 1e3
    return [xs[-1], gg, lam]


def exact(case, seed):
    op = case["op"]
    if op == "amul":
        s = _system(case, seed)
        if case["dtype"] == "float32":
            s = {k: v.float() if k in ("diag", "lower", "upper", "x") else v for k, v in s.items()}
        return [_product(s, s["x"].double()), _product(s, s["x"].double(), transposed=True)]
    if op == "mesh_setup":
        return list(_geometry(_polymesh(case, seed)))
    if op in ("momentum_assembly", "pressure_step"):
        pm = _polymesh(case, seed)
        fc, S, V, cc, w, dl = _geometry(pm)
        own, nei, n = pm["owner"], pm["neighbour"], pm["n"]
        ni, nf = nei.shape[0], own.shape[0]
        P, N = own[:ni], nei
        f = _mesh_fields(case, pm, n, nf)
        wi = w[:ni]

        def lap(D):  # (lower, upper, diag): boundary faces have no delta
            c = D * S[:ni].norm(dim=1) * dl[:ni]
            return [-c / V[P], -c / V[N], _sum_faces(n, P, N, c / V[P], c / V[N])]

        if op == "momentum_assembly":
            F = f["phi"][:ni]
            out, back = F.clamp(min=0.0), F.clamp(max=0.0)
            D = f["D"]
            if case["d"] == "cell":
                D = wi * D[P] + (1.0 - wi) * D[N]
            elif case["d"] == "face":
                D = D[:ni]
            return [back / V[P], out / V[N], _sum_faces(n, P, N, -out / V[P], -back / V[N])] + lap(D)
        H, p, A = f["H"], f["p"], f["A"]
        iA = wi / A[P] + (1.0 - wi) / A[N]
        rc = iA * (p[P] - p[N]) * S[:ni].norm(dim=1) * dl[:ni]
        phi = (H[own] * S).sum(1)
        phi[:ni] = ((wi[:, None] * H[P] + (1.0 - wi[:, None]) * H[N]) * S[:ni]).sum(1) + rc
        div = torch.zeros(n, device=DEV, dtype=F64).index_add_(0, own, phi)
        div.index_add_(0, N, -phi[:ni])
        phi2 = phi.clone()
        phi2[:ni] += rc
        pf = p[own]
        pf[:ni] = wi * p[P] + (1.0 - wi) * p[N]
        grad = torch.zeros(n, 3, device=DEV, dtype=F64).index_add_(0, own, pf[:, None] * S)
        grad.index_add_(0, N, -pf[:ni, None] * S[:ni])
        U = H - grad / V[:, None] / A[:, None]
        return [phi] + lap(iA) + [-div / V, phi2, U * (1e4 / U.norm(dim=1, keepdim=True)).clamp(
            max=1.0)]
    if op == "batched":
        return [s["x"] for s in _batch(case, seed)]
    if op == "adjoint":
        return _exact_adjoint(case, seed)
    x = _system(case, seed)["x"]
    return None if x is None else [x, None]
