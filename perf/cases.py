"""Measured workloads of the package: what its users have it do, over the sizes they do it at.

Every case goes through the public Python entry points (kcfd.SIMPLESolver, TwoFluidSolver,
DeviceSystem, DeviceCSR.spmv, BatchSolver, solve_linear_system). Sizes are those of the
repository's own configurations and tests (64^2 and 128^3 cavities, split-quad triangle
channels, the 30 x 90 bubble column, Delaunay tetrahedra, uneven Delaunay p' batches) and
sizes between them.

Linear solves run to a 1e-12 relative residual, which is what the package uses in place of
the reference's sparse direct solves; the FP64 SIMPLE solves to 1e-13, because the cavity's
pinned pressure correction leaves the pressure's level to the last digits of the residual.

  listed()              the measured cases
  draw(rng)             one more case of the same ranges
  prepare(case, seed)   the handle, mesh and device inputs a program holds before the call
  run(state)            one pass, returning what it computes
  work(case)            bytes each input read once and each output written once
  exact(case, seed)     the same outputs from plain torch in 64 bits (None where there is none)
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "k-cfd_b200"))

from kcfd import meshgen  # noqa: E402
from kcfd.assembly import DeviceSystem, boundary_arrays, muscl_deferred_correction  # noqa: E402
from kcfd.batch import BatchSolver, p_prime_sizes  # noqa: E402
from kcfd.device_mesh import DeviceMesh  # noqa: E402
from kcfd.fvm_operators import FVMSystem  # noqa: E402
from kcfd.linear_solver import solve_linear_system  # noqa: E402
from kcfd.mesh import build_mesh  # noqa: E402
from kcfd.simple import SIMPLESolver  # noqa: E402
from kcfd.solver import DeviceCSR  # noqa: E402
from kcfd.two_fluid import TwoFluidSolver  # noqa: E402

RTOL = 1e-12
F64 = torch.float64


def listed():
    return [
        # y = A x on the largest 7-point pattern the benchmark runs (gpu_spmv's device half)
        {"name": "spmv-hex-128", "kind": "spmv", "mesh": "hex", "n": 128, "nrhs": 1},
        # a scalar transport system assembled on a small 2D mesh: launches and latency
        {"name": "assemble-tri-2k", "kind": "assemble", "mesh": "tri", "n": 32},
        # the same operators on a large 3D mesh: memory traffic
        {"name": "assemble-hex-96", "kind": "assemble", "mesh": "hex", "n": 96},
        # the reference's own CPU case: 64^2 cavity, upwind, Jacobi for momentum and p'
        {"name": "simple-quad-64", "kind": "simple", "mesh": "quad", "n": 64, "muscl": "none", "nonorth": False,
         "precond": "jacobi", "precision": "fp64"},
        # channel with inlet and outlet on triangles, ILU(0) p': an ordinary 2D case
        {"name": "simple-tri-7k", "kind": "simple", "mesh": "tri", "n": 60, "muscl": "none", "nonorth": True,
         "precond": "ilu0", "precision": "fp64"},
        # a mid-sized 3D cavity with the configured red-black ILU(0) p'
        {"name": "simple-hex-48-ilu0", "kind": "simple", "mesh": "hex", "n": 48, "muscl": "van_leer", "nonorth": True,
         "precond": "ilu0", "precision": "fp64"},
        # the benchmark's outer iteration: 128^3 jittered cavity, MUSCL, multigrid p'
        {"name": "simple-hex-128-amg", "kind": "simple", "mesh": "hex", "n": 128, "muscl": "van_leer",
         "nonorth": True, "precond": "amg", "precision": "fp64"},
        # the mixed form of the same outer iteration on a quarter-million cells
        {"name": "simple-hex-64-mixed", "kind": "simple", "mesh": "hex", "n": 64, "muscl": "van_leer",
         "nonorth": True, "precond": "amg", "precision": "mixed"},
        # the reference's bubble column (30 x 90 quads): two inner iterations of a time step
        {"name": "twofluid-column-30x90", "kind": "twofluid", "mesh": "column", "n": 30, "inner": 2},
        # two-fluid step with energy on Delaunay tetrahedra, multigrid p'
        {"name": "twofluid-tet-40k", "kind": "twofluid", "mesh": "tet", "n": 40000, "inner": 2},
        # many pressure-correction systems of uneven size solved together
        {"name": "batch-tri-48", "kind": "batch", "systems": 48, "n_min": 2000, "n_max": 20000},
        # the drop-in's default call (method 'direct') on a host CSR system, host to host
        {"name": "dropin-tri-5k", "kind": "dropin", "mesh": "delaunay", "n": 5000},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed kinds with its own size and options."""
    kind = rng.choice(["spmv", "assemble", "assemble", "simple", "simple", "simple", "twofluid", "batch", "dropin"])
    if kind == "spmv":
        mesh = rng.choice(["hex", "tri", "quad"])
        n = _logint(rng, 12, 120) if mesh == "hex" else _logint(rng, 24, 700)
        return {"kind": kind, "mesh": mesh, "n": n, "nrhs": rng.choice([1, 1, 2, 3])}
    if kind == "assemble":
        mesh = rng.choice(["hex", "tri", "quad"])
        return {"kind": kind, "mesh": mesh, "n": _logint(rng, 8, 90) if mesh == "hex" else _logint(rng, 16, 500)}
    if kind == "simple":
        mesh = rng.choice(["hex", "tri", "quad"])
        n = _logint(rng, 10, 72) if mesh == "hex" else _logint(rng, 20, 130) if mesh == "quad" else _logint(rng, 16, 90)
        precision = rng.choice(["fp64", "fp64", "mixed"])
        precond = rng.choice(["ilu0", "amg"]) if precision == "fp64" else "amg"
        if precision == "fp64" and mesh == "quad" and n <= 80:
            precond = "jacobi"
        return {"kind": kind, "mesh": mesh, "n": n, "muscl": rng.choice(["none", "minmod", "van_leer"]),
                "nonorth": rng.choice([True, False]), "precond": precond, "precision": precision}
    if kind == "twofluid":
        if rng.random() < 0.5:
            return {"kind": kind, "mesh": "column", "n": rng.randint(14, 48), "inner": rng.randint(1, 2)}
        return {"kind": kind, "mesh": "tet", "n": _logint(rng, 4000, 36000), "inner": rng.randint(1, 2)}
    if kind == "batch":
        lo = _logint(rng, 300, 2000)
        return {"kind": kind, "systems": rng.randint(6, 40), "n_min": lo, "n_max": _logint(rng, 3 * lo, 18000)}
    return {"kind": kind, "mesh": "delaunay", "n": _logint(rng, 600, 5000)}


# ------------------------------------------------------------------------ meshes --
@functools.lru_cache(maxsize=3)
def _mesh(kind, n):
    """The host mesh; a program keeps it over many runs. Its shape does not depend on the inputs' seed."""
    if kind == "hex":
        nodes, cells, cf, bd = meshgen.hex_box_arrays(1.0, 1.0, 1.0, n, n, n, meshgen.CAVITY_3D_NAMES)
        nodes = meshgen.jitter_interior(nodes, (n, n, n), (1.0 / n,) * 3, 0.2, seed=0)
        return build_mesh(nodes, cells, bd, ndim=3, cell_face_node_list=cf)
    if kind == "quad":
        return build_mesh(*meshgen.quad_box_arrays(0.0, 0.0, 1.0, 1.0, n, n, meshgen.CAVITY_2D_NAMES))
    if kind == "tri":
        return build_mesh(*meshgen.tri_channel_arrays(2.0, 2.0, n, n))
    if kind == "column":
        return build_mesh(*meshgen.bubble_column_arrays(0.15, 0.45, n, 3 * n))
    if kind == "tet":
        nodes, cells, cf, bd = meshgen.delaunay_tet_arrays((0.2, 0.2, 1.0), n, np.random.default_rng(0))
        return build_mesh(nodes, cells, bd, ndim=3, cell_face_node_list=cf)
    pts, cells, bd = meshgen.delaunay_tri_arrays(max(n // 2, 4), np.random.default_rng(0),
                                                 side_points=int(math.ceil(math.sqrt(n / 2))))
    return build_mesh(pts, cells, bd)


@functools.lru_cache(maxsize=3)
def _batch_meshes(systems, n_min, n_max):
    out = []
    for k, n in enumerate(p_prime_sizes(systems, n_min, n_max, 0)):
        npts = max(int(n) // 2, 4)
        pts, cells, bd = meshgen.delaunay_tri_arrays(npts, np.random.default_rng((0, k)),
                                                     side_points=int(math.ceil(math.sqrt(npts))))
        out.append(build_mesh(pts, cells, bd))
    return out


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _smooth(x, rng, modes=4):
    """A smooth field of the points x [n, D]: a few random cosine modes, amplitude falling with the wave number."""
    f = np.zeros(len(x))
    for _ in range(modes):
        k = rng.integers(1, 4, x.shape[1])
        ph = rng.uniform(0.0, 2.0 * math.pi, x.shape[1])
        t = np.ones(len(x))
        for d in range(x.shape[1]):
            t = t * np.cos(math.pi * k[d] * x[:, d] + ph[d])
        f += rng.normal() / float(np.sum(k)) * t
    return f


def _vortex(x, rng):
    """A developing cavity flow: u = curl of a random smooth streamfunction that vanishes on the unit box's walls."""
    a, b = rng.uniform(0.2, 0.8), rng.uniform(-0.3, 0.3)
    sx, sy = np.sin(math.pi * x[:, 0]), np.sin(math.pi * x[:, 1])
    cx, cy = np.cos(math.pi * x[:, 0]), np.cos(math.pi * x[:, 1])
    u = np.zeros_like(x)
    # psi = (a + b x) sx^2 sy^2
    w = a + b * x[:, 0]
    u[:, 0] = w * sx ** 2 * 2.0 * math.pi * sy * cy
    u[:, 1] = -(w * 2.0 * math.pi * sx * cx + b * sx ** 2) * sy ** 2
    u /= math.pi
    if x.shape[1] == 3:
        u *= np.sin(math.pi * x[:, 2])[:, None] ** 2
    return u + 1e-3 * rng.standard_normal(x.shape)


# ------------------------------------------------------------- operator assembly --
def _transport_inputs(mesh, seed):
    """Host inputs of a scalar transport system: diffusivity, mass flux, fields, gradient, sources."""
    rng = np.random.default_rng(seed)
    n, D = mesh.n_cells, mesh.ndim
    U = np.stack([_smooth(mesh.ccenter, rng) for _ in range(D)], 1)
    nb = np.where(mesh.neighbour >= 0, mesh.neighbour, mesh.owner)
    uf = 0.5 * (U[mesh.owner] + U[nb])
    mf = (uf * mesh.normal).sum(1) * mesh.area
    phi = _smooth(mesh.ccenter, rng)
    return {"gamma": np.exp(rng.uniform(math.log(0.1), math.log(10.0), n)) * 1e-2, "mf": mf, "phi": phi,
            "phi_old": phi + 0.01 * rng.standard_normal(n), "Sp": -rng.uniform(0.0, 1.0, n), "Su": rng.standard_normal(n),
            "grad": rng.standard_normal((n, D)), "phi_b": {nm: _smooth(mesh.fcenter[f], rng)
                                                            for nm, f in mesh.boundary_patches.items()}}


def _transport_bc(mesh):
    """Dirichlet on every second patch, a fixed gradient on one, zero gradient on the rest."""
    types = ["dirichlet", "zero_gradient", "neumann", "zero_gradient"]
    return {nm: ({"type": "neumann", "value": 0.3} if types[i % 4] == "neumann" else {"type": types[i % 4]})
            for i, nm in enumerate(mesh.boundary_patches)}


def _prepare_assemble(case, seed):
    mesh = _mesh(case["mesh"], case["n"])
    h = _transport_inputs(mesh, seed)
    dm = DeviceMesh(mesh)
    bt, bv, bg = boundary_arrays(dm, _transport_bc(mesh), h["phi_b"])
    st = {k: _cuda(h[k]) for k in ("gamma", "phi", "phi_old", "Sp", "Su", "grad")}
    st.update(kind="assemble", dm=dm, sys=DeviceSystem(dm), mf=_cuda(h["mf"][dm.face_ref]), bt=bt, bv=bv, bg=bg)
    return st


def _run_assemble(st):
    s = st["sys"]
    s.reset()
    s.diffusion_operator(st["gamma"])
    s.convection_operator_upwind(st["mf"])
    s.temporal_operator(1.0, 0.01, st["phi_old"])
    s.linearized_source(st["Sp"], st["Su"])
    s.apply_boundary_conditions(st["bt"], st["bv"], st["bg"], st["gamma"], st["mf"])
    corr = muscl_deferred_correction(st["dm"], st["phi"], st["mf"], st["grad"], "van_leer")
    s.under_relax(st["phi"], 0.7)
    return {"vals": s.vals, "diag": s.diag, "rhs": s.rhs, "corr": corr}


class _Geometry:
    """A mesh's arrays as torch tensors, with the face distances and weights of the discretisation."""

    def __init__(self, mesh):
        self.D, self.n = mesh.ndim, mesh.n_cells
        self.o, self.it = _cuda(mesh.owner), _cuda(mesh.neighbour >= 0)
        self.nb = torch.where(self.it, _cuda(mesh.neighbour), self.o)
        self.S, self.nrm, self.fc = _cuda(mesh.area), _cuda(mesh.normal), _cuda(mesh.fcenter)
        self.cc, self.vol = _cuda(mesh.ccenter), _cuda(mesh.volume)
        self.dvec = self.cc[self.nb] - self.cc[self.o]
        self.d = torch.where(self.it, self.dvec.norm(dim=1), (self.fc - self.cc[self.o]).norm(dim=1))
        self.dorth = torch.maximum((self.dvec * self.nrm).sum(1).abs(), 0.1 * self.dvec.norm(dim=1))
        dO, dN = (self.fc - self.cc[self.o]).norm(dim=1), (self.fc - self.cc[self.nb]).norm(dim=1)
        self.gc = dN / (dO + dN)
        self.i = self.it.nonzero().reshape(-1)     # internal faces
        self.b = (~self.it).nonzero().reshape(-1)  # boundary faces
        self.oi, self.ni, self.ob = self.o[self.i], self.nb[self.i], self.o[self.b]

    def cells(self, *shape):
        return torch.zeros(self.n, *shape, dtype=F64, device="cuda")

    def gradient(self, phi, face_b):
        """Green-Gauss; face_b holds the boundary faces' values."""
        g = self.gc[self.i]
        fl = ((g * phi[self.oi] + (1.0 - g) * phi[self.ni]) * self.S[self.i])[:, None] * self.nrm[self.i]
        out = self.cells(self.D)
        out.index_add_(0, self.oi, fl)
        out.index_add_(0, self.ni, -fl)
        out.index_add_(0, self.ob, (face_b * self.S[self.b])[:, None] * self.nrm[self.b])
        return out / self.vol[:, None]

    def muscl(self, phi, mf, grad, name):
        pos = mf[self.i] >= 0
        up, dn = torch.where(pos, self.oi, self.ni), torch.where(pos, self.ni, self.oi)
        dcd = phi[dn] - phi[up]
        lin = (grad[up] * (self.fc[self.i] - self.cc[up])).sum(1)
        keep = dcd.abs() >= 1e-15
        r = 2.0 * lin / torch.where(keep, dcd, torch.ones_like(dcd)) - 1.0
        if name == "minmod":
            psi = r.clamp(0.0, 1.0)
        else:  # van_leer
            psi = torch.where(r > 0, 2.0 * r / (1.0 + r.clamp(min=0.0)), torch.zeros_like(r))
        fc = torch.where(keep, mf[self.i].abs() * 0.5 * psi * dcd, torch.zeros_like(dcd))
        out = self.cells()
        out.index_add_(0, up, -fc)
        out.index_add_(0, dn, fc)
        return out


def _transport_system(mesh, h):
    """(off-diagonals owner->neighbour and back per face, diagonal, rhs, relaxed-diagonal addition) in 64 bits."""
    g = _Geometry(mesh)
    gam, mf, phi = _cuda(h["gamma"]), _cuda(h["mf"]), _cuda(h["phi"])
    gf = 2.0 * gam[g.oi] * gam[g.ni] / (gam[g.oi] + gam[g.ni]) * g.S[g.i] / g.d[g.i]
    F = mf[g.i]
    on, no = -gf + F.clamp(max=0.0), -gf + (-F).clamp(max=0.0)
    diag, rhs = g.cells(), g.cells()
    diag.index_add_(0, g.oi, gf + F.clamp(min=0.0))
    diag.index_add_(0, g.ni, gf + (-F).clamp(min=0.0))
    diag.index_add_(0, g.ob, mf[g.b].clamp(min=0.0))
    diag += g.vol / 0.01 - _cuda(h["Sp"]) * g.vol
    rhs += g.vol / 0.01 * _cuda(h["phi_old"]) + _cuda(h["Su"]) * g.vol
    bc = _transport_bc(mesh)
    for nm, f in mesh.boundary_patches.items():
        f = _cuda(f)
        own, Fb, t = g.o[f], mf[f], bc[nm]["type"]
        if t == "dirichlet":
            c, pb = gam[own] * g.S[f] / g.d[f], _cuda(h["phi_b"][nm])
            diag.index_add_(0, own, c)
            rhs.index_add_(0, own, (c + (-Fb).clamp(min=0.0)) * pb)
        elif t == "neumann":
            rhs.index_add_(0, own, bc[nm]["value"] * g.S[f])
        else:
            diag.index_add_(0, own, (-Fb).clamp(min=0.0))
    corr = g.muscl(phi, mf, _cuda(h["grad"]), "van_leer")
    return g, on, no, diag, rhs, corr, phi


def _exact_assemble(case, seed):
    mesh = _mesh(case["mesh"], case["n"])
    g, on, no, diag, rhs, corr, phi = _transport_system(mesh, _transport_inputs(mesh, seed))
    add = diag * (1.0 - 0.7) / 0.7
    vals = torch.zeros(mesh.nnz, dtype=F64, device="cuda")
    fi = g.i.cpu().numpy()
    vals[_cuda(mesh.slot_on[fi].astype(np.int64))] = on
    vals[_cuda(mesh.slot_no[fi].astype(np.int64))] = no
    vals[_cuda(mesh.diag_slot.astype(np.int64))] = diag + add
    return {"vals": vals, "diag": diag + add, "rhs": rhs + add * phi, "corr": corr}


# ------------------------------------------------------------------------- SpMV ----
def _spmv_inputs(mesh, nrhs, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1.0, 1.0, mesh.nnz), rng.standard_normal((mesh.n_cells, nrhs))


def _prepare_spmv(case, seed):
    mesh = _mesh(case["mesh"], case["n"])
    vals, x = _spmv_inputs(mesh, case["nrhs"], seed)
    A = DeviceCSR(_cuda(mesh.indptr), _cuda(mesh.indices), _cuda(vals))
    x = _cuda(x)
    return {"kind": "spmv", "A": A, "x": x, "y": torch.empty_like(x), "nrhs": case["nrhs"]}


def _exact_spmv(case, seed):
    mesh = _mesh(case["mesh"], case["n"])
    vals, x = _spmv_inputs(mesh, case["nrhs"], seed)
    rows = _cuda(np.repeat(np.arange(mesh.n_cells), np.diff(mesh.indptr)))
    y = torch.zeros(x.shape, dtype=F64, device="cuda")
    return y.index_add_(0, rows, _cuda(vals)[:, None] * _cuda(x)[_cuda(mesh.indices.astype(np.int64))])


# ----------------------------------------------------------------------- SIMPLE ----
SIMPLE_MU = {"hex": 0.0025, "quad": 0.01, "tri": 0.02}


def _simple_inputs(mesh, kind, seed):
    rng = np.random.default_rng(seed)
    x = np.asarray(mesh.ccenter)
    if kind == "tri":   # channel of height 2: a perturbed parabolic profile
        U = np.stack([x[:, 1] * (2.0 - x[:, 1]), np.zeros(len(x))], 1) * rng.uniform(0.7, 1.3)
        return U + 0.02 * rng.standard_normal(U.shape), 0.1 * _smooth(x, rng)
    return _vortex(x, rng), 0.1 * _smooth(x, rng)


def _simple_bc(mesh, kind):
    """[(patch, velocity type, velocity, pressure type)] of the cavity or the channel."""
    out = []
    for nm, f in mesh.boundary_patches.items():
        if kind == "tri" and nm == "inlet":
            y = np.asarray(mesh.fcenter)[f][:, 1]
            out.append((nm, "dirichlet", np.stack([y * (2.0 - y), np.zeros_like(y)], 1), "zero_gradient"))
        elif kind == "tri" and nm == "outlet":
            out.append((nm, "zero_gradient", np.zeros((len(f), mesh.ndim)), "dirichlet"))
        else:
            v = np.zeros((len(f), mesh.ndim))
            if nm == "lid":
                v[:, 0] = 1.0
            out.append((nm, "dirichlet", v, "zero_gradient"))
    return out


def _prepare_simple(case, seed):
    mesh = _mesh(case["mesh"], case["n"])
    U, p = _simple_inputs(mesh, case["mesh"], seed)
    s = SIMPLESolver(mesh, rho=1.0, mu=SIMPLE_MU[case["mesh"]], precision=case["precision"],
                     precond_p=case["precond"], rtol=RTOL if case["precision"] == "mixed" else 0.1 * RTOL, maxiter=20000,
                     muscl=None if case["muscl"] == "none" else case["muscl"], nonorth=case["nonorth"], graph=True)
    for nm, ut, uv, pt in _simple_bc(mesh, case["mesh"]):
        s.set_velocity_bc(nm, ut, uv)
        s.set_pressure_bc(nm, pt, 0.0 if pt == "dirichlet" else None)
    s.alpha_u, s.alpha_p, s.tol = 0.7, 0.3, 0.0
    return {"kind": "simple", "s": s, "U": _cuda(U), "p": _cuda(p)}


def _run_simple(st):
    """One outer iteration from the given fields."""
    s = st["s"]
    s.U_t.copy_(st["U"])
    s.p_t.copy_(st["p"])
    s.iterate(1)
    return {"U": s.U_t, "p": s.p_t}


def _solve_dominant(apply, diag, b, x):
    """A x = b for a diagonally dominant A: Jacobi sweeps down to rounding."""
    best = math.inf
    for k in range(400):
        r = b - apply(x)
        x = x + r / diag
        if k % 10 == 9:
            rn = float(r.norm())
            if rn > 0.5 * best:
                break
            best = rn
    return x


def _solve_spd(apply, diag, b, free):
    """A x = b on the free cells (x = 0 elsewhere): conjugate gradients, restarted from the true residual until it
    no longer falls."""
    x, last = torch.zeros_like(b), math.inf
    for _ in range(6):
        r = (b - apply(x)) * free
        start = float(r.norm())
        if start == 0.0 or start > 0.5 * last:
            break
        last = start
        z = r / diag
        p, rz = z.clone(), torch.dot(r, z)
        for k in range(1, 12000):
            q = apply(p) * free
            a = rz / torch.dot(p, q)
            x += a * p
            r -= a * q
            if k % 50 == 0 and float(r.norm()) < 1e-10 * start:
                break
            z = r / diag
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
    return x


def _exact_simple(case, seed):
    mesh = _mesh(case["mesh"], case["n"])
    g = _Geometry(mesh)
    mu, D = SIMPLE_MU[case["mesh"]], mesh.ndim
    U, p = (_cuda(a) for a in _simple_inputs(mesh, case["mesh"], seed))
    F = mesh.n_faces
    ub, udir, pdir = np.zeros((F, D)), np.zeros(F, bool), np.zeros(F, bool)
    for nm, ut, uv, pt in _simple_bc(mesh, case["mesh"]):
        f = mesh.boundary_patches[nm]
        ub[f], udir[f], pdir[f] = uv, ut == "dirichlet", pt == "dirichlet"
    ub, udir, pdir = _cuda(ub)[g.b], _cuda(udir)[g.b], _cuda(pdir)[g.b]
    w, S = g.gc[g.i], g.S

    def face_u(U):
        return torch.where(udir[:, None], ub, U[g.ob])

    def mass_flux(U):
        mf = torch.empty(F, dtype=F64, device="cuda")
        mf[g.i] = ((w[:, None] * U[g.oi] + (1.0 - w)[:, None] * U[g.ni]) * g.nrm[g.i]).sum(1) * S[g.i]
        mf[g.b] = (face_u(U) * g.nrm[g.b]).sum(1) * S[g.b]
        return mf

    mf = mass_flux(U)
    Fi, Fb = mf[g.i], mf[g.b]
    Df, Db = mu * S[g.i] / g.dorth[g.i], mu * S[g.b] / g.d[g.b]
    aP = g.cells()
    aP.index_add_(0, g.oi, Df + Fi.clamp(min=0.0))
    aP.index_add_(0, g.ni, Df + (-Fi).clamp(min=0.0))
    aP.index_add_(0, g.ob, torch.where(udir, Db + Fb.clamp(min=0.0), Fb.abs()))
    on, no = -(Df + (-Fi).clamp(min=0.0)), -(Df + Fi.clamp(min=0.0))
    ar = aP / 0.7

    def apply_m(x):
        y = ar * x
        y.index_add_(0, g.oi, on * x[g.ni])
        y.index_add_(0, g.ni, no * x[g.oi])
        return y

    new = torch.empty_like(U)
    for c in range(D):
        b = (1.0 - 0.7) / 0.7 * aP * U[:, c]
        src = 0.5 * (p[g.oi] + p[g.ni]) * g.nrm[g.i, c] * S[g.i]
        b.index_add_(0, g.oi, -src)
        b.index_add_(0, g.ni, src)
        pb = torch.where(pdir, torch.zeros_like(Fb), p[g.ob])
        b.index_add_(0, g.ob, -pb * g.nrm[g.b, c] * S[g.b])
        b.index_add_(0, g.ob, torch.where(udir, (Db + (-Fb).clamp(min=0.0)) * ub[:, c], torch.zeros_like(Fb)))
        if case["muscl"] != "none" or case["nonorth"]:
            gr = g.gradient(U[:, c], face_u(U)[:, c])
            if case["muscl"] != "none":
                b += g.muscl(U[:, c].contiguous(), mf, gr, case["muscl"])
            if case["nonorth"]:
                kv = g.nrm[g.i] * S[g.i][:, None] - (S[g.i] / g.dorth[g.i])[:, None] * g.dvec[g.i]
                fl = mu * (kv * (w[:, None] * gr[g.oi] + (1.0 - w)[:, None] * gr[g.ni])).sum(1)
                b.index_add_(0, g.oi, fl)
                b.index_add_(0, g.ni, -fl)
        new[:, c] = _solve_dominant(apply_m, ar, b, U[:, c].clone())
    U = new
    mf = mass_flux(U)
    dP = g.vol / aP
    df = 0.5 * (dP[g.oi] + dP[g.ni]) * S[g.i] / g.dorth[g.i]
    dg, b = g.cells(), g.cells()
    dg.index_add_(0, g.oi, df)
    dg.index_add_(0, g.ni, df)
    dg.index_add_(0, g.ob, torch.where(pdir, dP[g.ob] * S[g.b] / g.d[g.b], torch.zeros_like(Fb)))
    b.index_add_(0, g.oi, -mf[g.i])
    b.index_add_(0, g.ni, mf[g.i])
    b.index_add_(0, g.ob, -mf[g.b])

    def apply_p(x):
        y = dg * x
        y.index_add_(0, g.oi, -df * x[g.ni])
        y.index_add_(0, g.ni, -df * x[g.oi])
        return y

    free = torch.ones_like(b)
    if not bool(pdir.any()):
        free[0] = 0.0   # the pinned cell
    pp = _solve_spd(apply_p, dg, b, free)
    gp = g.gradient(pp, torch.where(pdir, torch.zeros_like(Fb), pp[g.ob]))
    return {"U": U - dP[:, None] * gp, "p": p + 0.3 * pp}


# -------------------------------------------------------------------- two-fluid ----
TF_FIELDS = ("alpha_g", "alpha_l", "U_l", "U_g", "p", "T_l", "T_g")


def _prepare_twofluid(case, seed):
    mesh = _mesh(case["mesh"], case["n"])
    rng = np.random.default_rng(seed)
    tet = case["mesh"] == "tet"
    s = TwoFluidSolver(mesh, rtol=RTOL, p_precond="amg" if tet else "ilu0")
    n, D = mesh.n_cells, mesh.ndim
    s.rho_l, s.mu_l, s.cp_l, s.rho_g, s.mu_g = 998.0, 1e-3, 4182.0, 1.2, 1.8e-5
    s.d_b, s.solve_energy, s.max_outer_iter, s.tol, s.dt = 0.003, tet, case["inner"], 0.0, 1e-3
    s.initialize(0.05)
    up = [0.0] * (D - 1) + [0.2]
    s.set_inlet_bc("inlet_gas", 0.05, U_l=[0.0] * D, U_g=up, T_l=372.0, T_g=373.15)
    s.set_outlet_bc("outlet", 0.0)
    for nm in mesh.boundary_patches:
        if nm.startswith("wall"):
            s.set_wall_bc(nm)
    ag = rng.uniform(0.02, 0.08, n)
    T = 370.0 + rng.uniform(0.0, 6.0, n)
    scale = np.asarray(mesh.ccenter).max(0)
    x = np.asarray(mesh.ccenter) / scale
    init = {"alpha_g": ag, "alpha_l": 1.0 - ag, "U_l": 0.05 * _vortex(x, rng), "U_g": 0.1 * _vortex(x, rng),
            "p": 10.0 * _smooth(x, rng), "T_l": T, "T_g": T + rng.uniform(0.0, 1.0, n)}
    return {"kind": "twofluid", "s": s, "init": init}


def _run_twofluid(st):
    """One time step from host fields, and the host fields after it."""
    s = st["s"]
    for k, v in st["init"].items():
        getattr(s, k).values = v
    s.step()
    return {k: getattr(s, k).values for k in TF_FIELDS}


# ------------------------------------------------------------- batched p' systems --
def _pprime_inputs(mesh, rng):
    n = mesh.n_cells
    return np.exp(rng.uniform(math.log(0.1), math.log(10.0), n)), rng.standard_normal(n)


def _pprime_values(mesh, gamma):
    """CSR values of the diffusion operator with the 'dirichlet' patch held, assembled on the device."""
    dm = DeviceMesh(mesh)
    s = DeviceSystem(dm)
    gam = _cuda(gamma)
    s.diffusion_operator(gam)
    bt, bv, bg = boundary_arrays(dm, {"dirichlet": {"type": "dirichlet"}, "wall": {"type": "zero_gradient"}}, {})
    s.apply_boundary_conditions(bt, bv, bg, gam, torch.zeros(mesh.n_faces, dtype=F64, device="cuda"))
    return s


def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    meshes = _batch_meshes(case["systems"], case["n_min"], case["n_max"])
    vals, rhs = [], []
    for m in meshes:
        gamma, b = _pprime_inputs(m, rng)
        vals.append(_pprime_values(m, gamma).vals)
        rhs.append(b)
    B = BatchSolver([(m.indptr, m.indices) for m in meshes], mode="fp64", precond="jacobi", rtol=RTOL, maxiter=20000)
    b = _cuda(np.concatenate(rhs))
    return {"kind": "batch", "B": B, "vals": torch.cat(vals), "b": b, "x": torch.empty_like(b)}


def _run_batch(st):
    st["x"].zero_()
    _, _, status = st["B"].solve(st["vals"], st["b"], st["x"])
    return {"x": st["x"], "status": status}


def _exact_pprime(mesh, gamma, b):
    """Dense 64-bit solve of the diffusion system, refined twice."""
    g = _Geometry(mesh)
    gam = _cuda(gamma)
    c = 2.0 * gam[g.oi] * gam[g.ni] / (gam[g.oi] + gam[g.ni]) * g.S[g.i] / g.d[g.i]
    dg = g.cells()
    dg.index_add_(0, g.oi, c)
    dg.index_add_(0, g.ni, c)
    f = _cuda(mesh.boundary_patches["dirichlet"])
    dg.index_add_(0, g.o[f], gam[g.o[f]] * g.S[f] / g.d[f])
    A = torch.zeros(g.n, g.n, dtype=F64, device="cuda")
    A[g.oi, g.ni] = -c
    A[g.ni, g.oi] = -c
    A.diagonal().copy_(dg)
    LU, piv = torch.linalg.lu_factor(A)
    b = _cuda(b)[:, None]
    x = torch.linalg.lu_solve(LU, piv, b)
    for _ in range(2):
        x = x + torch.linalg.lu_solve(LU, piv, b - A @ x)
    return x[:, 0]


def _exact_batch(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for m in _batch_meshes(case["systems"], case["n_min"], case["n_max"]):
        out.append(_exact_pprime(m, *_pprime_inputs(m, rng)))
    return {"x": torch.cat(out), "status": None}


# ------------------------------------------------------------------ host drop-in ---
def _prepare_dropin(case, seed):
    mesh = _mesh(case["mesh"], case["n"])
    gamma, b = _pprime_inputs(mesh, np.random.default_rng(seed))
    return {"kind": "dropin", "sys": FVMSystem.from_csr(_pprime_values(mesh, gamma).to_sparse(), b)}


def _exact_dropin(case, seed):
    mesh = _mesh(case["mesh"], case["n"])
    return _exact_pprime(mesh, *_pprime_inputs(mesh, np.random.default_rng(seed)))


# --------------------------------------------------------------------- interface ---
def prepare(case, seed):
    return {"spmv": _prepare_spmv, "assemble": _prepare_assemble, "simple": _prepare_simple,
            "twofluid": _prepare_twofluid, "batch": _prepare_batch, "dropin": _prepare_dropin}[case["kind"]](case, seed)


def run(st):
    kind = st["kind"]
    if kind == "spmv":
        return st["A"].spmv(st["x"], st["y"], nrhs=st["nrhs"])
    if kind == "assemble":
        return _run_assemble(st)
    if kind == "simple":
        return _run_simple(st)
    if kind == "twofluid":
        return _run_twofluid(st)
    if kind == "batch":
        return _run_batch(st)
    return solve_linear_system(st["sys"])


def exact(case, seed):
    if case["kind"] == "twofluid":
        return None   # a whole model step: no short restatement, and its large solves take over 20 s on plain torch
    return {"spmv": _exact_spmv, "assemble": _exact_assemble, "simple": _exact_simple, "batch": _exact_batch,
            "dropin": _exact_dropin}[case["kind"]](case, seed)


def work(case):
    if case["kind"] == "batch":
        ms = _batch_meshes(case["systems"], case["n_min"], case["n_max"])
        n, nnz = sum(m.n_cells for m in ms), sum(m.nnz for m in ms)
        return {"bytes": 12.0 * nnz + 4.0 * n + 16.0 * n, "flops": 0.0}
    m = _mesh(case["mesh"], case["n"])
    n, D, F, Fi, nnz = m.n_cells, m.ndim, m.n_faces, m.n_internal_faces, m.nnz
    geometry = F * (4 + 8 * (1 + D)) + Fi * (4 + 8 + 8) + n * 8   # owner, area, normal; neighbour, weight, distance; volume
    if case["kind"] == "spmv":
        r = case["nrhs"]
        return {"bytes": 12.0 * nnz + 4.0 * (n + 1) + 16.0 * n * r, "flops": 2.0 * nnz * r}
    if case["kind"] == "assemble":
        # geometry with face and cell centres, mass flux and face->slot map; gamma, phi, phi_old, Sp, Su, grad in;
        # values, diagonal, rhs and correction out
        return {"bytes": float(geometry + F * 8 * (D + 1) + Fi * 8 + n * (8 * (5 + 2 * D) + 4) + 8 * nnz + 24 * n),
                "flops": 0.0}
    if case["kind"] == "dropin":
        return {"bytes": 12.0 * nnz + 4.0 * n + 16.0 * n, "flops": 0.0}
    if case["kind"] == "simple":
        extra = F * 8 * D + n * 8 * D if case["muscl"] != "none" or case["nonorth"] else 0
        return {"bytes": float(geometry + extra + n * 16 * (D + 1)), "flops": 0.0}
    return {"bytes": float(geometry + n * 16 * (2 * D + 5)), "flops": 0.0}   # two-fluid: seven fields in and out
