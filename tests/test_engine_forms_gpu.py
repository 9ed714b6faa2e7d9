"""The forms that large systems take, at sizes that would otherwise be solved on chip: the graph engine's FP32 momentum
solve in SIMPLE and in the two-fluid model, and the engine as the automatic choice for what does not fit on chip."""
import numpy as np
import pytest

from test_resident_gpu import greedy_levels, system
from two_fluid_case import setup

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("pc", ["ilu0", "amg"])
def test_mixed_simple_on_the_engine(pc):
    """72^2 cavity, team 3: momentum in the engine's FP32 form, p' in FP64 (above 4,096 cells) or over an FP32
    hierarchy; after 5 outer iterations every solve met its FP64 test of 1e-8 and the fields agree with the FP64 engine's
    within 1e-6 relative L2."""
    from kcfd import mesh as km, meshgen
    from kcfd.simple import SIMPLESolver
    N = 72
    m = km.build_mesh(*meshgen.quad_box_arrays(0, 0, 1, 1, N, N, meshgen.CAVITY_2D_NAMES))
    runs = []
    for prec in ("fp64", "mixed"):
        s = SIMPLESolver(m, rho=1.0, mu=0.01, precision=prec, precond_p=pc, rtol=1e-8, team=3)
        assert s.s_m.graph_engine and not s.s_m.on_chip and s.s_p.graph_engine and not s.s_p.on_chip
        for nm in m.boundary_patches:
            s.set_velocity_bc(nm, "dirichlet", [1.0, 0.0] if nm == "lid" else [0.0, 0.0])
            s.set_pressure_bc(nm, "zero_gradient")
        s.max_outer_iter, s.tol = 5, 0.0
        s.solve_steady()
        assert int(s.s_p.status[0]) == 0 and s.s_m.status.tolist() == [0, 0]
        runs.append((s.U.values.copy(), s.p.values.copy()))
    for a, b in zip(*runs):
        assert _rel(b, a) < 1e-6


def test_mixed_two_fluid_on_the_engine(monkeypatch):
    """42,000-cell channel whose MIXED systems are kept off the chip, against the FP64 model: every field within 1e-6
    relative L2 after a step (every solve stops at the same 1e-12 FP64 relative residual)."""
    import kcfd.solver as ks
    from kcfd import mesh as km, meshgen
    from kcfd.two_fluid import TwoFluidSolver
    m = km.build_mesh(*meshgen.quad_box_arrays(0.0, 0.0, 2.0, 1.0, 210, 200, meshgen.CHANNEL_2D_NAMES))
    monkeypatch.setattr(ks, "on_chip_ctas", lambda *a: 0)
    runs = []
    for precision in ("fp64", "mixed"):
        sv = TwoFluidSolver(m, p_precond="amg", precision=precision)
        setup(sv, list(m.boundary_patches), m.ndim, m.n_cells, 7, lambda nm, a: setattr(getattr(sv, nm), "values", a))
        for s in (sv._s1, sv._sg):
            assert bool(s.on_chip) == (precision == "fp64") and s.graph_engine
        sv.step()
        runs.append({f: getattr(sv, f).values.copy() for f in ("alpha_g", "U_l", "U_g", "p", "T_l", "T_g")})
    for f in runs[0]:
        assert _rel(runs[1][f], runs[0][f]) < 1e-6, f


@pytest.mark.parametrize("prec,nrhs", [("jacobi", 1), ("ilu0", 1), ("ilu0", 3)])
def test_automatic_beyond_the_chip(prec, nrhs):
    import torch
    from kcfd.solver import DeviceCSR, Solver
    n = 310001
    A = system(n, seed=2)
    d = DeviceCSR.from_scipy(A)
    s = Solver(d, precond=prec, nrhs=nrhs, rtol=1e-10, maxiter=4000, levels=greedy_levels(A) if prec == "ilu0" else None)
    assert s.graph_engine and not s.on_chip
    s.setup(d)
    b = np.random.default_rng(3).standard_normal((n, nrhs))
    x = torch.zeros((n, nrhs), dtype=torch.float64, device="cuda")
    s.solve(d, torch.from_numpy(b).cuda(), x)
    assert s.status.tolist() == [0] * nrhs
    assert (np.linalg.norm(A @ x.cpu().numpy() - b, axis=0) <= 2e-10 * np.linalg.norm(b, axis=0)).all()
