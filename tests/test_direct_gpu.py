"""solve_linear_system(method='direct') on matrices without ILU levels: the residual that it promises, and its two tries
(the coloured ILU(0) first, the natural order when that does not converge)."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def chain(n, pe):
    """Convection-diffusion in 1D, pe = 1: pure upwind."""
    e = np.ones(n - 1)
    A = sp.diags([-(1 + pe) * e, np.full(n, 2.0) + 0.01 * (1 - pe), -(1 - pe) * e], [-1, 0, 1]).tocsr()
    A.sort_indices()
    return A


def box(N, pe):
    e = np.ones(N - 1)
    T, I = sp.diags([-(1 + pe) * e, np.full(N, 2.0), -(1 - pe) * e], [-1, 0, 1]), sp.identity(N)
    A = (sp.kron(I, T) + sp.kron(T, I)).tocsr()
    A.sort_indices()
    return A


def solve(A, b, **kw):
    from kcfd.fvm_operators import FVMSystem
    from kcfd.linear_solver import solve_linear_system
    return solve_linear_system(FVMSystem.from_csr(A, b), **kw)


@pytest.mark.parametrize("A", [chain(3, 0.9), chain(200, 0.999), chain(2000, 0.999), chain(2000, 0.9), chain(5000, 1.0),
                               box(30, 0.0), box(70, 0.99)], ids=lambda A: str(A.shape[0]))
def test_residual(A):
    """To 1e-12 of ||b||, or the rounding of the residual itself, at most 5 products a row."""
    b = np.random.default_rng(0).standard_normal(A.shape[0])
    x = solve(A, b)
    floor = np.linalg.norm(abs(A) @ abs(x) + abs(b))
    assert np.linalg.norm(A @ x - b) <= max(1e-12 * np.linalg.norm(b), 4 * np.finfo(float).eps * floor)


class Recorder:
    """Stands in for Solver: keeps what each handle was given and may replace its status."""

    def __init__(self, real, statuses):
        self.real, self.statuses, self.seen = real, list(statuses), []

    def __call__(self, d, **kw):
        s = self.real(d, **kw)
        rec = dict(maxiter=kw["maxiter"], coloured=kw["levels"] is not None, x=None)
        self.seen.append(rec)
        status = self.statuses.pop(0) if self.statuses else None
        inner = s.solve

        def solve(d, b, x):
            if rec["x"] is None:
                rec["x"] = x.cpu().numpy()
            it, rr, st = inner(d, b, x)
            if status is not None:
                st = st.clone().fill_(status)
            return it, rr, st

        s.solve = solve
        return s


@pytest.mark.parametrize("status", ["MAXITER", "BREAKDOWN", "TIMEOUT"])
def test_first_try_fails(monkeypatch, status):
    from kcfd import _lib, linear_solver as ls
    A = box(24, 0.3)
    n = A.shape[0]
    rng = np.random.default_rng(1)
    b, x0 = rng.standard_normal(n), rng.standard_normal(n)
    rec = Recorder(ls.Solver, [getattr(_lib, status)])
    monkeypatch.setattr(ls, "Solver", rec)
    if status == "TIMEOUT":
        with pytest.raises(_lib.KcfdError):
            solve(A, b, x0=x0)
        assert len(rec.seen) == 1
        return
    x = solve(A, b, x0=x0)
    assert np.linalg.norm(A @ x - b) <= 1e-12 * np.linalg.norm(b)
    first, second = rec.seen
    assert first["coloured"] and not second["coloured"]
    np.testing.assert_array_equal(first["x"], x0)
    np.testing.assert_array_equal(second["x"], x0)
    assert second["maxiter"] == 20 * n and first["maxiter"] == 200 + 20 * (2 * 24 - 1) < second["maxiter"]


def test_given_levels_are_the_only_try(monkeypatch):
    from kcfd import _lib, linear_solver as ls
    A = box(24, 0.3)
    b = np.ones(A.shape[0])
    rec = Recorder(ls.Solver, [_lib.BREAKDOWN])
    monkeypatch.setattr(ls, "Solver", rec)
    solve(A, b, levels=np.arange(A.shape[0], dtype=np.int32))
    assert len(rec.seen) == 1 and rec.seen[0]["maxiter"] == 20 * A.shape[0]


def test_natural_levels_on_the_host():
    from kcfd import _lib
    A = box(24, 0.3)
    ip, ix = A.indptr.astype(np.int32), A.indices.astype(np.int32)
    lev = np.full(A.shape[0], -1, np.int32)
    assert _lib.lib().kcfd_natural_levels(A.shape[0], ip.ctypes.data, ix.ctypes.data, lev.ctypes.data) == _lib.OK
    i = np.arange(A.shape[0])
    np.testing.assert_array_equal(lev, i // 24 + i % 24)
