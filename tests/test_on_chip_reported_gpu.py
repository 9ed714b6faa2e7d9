"""Where a handle or a batch solves, as it reports it: on chip, or by its team or tier."""
import numpy as np
import pytest

from test_resident_gpu import greedy_levels, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,chip", [
    (dict(), True), (dict(precond="ilu0"), True), (dict(nrhs=3), True), (dict(mode="mixed"), True),
    (dict(team=1), False), (dict(team=1, n=900), True), (dict(team=2), False), (dict(team=3), False),
    (dict(team=3, mode="mixed"), False), (dict(lanes=2), False), (dict(block=512), False), (dict(precond="amg"), False),
    (dict(method="cg"), False), (dict(n=60001), True), (dict(n=310001), False), (dict(n=310001, precond="ilu0"), False)])
def test_solver(kw, chip):
    from kcfd import _lib
    from kcfd.solver import DeviceCSR, Solver
    kw = dict(kw)
    n = kw.pop("n", 5000)
    mode = _lib.MODE_MIXED if kw.pop("mode", "") == "mixed" else _lib.MODE_FP64
    A = system(n, seed=1)
    levels = greedy_levels(A) if kw.get("precond") == "ilu0" else None
    s = Solver(DeviceCSR.from_scipy(A), mode=mode, levels=levels, **kw)
    assert (s.on_chip > 0) == chip
    if chip:
        assert s.on_chip == 1 if kw.get("team") == 1 else s.on_chip <= 160
    if kw.get("team"):
        assert s.info()["team"] == kw["team"]


def test_batch():
    from kcfd.batch import BatchSolver
    sizes = [1, 300, 2048, 20000, 32768, 32769, 40000]
    pats = [(A.indptr.astype(np.int32), A.indices.astype(np.int32)) for A in (system(n, seed=n) for n in sizes)]
    B = BatchSolver(pats, mode="fp64")
    t, c = B.tiers(), B.on_chip()
    assert c["systems"] == 5 and 1 <= c["launches"] <= 5
    assert t["cluster"] + t["big"] + t["small"] == 2
    for kw in (dict(mode="mixed"), dict(cluster_rows=2000), dict(big_rows=-1), dict(lanes=2)):
        B = BatchSolver(pats, **{"mode": "fp64", **kw})
        t = B.tiers()
        assert B.on_chip() == {"systems": 0, "launches": 0}
        assert t["cluster"] + t["big"] + t["small"] == len(sizes)


@pytest.mark.parametrize("N,prec,nrhs,lanes,chip,team", [(30, "jacobi", 3, 0, True, 3), (36, "ilu0", 1, 0, True, 3),
                                                         (62, "ilu0", 1, 0, False, 3), (36, "jacobi", 1, 4, False, 3),
                                                         (20, "jacobi", 1, 0, True, 2)])
def test_mixed_handle_makes_one(monkeypatch, N, prec, nrhs, lanes, chip, team):
    """The handle is made once, also where the system does not fit; the plan agrees with the handle."""
    from scipy import sparse
    import kcfd.solver as ks
    T, I = sparse.diags([-np.ones(N - 1), np.full(N, 2.1), -np.ones(N - 1)], [-1, 0, 1]), sparse.identity(N)
    A = (sparse.kron(sparse.kron(T, I), I) + sparse.kron(sparse.kron(I, T), I) + sparse.kron(sparse.kron(I, I), T)).tocsr()
    d = ks.DeviceCSR.from_scipy(A, fp32=True)
    i = np.arange(N ** 3)
    levels = ((i + i // N + i // N ** 2) % 2).astype(np.int32) if prec == "ilu0" else None
    made = []

    class Counted(ks.Solver):
        def __init__(self, *a, **kw):
            made.append(1)
            super().__init__(*a, **kw)

    monkeypatch.setattr(ks, "Solver", Counted)
    s = ks.mixed_handle(d, precond=prec, nrhs=nrhs, levels=levels, lanes=lanes, rtol=1e-8)
    assert len(made) == 1
    assert (s.on_chip > 0) == chip and s.info()["team"] == team
    assert lanes or ks.on_chip_ctas(d, prec, nrhs, levels) == s.on_chip
