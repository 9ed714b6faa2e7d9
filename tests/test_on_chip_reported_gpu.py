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
