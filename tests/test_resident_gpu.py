"""On-chip BiCGSTAB (csrc/resident.cuh) against the persistent grid kernel at the sizes where its row split changes:
one row, one warp, one CTA, ragged last CTAs, the steps in rows per thread, the largest of a cluster, the grid form."""
import numpy as np
import pytest
from scipy import sparse

pytestmark = pytest.mark.gpu


def system(n, seed=0, nonsym=0.3):
    """A diagonally dominant 2D five-point matrix on a ragged last row, slightly non-symmetric."""
    rng = np.random.default_rng(seed)
    w = max(1, int(np.sqrt(n)))
    i = np.arange(n)
    r, c = [], []
    for d, ok in ((1, (i + 1) % w != 0), (w, np.ones(n, bool))):
        m = ok & (i + d < n)
        r += [i[m], i[m] + d]
        c += [i[m] + d, i[m]]
    r, c = np.concatenate(r or [np.zeros(0, int)]), np.concatenate(c or [np.zeros(0, int)])
    v = -rng.uniform(1.0 - nonsym, 1.0 + nonsym, len(r))
    A = sparse.csr_matrix((v, (r, c)), shape=(n, n))
    A = (A + sparse.diags(np.asarray(abs(A).sum(1)).ravel() * 1.02 + 0.01)).tocsr()
    A.sort_indices()
    return A


def greedy_levels(A):
    lev = -np.ones(A.shape[0], np.int32)
    for i in range(A.shape[0]):
        used = {lev[j] for j in A.indices[A.indptr[i]:A.indptr[i + 1]] if j != i}
        lev[i] = next(k for k in range(64) if k not in used)
    return lev


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 1025, 4096, 4097, 8193, 11001, 16385, 32768, 32769, 37889, 150001])
@pytest.mark.parametrize("prec,nrhs", [("none", 1), ("jacobi", 1), ("jacobi", 2), ("jacobi", 3), ("ilu0", 1), ("ilu0", 3)])
def test_matches_grid_kernel(n, prec, nrhs):
    import torch
    from kcfd.solver import DeviceCSR, Solver
    A = system(n, seed=n)
    d = DeviceCSR.from_scipy(A)
    rng = np.random.default_rng(n + 1)
    b = rng.standard_normal((n, nrhs))
    levels = greedy_levels(A) if prec == "ilu0" else None
    out = []
    for team in (0, 2):
        s = Solver(d, precond=prec, nrhs=nrhs, rtol=1e-12, maxiter=4000, team=team, levels=levels)
        s.setup(d)
        x = torch.from_numpy(0.1 * rng.standard_normal((n, nrhs)) * 0 + 0.25).cuda()
        s.solve(d, torch.from_numpy(b).cuda(), x)
        assert s.status.tolist() == [0] * nrhs
        out.append(x.cpu().numpy())
    # both stop at ||r|| < 1e-12 ||b||; the matrix is dominant by 2 %, so its condition number is below 200
    for c in range(nrhs):
        bn = np.linalg.norm(b[:, c])
        assert np.linalg.norm(A @ out[0][:, c] - b[:, c]) <= 2e-12 * bn
        assert np.linalg.norm(out[0][:, c] - out[1][:, c]) <= 1e-9 * np.linalg.norm(out[1][:, c])


@pytest.mark.parametrize("n", [700, 5000])
def test_many_levels_and_stop_rules(n):
    """Natural-order ILU(0) (many short levels), x0 kept, zero rhs, and the GPU path's stopping rule."""
    import torch
    from kcfd import _lib
    from kcfd.solver import DeviceCSR, Solver
    A = system(n, seed=3)
    d = DeviceCSR.from_scipy(A)
    b = np.random.default_rng(4).standard_normal(n)
    for kw in (dict(precond="ilu0"), dict(precond="jacobi", stop=_lib.STOP_GPU)):
        s = Solver(d, rtol=1e-10, maxiter=4000, **kw)
        s.setup(d)
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        it, rr, st = s.solve(d, torch.from_numpy(b).cuda(), x)
        assert int(st[0]) == 0 and int(it[0]) > 0 and float(rr[0]) < 1e-10
        assert np.linalg.norm(A @ x.cpu().numpy() - b) <= 2e-10 * np.linalg.norm(b)
        again = x.clone()
        s.solve(d, torch.from_numpy(b).cuda(), again)  # starts at the solution: the scipy rule stops before a step
        if "stop" not in kw:
            assert int(s.iters[0]) == 0 and torch.equal(again, x)
        s.solve(d, torch.zeros(n, dtype=torch.float64, device="cuda"), again)
        if "stop" not in kw:
            assert float(again.abs().max()) == 0.0
    s = Solver(d, precond="jacobi", rtol=1e-14, maxiter=3)
    s.setup(d)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    it, rr, st = s.solve(d, torch.from_numpy(b).cuda(), x)
    assert int(st[0]) == _lib.MAXITER and int(it[0]) == 3


@pytest.mark.parametrize("prec", ["none", "jacobi"])
def test_batch_on_chip(prec):
    """A batch around the steps of the on-chip shapes (CTAs, rows per thread) and one system past the largest:
    against the grid kernel, and bitwise the same alone."""
    import torch
    from kcfd.batch import BatchSolver
    from kcfd.solver import DeviceCSR, Solver
    sizes = [1, 40, 256, 257, 1025, 2047, 2048, 2049, 3073, 4097, 10241, 12289, 20481, 32768, 32769]
    mats = [system(n, seed=n, nonsym=0.2) for n in sizes]
    rng = np.random.default_rng(7)
    rhs = [rng.standard_normal(n) for n in sizes]
    pats = [(A.indptr.astype(np.int32), A.indices.astype(np.int32)) for A in mats]

    def solve(ids):
        B = BatchSolver([pats[k] for k in ids], mode="fp64", precond=prec, rtol=1e-12, maxiter=5000)
        x = torch.zeros(B.n_total, dtype=torch.float64, device="cuda")
        vals = torch.from_numpy(np.concatenate([mats[k].data for k in ids])).cuda()
        _, rr, st = B.solve(vals, B.pack([rhs[k] for k in ids]), x)
        assert st.tolist() == [0] * len(ids) and float(rr.max()) < 1e-12
        return B.unpack(x)

    xs = solve(range(len(sizes)))
    for k, n in enumerate(sizes):
        d = DeviceCSR.from_scipy(mats[k])
        s = Solver(d, precond=prec, rtol=1e-12, maxiter=5000, team=2)
        s.setup(d)
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        s.solve(d, torch.from_numpy(rhs[k]).cuda(), x)
        ref = x.cpu().numpy()
        assert np.linalg.norm(xs[k] - ref) <= 1e-9 * np.linalg.norm(ref)
    for k in (3, 9, 12):
        np.testing.assert_array_equal(solve([k])[0], xs[k])


@pytest.mark.parametrize("n,nrhs", [(150001, 3)])
def test_components_one_after_another(n, nrhs):
    """Right-hand sides that do not fit on chip together, against each alone."""
    import torch
    from kcfd.solver import DeviceCSR, Solver
    A = system(n, seed=5)
    d = DeviceCSR.from_scipy(A)
    b = torch.from_numpy(np.random.default_rng(6).standard_normal((n, nrhs))).cuda()
    s = Solver(d, precond="jacobi", nrhs=nrhs, rtol=1e-12, maxiter=4000)
    s.setup(d)
    x = torch.full_like(b, 0.5)
    s.solve(d, b, x)
    assert s.status.tolist() == [0] * nrhs
    one = Solver(d, precond="jacobi", rtol=1e-12, maxiter=4000)
    one.setup(d)
    for c in range(nrhs):
        xc = torch.full((n,), 0.5, dtype=torch.float64, device="cuda")
        one.solve(d, b[:, c].contiguous(), xc)
        assert torch.equal(xc, x[:, c]) and int(one.iters[0]) == int(s.iters[c])


@pytest.mark.parametrize("n,nrhs,prec", [(300, 1, "jacobi"), (5000, 2, "ilu0"), (60001, 3, "jacobi")])
def test_mixed_on_chip(n, nrhs, prec):
    """A MIXED handle that fits on chip meets the FP64 stopping test, and still refuses the FP64-only calls."""
    import torch
    from kcfd import _lib
    from kcfd.solver import DeviceCSR, Solver
    A = system(n, seed=8)
    d = DeviceCSR.from_scipy(A, fp32=True)
    b = np.random.default_rng(9).standard_normal((n, nrhs))
    s = Solver(d, precond=prec, mode=_lib.MODE_MIXED, nrhs=nrhs, rtol=1e-11, maxiter=4000,
               levels=greedy_levels(A) if prec == "ilu0" else None)
    s.setup(d)
    x = torch.zeros((n, nrhs), dtype=torch.float64, device="cuda")
    s.solve(d, torch.from_numpy(b).cuda(), x)
    assert s.status.tolist() == [0] * nrhs
    r = A @ x.cpu().numpy() - b
    assert (np.linalg.norm(r, axis=0) <= 2e-11 * np.linalg.norm(b, axis=0)).all()
    if nrhs == 1:
        with pytest.raises(_lib.KcfdError):
            s.apply_precond(d, x[:, 0].contiguous())
