"""The graph engine's FP64 Jacobi form, which multiplies by A D^-1 in its loop: badly scaled columns, warm starts, a
second solve after the values changed, and both stopping rules, against the true residual of the caller's matrix."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stop", [0, 1])  # _lib.STOP_SCIPY, _lib.STOP_GPU
@pytest.mark.parametrize("nrhs", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 33, 1025, 70001])
def test_scaled_engine(n, nrhs, stop):
    import torch
    from kcfd.solver import DeviceCSR, Solver
    rng = np.random.default_rng(n + nrhs)
    off = [k for k in (1, 7) if k < n]
    A = sp.diags([np.full(n, 6.0)] + [rng.uniform(-1, 0, n - k) for k in off for _ in (0, 1)],
                 [0] + [s * k for k in off for s in (1, -1)]).tocsr()
    A.sort_indices()
    d = s = None
    for decades in (0, 6):  # the second solve: same handle, columns scaled over twelve decades
        w = 10.0 ** rng.uniform(-decades, decades, n)
        M = (A @ sp.diags(w)).tocsr()
        M.sort_indices()
        if s is None:
            d = DeviceCSR(torch.from_numpy(M.indptr.astype(np.int32)).cuda(),
                          torch.from_numpy(M.indices.astype(np.int32)).cuda(), torch.from_numpy(M.data.copy()).cuda())
            s = Solver(d, precond="jacobi", nrhs=nrhs, rtol=1e-10, maxiter=500, team=3, stop=stop)
            assert s.graph_engine
        d.vals64.copy_(torch.from_numpy(M.data))
        b = rng.standard_normal((n, nrhs))
        b[:, -1] *= 1e-3
        x = torch.from_numpy(0.1 * rng.standard_normal((n, nrhs)) / w[:, None]).cuda()  # a residual of ||b||'s size
        s.setup(d)
        s.solve(d, torch.from_numpy(b).cuda(), x)
        assert s.status.cpu().numpy().tolist() == [0] * nrhs
        # the rule's 1e-10 on the recursive residual; the true one differs by rounding, 1e-16 of a start up to
        # 1,000 ||b|| (the last column) over some 20 iterations
        res = np.linalg.norm(b - M @ x.cpu().numpy(), axis=0) / np.linalg.norm(b, axis=0)
        assert (res < 2e-10).all(), res
