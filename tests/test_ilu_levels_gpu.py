"""The launch-per-level ILU(0) set-up (short rows, few levels) against the persistent factor kernel, which the same
levels behind empty ones take: the same elimination order within a row, so bitwise the same preconditioner."""
import numpy as np
import pytest
from scipy import sparse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 129, 1000])
def test_level_kernel_factors_as_the_persistent_kernel(n):
    import torch
    from kcfd.solver import DeviceCSR, Solver
    rng = np.random.default_rng(n)
    i = np.arange(n)
    rows, cols = [i], [i]
    for d in (1, 7):
        rows += [i[:max(n - d, 0)], i[d:]]
        cols += [i[d:], i[:max(n - d, 0)]]
    r, c = np.concatenate(rows), np.concatenate(cols)
    A = sparse.csr_matrix((np.where(r == c, 4.0, -1.0) + 0.1 * rng.standard_normal(len(r)), (r, c)), shape=(n, n))
    A.sort_indices()
    d = DeviceCSR.from_scipy(A)
    few = (i % 8).astype(np.int32)   # rows 1 and 7 apart differ modulo 8
    many = few + 32                  # levels 0 to 31 empty
    q = torch.from_numpy(rng.standard_normal(n)).cuda()
    out = []
    for lev in (few, many):
        s = Solver(d, precond="ilu0", levels=lev, team=2)
        s.setup(d)
        out.append(s.apply_precond(d, q).cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])
