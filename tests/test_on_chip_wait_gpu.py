"""The waits of the on-chip solves' teams: a CTA that comes late to a reduction, within the wait's limit (the sums are
right) and beyond it (every CTA gives up together and reports KCFD_TIMEOUT, whichever was late, and the context stays
usable)."""
import numpy as np
import pytest

from case16 import channel_mesh, convdiff_system

pytestmark = pytest.mark.gpu

FORMS = [(0, 1), (0, 2), (0, 7), (0, 8), (1, 1), (1, 5), (1, 64)]


def run(grid, ctas, budget, late, cycles):
    import torch
    from kcfd import _lib
    scratch = torch.zeros(19 * ctas, dtype=torch.float64, device="cuda")
    status = torch.full((ctas + 2,), -1, dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().kcfd_selftest_on_chip(grid, ctas, budget, late, cycles, _lib.ptr(scratch), _lib.ptr(status),
                                                _lib.stream_handle()), "kcfd_selftest_on_chip")
    torch.cuda.synchronize()
    s = status.tolist()
    return s[:ctas], s[-1]


@pytest.mark.parametrize("grid,ctas", FORMS)
def test_in_time(grid, ctas):
    for late in (-1, 0, ctas - 1):
        assert run(grid, ctas, 400_000_000, late, 1_000_000) == ([0] * ctas, 0)


@pytest.mark.parametrize("grid,ctas", [f for f in FORMS if f[1] > 1])
def test_too_late(grid, ctas):
    import torch
    from kcfd import _lib
    from kcfd.solver import DeviceCSR, Solver
    for late in (0, ctas - 1):
        assert run(grid, ctas, 1_000_000, late, 20_000_000) == ([_lib.TIMEOUT] * ctas, _lib.TIMEOUT if grid else 0)
    A, b = convdiff_system(channel_mesh(24, 16))
    d = DeviceCSR.from_scipy(A)
    s = Solver(d, precond="jacobi", rtol=1e-10, maxiter=3000)
    s.setup(d)
    x = torch.zeros(len(b), dtype=torch.float64, device="cuda")
    s.solve(d, torch.from_numpy(b).cuda(), x)
    assert int(s.status[0]) == 0 and s.barrier_error() == 0
    assert np.linalg.norm(A @ x.cpu().numpy() - b) <= 2e-10 * np.linalg.norm(b)


def test_bad_arguments():
    import torch
    from kcfd import _lib
    t = torch.zeros(64, dtype=torch.float64, device="cuda")
    for grid, ctas, budget, late, cycles in ((0, 9, 1000, -1, 0), (1, 65, 1000, -1, 0), (0, 0, 1000, -1, 0),
                                             (0, 2, 0, -1, 0), (0, 2, 1000, 2, 0), (0, 2, 1000, 0, 10 ** 9)):
        assert _lib.lib().kcfd_selftest_on_chip(grid, ctas, budget, late, cycles, _lib.ptr(t), _lib.ptr(t),
                                                None) == _lib.BAD_INPUT
