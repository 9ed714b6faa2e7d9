"""Infinite and very large cell values in the by-cell terms of the two-fluid model: a boundary face adds no p' difference
and takes the cell's own pressure as it is, as colour by colour."""
import ctypes as C

import numpy as np
import pytest

from test_by_cell_gpu import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["quad1", "tri", "hex"])
def test_boundary_faces(which):
    import torch
    from kcfd import _lib
    from kcfd.device_mesh import DeviceMesh
    mesh = dict(meshes())[which]
    n, D = mesh.n_cells, mesh.ndim
    rng = np.random.default_rng(3)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    cell = int(mesh.owner[np.nonzero(mesh.neighbour < 0)[0][0]])  # a boundary cell
    pp = rng.standard_normal(n)
    big = rng.standard_normal(n)
    pp[cell], big[cell] = np.inf, 1.2e308
    pos = [dev(rng.uniform(0.1, 2.0, n)) for _ in range(4)]
    alpha, K = dev(rng.uniform(0.1, 0.2, n)), dev(np.zeros(n))
    U = rng.standard_normal((n, D))
    prm = _lib.TfParams()
    prm.rho_l, prm.rho_g, prm.dt = 998.0, 1.2, 1e-3
    L, P, st = _lib.lib(), _lib.ptr, _lib.stream_handle()

    def run(lists):
        dm = DeviceMesh(mesh)
        if not lists:
            dm.desc.cf_ptr = dm.desc.cf_face = None
        m = C.byref(dm.desc)
        g, Ul, Ug, p = torch.zeros(n, D, dtype=torch.float64, device="cuda"), dev(U), dev(2 * U), dev(np.zeros(n))
        _lib.check(L.kcfd_tf_correct(m, 0.3, P(dev(pp)), *[P(a) for a in pos], P(g), P(Ul), P(Ug), P(p), st), "correct")
        v, d, r = (dev(np.ones(s)) for s in (mesh.nnz, n, n * D))
        _lib.check(L.kcfd_tf_momentum_sources(m, C.byref(prm), 0, D, 1.0, P(alpha), P(dev(big)), P(K), P(dev(U)), None, P(v),
                                              P(d), P(r), st), "momentum")
        return [t.cpu().numpy() for t in (g, Ul, Ug, p, r)]

    for a, b in zip(run(True), run(False)):
        fin = np.isfinite(b)
        np.testing.assert_array_equal(np.isfinite(a), fin)
        np.testing.assert_array_equal(a[~fin], b[~fin])
        np.testing.assert_allclose(a[fin], b[fin], rtol=0, atol=64 * np.finfo(float).eps * np.abs(b[fin]).max(initial=0.0))
