"""SIMPLE's momentum and pressure-correction systems assembled by cell against the colour-by-colour assembly of the
same terms (a mesh descriptor without cell lists), on meshes with 3 to 7 faces a cell and ragged sizes. The two add
the same terms (at most 7 faces and 2 cell terms an entry) in another order."""
import ctypes as C

import numpy as np
import pytest

from test_by_cell_gpu import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limiter,nonorth,dt", [(-1, 0, 0.0), (3, 0, 0.01), (-1, 1, 0.0), (1, 1, 0.01)])
@pytest.mark.parametrize("which", ["hex", "hybrid", "tri", "quad1", "quad"])
def test_simple_systems_by_cell(which, limiter, nonorth, dt):
    import torch
    from kcfd import _lib
    from kcfd.device_mesh import BCDesc, DeviceMesh
    mesh = dict(meshes())[which]
    n, D, F, Fb, nnz = mesh.n_cells, mesh.ndim, mesh.n_faces, mesh.n_boundary_faces, mesh.nnz
    rng = np.random.default_rng(4)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    U, Uo, p, mf = (dev(rng.standard_normal(s)) for s in ((n, D), (n, D), n, F))
    gU, dP0 = dev(rng.standard_normal((n, D, D))), dev(rng.uniform(0.1, 2.0, n))
    ut, pt = (dev(rng.integers(0, 2, Fb).astype(np.int8)) for _ in range(2))
    ub, pv = dev(rng.standard_normal((Fb, D))), dev(rng.standard_normal(Fb))
    prm = _lib.MomParams()
    prm.rho, prm.mu, prm.alpha_u, prm.dt, prm.limiter, prm.nonorth = 1.3, 0.02, 0.7, dt, limiter, nonorth
    L, P, st = _lib.lib(), _lib.ptr, _lib.stream_handle()

    def run(lists):
        dm = DeviceMesh(mesh)
        if not lists:
            dm.desc.cf_ptr = dm.desc.cf_face = None
        out = []
        for pinned, single in ((0, True), (1, False)):
            bc = BCDesc()
            bc.u_type, bc.u_val, bc.p_type, bc.p_val = (t.data_ptr() for t in (ut, ub, pt, pv))
            bc.has_p_dirichlet = 1 - pinned
            # what the kernels must overwrite
            aP, v64, b, dP = (torch.full(s, 7.0, dtype=torch.float64, device="cuda") for s in ((n,), (nnz,), (n, D), (n,)))
            v32 = torch.full((nnz,), 7.0, dtype=torch.float32, device="cuda") if single else None
            _lib.check(L.kcfd_momentum_assemble(C.byref(dm.desc), C.byref(bc), C.byref(prm), P(U), P(Uo), P(p), P(mf),
                                                P(gU), P(aP), P(v64), P(v32), P(b), P(dP), st), "momentum")
            out += [t.cpu().numpy() for t in (aP, v64, b, dP, v32) if t is not None]
            aP, v64, b = (torch.full(s, 7.0, dtype=torch.float64, device="cuda") for s in ((n,), (nnz,), (n,)))
            _lib.check(L.kcfd_pressure_assemble(C.byref(dm.desc), C.byref(bc), 1.3, P(dP0), P(mf), P(aP), P(v64), P(v32),
                                                P(b), st), "pressure")
            out += [t.cpu().numpy() for t in (aP, v64, b, v32) if t is not None]
        return out

    for k, (u, w) in enumerate(zip(run(True), run(False))):
        # sums of terms up to the largest of the array, in another order; FP32 copies: one rounding of those
        eps = np.finfo(u.dtype).eps
        np.testing.assert_allclose(u, w, rtol=0, atol=64 * eps * np.abs(w).max(), err_msg=str(k))
