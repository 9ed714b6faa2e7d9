"""Face loops by cell (csrc/by_cell.cuh) against the colour-by-colour scatter of the same operators (a mesh
descriptor without cell lists), on meshes with 3 to 7 faces a cell and ragged sizes. The two add the same terms in
another order: differences stay within the rounding of sums of at most 7 terms per entry."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def meshes():
    from kcfd import meshgen
    from kcfd.mesh import build_mesh
    n, c, cf, b = meshgen.hex_box_arrays(1.0, 1.0, 1.0, 5, 7, 3, meshgen.CAVITY_3D_NAMES)
    n = meshgen.jitter_interior(n, (5, 7, 3), (1 / 5, 1 / 7, 1 / 3), 0.2, seed=1)
    yield "hex", build_mesh(n, c, b, ndim=3, cell_face_node_list=cf)
    n, c, cf, b = meshgen.hybrid_hex_tet_arrays(2.0, 0.4, 0.3, 6, 3, 2)
    yield "hybrid", build_mesh(n, c, b, ndim=3, cell_face_node_list=cf)
    yield "tri", build_mesh(*meshgen.tri_channel_arrays(1.0, 0.7, 13, 9))
    yield "quad1", build_mesh(*meshgen.quad_box_arrays(0.0, 0.0, 1.0, 1.0, 1, 1, meshgen.CAVITY_2D_NAMES))
    yield "quad", build_mesh(*meshgen.quad_box_arrays(0.0, 0.0, 1.0, 1.0, 33, 31, meshgen.CAVITY_2D_NAMES))


@pytest.mark.parametrize("which", ["hex", "hybrid", "tri", "quad1", "quad"])
def test_by_cell_equals_colours(which):
    import torch
    from kcfd import _lib
    from kcfd.assembly import DeviceSystem, muscl_deferred_correction
    from kcfd.device_mesh import DeviceMesh
    mesh = dict(meshes())[which]
    n, D, F, Fb = mesh.n_cells, mesh.ndim, mesh.n_faces, mesh.n_boundary_faces
    rng = np.random.default_rng(2)

    def dev(a, **kw):
        return torch.from_numpy(np.ascontiguousarray(a, **kw)).cuda()

    phi = dev(rng.standard_normal(n))
    args = {k: dev(rng.uniform(0.1, 2.0, n)) for k in ("gamma", "al", "ag", "apl", "apg", "K", "To", "h", "dm")}
    mf, mf2 = dev(rng.standard_normal(F)), dev(rng.standard_normal(F))
    bt, qm = dev(rng.integers(-1, 3, Fb).astype(np.int8)), dev(rng.integers(0, 2, Fb).astype(np.int8))
    bv, bv3, bg = dev(rng.standard_normal(Fb)), dev(rng.standard_normal((Fb, D))), dev(rng.standard_normal(Fb))
    grad, U, Uold = (dev(rng.standard_normal((n, D))) for _ in range(3))
    prm = _lib.TfParams()
    for k, v in dict(rho_l=998.0, rho_g=1.2, dt=1e-3, h_fg=2e6).items():
        setattr(prm, k, v)
    for k in range(3):
        prm.g[k] = -1.0 - k
    start = [rng.standard_normal(s) for s in (mesh.nnz, n, n * D)]
    L, P, st = _lib.lib(), _lib.ptr, _lib.stream_handle()

    def run(lists):
        dm = DeviceMesh(mesh)
        if not lists:
            dm.desc.cf_ptr = dm.desc.cf_face = None
        m = C.byref(dm.desc)
        out = {}

        def fresh(nr=1):
            return dev(start[0]), dev(start[1]), dev(start[2][: n * nr])

        def op(name, call, *keep):
            _lib.check(call(), name)
            out[name] = [t.cpu().numpy() for t in keep]

        s = DeviceSystem(dm)
        s.vals, s.diag, s.rhs = fresh()
        s.diffusion_operator(args["gamma"])
        s.convection_operator_upwind(mf)
        s.apply_boundary_conditions(bt, bv, bg, args["gamma"], mf)
        out["system"] = [t.cpu().numpy() for t in (s.vals, s.diag, s.rhs)]
        for lim in ("minmod", "superbee", "van_albada", "van_leer"):
            out[lim] = [muscl_deferred_correction(dm, phi, mf, grad, lim).cpu().numpy()]
        a, pr = args, C.byref(prm)
        for c0, nc, old in ((0, D, Uold), (D - 1, 1, None)):
            v, d, r = fresh(nc)
            op(f"momentum{nc}", lambda: L.kcfd_tf_momentum_sources(m, pr, c0, nc, 998.0, P(a["al"]), P(phi), P(a["K"]),
                                                                  P(U), P(old), P(v), P(d), P(r), st), v, d, r)
            v, d, r = fresh(nc)
            op(f"boundary{nc}", lambda: L.kcfd_tf_boundary(m, P(bt), P(bv3 if nc == D else bv), P(bg), nc, P(a["gamma"]),
                                                          P(mf), P(v), P(d), P(r), st), v, d, r)
        v, d, r = fresh()
        op("pressure", lambda: L.kcfd_tf_pressure_assemble(m, pr, P(a["al"]), P(a["ag"]), P(a["apl"]), P(a["apg"]), P(mf),
                                                          P(mf2), P(v), P(d), P(r), st), v, d, r)
        g, Ul, Ug, p = torch.zeros(n, D, dtype=torch.float64, device="cuda"), U.clone(), Uold.clone(), phi.clone()
        op("correct", lambda: L.kcfd_tf_correct(m, 0.3, P(a["To"]), P(a["al"]), P(a["ag"]), P(a["apl"]), P(a["apg"]), P(g),
                                               P(Ul), P(Ug), P(p), st), g, Ul, Ug, p)
        v, d, r = fresh()
        op("energy", lambda: L.kcfd_tf_energy_sources(m, pr, 998.0, 4182.0, P(a["al"]), None, P(a["To"]), P(a["h"]),
                                                     P(a["dm"]), 1.0, P(qm), P(bv), P(a["al"]), P(v), P(d), P(r), st), v, d, r)
        return out

    x, y = run(True), run(False)
    for k in y:
        for i, (u, w) in enumerate(zip(x[k], y[k])):
            # sums of terms up to the largest of the array, in another order
            np.testing.assert_allclose(u, w, rtol=0, atol=64 * np.finfo(float).eps * np.abs(w).max(), err_msg=f"{k}[{i}]")
