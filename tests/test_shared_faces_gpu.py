"""Pairs of cells that share several faces: the faces have one matrix entry between them, which holds the sum of their
terms. Two cells along a zigzag of k edges (2D) or quads (3D), beside the ordinary faces of the box around them."""
import numpy as np
import pytest

import test_by_cell_gpu

pytestmark = pytest.mark.gpu

CASES = [(2, 2), (2, 3), (2, 4), (2, 7), (3, 2), (3, 5)]


def zigzag_pair(ndim, k):
    """The unit box cut into two cells by a zigzag of k segments from (0.5, 0) to (0.5, 1), extruded in 3D."""
    from kcfd.mesh import build_mesh
    y = np.linspace(0.0, 1.0, k + 1)
    x = 0.5 + 0.1 * np.where(np.arange(k + 1) % 2, 1.0, -0.5) * (y > 0) * (y < 1)
    mid = list(range(k + 1))                          # the zigzag, bottom to top
    nodes = np.concatenate([np.stack([x, y], 1), [[0, 0], [0, 1], [1, 0], [1, 1]]])
    bl, tl, br, tr = k + 1, k + 2, k + 3, k + 4
    rings = [[bl] + mid + [tl], [br, tr] + mid[::-1]]  # counter-clockwise
    if ndim == 2:
        sides = {"left": [[tl, bl]], "right": [[br, tr]], "bottom": [[bl, 0], [0, br]], "top": [[tr, k], [k, tl]]}
        return build_mesh(nodes, [np.array(r) for r in rings], {n: [np.array(f) for f in fs] for n, fs in sides.items()})
    N = len(nodes)
    nodes3 = np.concatenate([np.column_stack([nodes, np.zeros(N)]), np.column_stack([nodes, np.ones(N)])])
    faces = []
    for r in rings:
        tris = [[r[0], a, b] for a, b in zip(r[1:], r[2:])]  # the ends, fans of triangles
        fl = [np.array(t[::-1]) for t in tris] + [np.array(t) + N for t in tris]
        fl += [np.array([a, b, b + N, a + N]) for a, b in zip(r, r[1:] + r[:1])]
        faces.append(fl)
    walls = [f for fl in faces for f in fl if not set(int(v) % N for v in f) <= set(mid)]
    cells = [np.array(r + [a + N for a in r]) for r in rings]
    return build_mesh(nodes3, cells, {"walls": walls}, ndim=3, cell_face_node_list=faces)


@pytest.mark.parametrize("ndim,k", CASES)
def test_operators_by_cell(monkeypatch, ndim, k):
    m = zigzag_pair(ndim, k)
    assert m.n_internal_faces == k and m.nnz == 4
    monkeypatch.setattr(test_by_cell_gpu, "meshes", lambda: [("pair", m)])
    test_by_cell_gpu.test_by_cell_equals_colours("pair")


@pytest.mark.parametrize("lists", [True, False])
@pytest.mark.parametrize("ndim,k", CASES)
def test_simple_systems(ndim, k, lists):
    """SIMPLE's momentum and p' matrices, by cell and (without cell lists) by colour, against sums over the faces on
    the host: at most 7 terms of one sign an entry, each rounded a few times."""
    import ctypes as C
    import torch
    from kcfd import _lib
    from kcfd.device_mesh import BCDesc, DeviceMesh, device_layout
    m = zigzag_pair(ndim, k)
    n, D, F, Fb, Fi = m.n_cells, m.ndim, m.n_faces, m.n_boundary_faces, m.n_internal_faces
    rng = np.random.default_rng(5)
    dm, lay = DeviceMesh(m), device_layout(m)
    if not lists:
        dm.desc.cf_ptr = dm.desc.cf_face = None
    mf, dP = rng.standard_normal(F), rng.uniform(0.1, 2.0, n)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    def full(*s, dt=torch.float64):  # what the kernels must overwrite
        return torch.full(s, 7.0, dtype=dt, device="cuda")

    t = {"ut": dev(np.ones(Fb, np.int8)), "ub": dev(rng.standard_normal((Fb, D))), "pt": dev(np.ones(Fb, np.int8)),
         "pv": dev(rng.standard_normal(Fb)), "U": dev(rng.standard_normal((n, D))), "p": dev(rng.standard_normal(n)),
         "mf": dev(mf), "dP": dev(dP)}
    rho, mu = 1.3, 0.02
    owner, neigh = lay["owner"][:Fi], lay["neigh"]
    area, dorth, F_ = lay["area"][:Fi], lay["dorth"], mf[:Fi]
    L, P, st = _lib.lib(), _lib.ptr, _lib.stream_handle()
    for pinned, single in ((0, True), (1, False)):
        bc = BCDesc()
        bc.u_type, bc.u_val, bc.p_type, bc.p_val = (t[q].data_ptr() for q in ("ut", "ub", "pt", "pv"))
        bc.has_p_dirichlet = 1 - pinned
        prm = _lib.MomParams()
        prm.rho, prm.mu, prm.alpha_u, prm.dt, prm.limiter, prm.nonorth = rho, mu, 0.7, 0.0, -1, 0
        df = mu * area / dorth
        mom = (-(df + np.maximum(-F_, 0.0)), -(df + np.maximum(F_, 0.0)))
        pp = -rho * 0.5 * (dP[owner] + dP[neigh]) * area / dorth
        for what, on, no in (("momentum", *mom), ("pressure", pp, pp)):
            v64, v32 = full(m.nnz), full(m.nnz, dt=torch.float32) if single else None
            if what == "momentum":
                _lib.check(L.kcfd_momentum_assemble(C.byref(dm.desc), C.byref(bc), C.byref(prm), P(t["U"]), None,
                                                    P(t["p"]), P(t["mf"]), None, P(full(n)), P(v64), P(v32),
                                                    P(full(n, D)), P(full(n)), st), what)
            else:
                _lib.check(L.kcfd_pressure_assemble(C.byref(dm.desc), C.byref(bc), rho, P(t["dP"]), P(t["mf"]), P(full(n)),
                                                    P(v64), P(v32), P(full(n)), st), what)
            want = np.zeros(m.nnz)
            np.add.at(want, lay["slot_on"], on)
            np.add.at(want, lay["slot_no"], no)
            if what == "pressure" and pinned:
                want[m.indptr[0]:m.indptr[1]] = 0.0
            off = np.setdiff1d(np.arange(m.nnz), m.diag_slot)
            got = v64.cpu().numpy()
            np.testing.assert_allclose(got[off], want[off], rtol=16 * np.finfo(np.float64).eps, atol=0, err_msg=what)
            if single:
                np.testing.assert_array_equal(v32.cpu().numpy(), got.astype(np.float32))
