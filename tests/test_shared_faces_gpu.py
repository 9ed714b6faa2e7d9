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
