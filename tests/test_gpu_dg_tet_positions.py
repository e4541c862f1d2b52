"""Tetrahedron faces in every position of their two elements (GPU, against
the oracle's sums over the points)."""
from itertools import permutations

import numpy as np
import pytest

import oracle as O
from _util import REL_TOL, dg_blocks_to_crs, sparse_rel_err, vec_rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import modfem_gb300 as g
    g.load_library()
    return g


@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("dword", [False, True])
def test_tet_faces_in_all_positions_vs_oracle(gb, seed, dword):
    """Every element's vertices in a random (even) order: faces meet in all
    positions of the two elements, degrees 1..4 on either side, to the FP64
    tolerance of the other systems in both arithmetics."""
    from modfem_gb300.mesh import anisotropic_tensors, structured_tet_mesh, tet_faces
    t = structured_tet_mesh(2, jitter=0.2, seed=seed)
    rng = np.random.default_rng(seed)
    even = [q for q in permutations(range(4)) if sum(q[a] > q[b] for a in range(4) for b in range(a + 1, 4)) % 2 == 0]
    t.el_nodes = np.stack([el[list(even[i])] for el, i in zip(t.el_nodes, rng.integers(0, 12, t.nel))])
    F = tet_faces(t)
    p = rng.integers(1, 5, t.nel)
    A = anisotropic_tensors(t.nel, seed=seed).reshape(-1, 9)
    c = gb.Context(0)
    c.set_mesh(t)
    c.set_coefficients(D=A, f=1.2, g=0.3)
    c.dg_set_degrees(p)
    c.dg_set_faces(F, penalty=10.0)
    c.dg_build_structure()
    if dword:
        c.dg_set_face_kernel(gb.DG_FACE_DWORD)
    c.dg_assemble()
    off, bptr, bcol, boff = c.dg_get_structure()
    vals, rhs = c.dg_get_matrix()
    rp, ci, v = dg_blocks_to_crs(off, bptr, bcol, boff, vals)
    B, R = O.dg_tet_assemble(t, F, p, A, pen=10.0, g=0.3, f=1.2)
    nd = off[-1]
    dense = np.zeros((nd, nd))
    for (i, j), K in B.items():
        dense[off[i]:off[i + 1], off[j]:off[j + 1]] = K
    ref = dense[np.repeat(np.arange(nd), np.diff(rp)), ci]
    assert sparse_rel_err(rp, ci, v, ref) < REL_TOL
    assert vec_rel_err(rhs, np.concatenate(R)) < REL_TOL


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("interior", [True, False])
def test_face_with_a_vertex_twice(gb, p, interior):
    """A face of no area (its first vertex named twice) has no normal: the
    blocks and load of its owners are NaN, every other row is untouched."""
    from modfem_gb300.mesh import structured_tet_mesh, tet_faces
    m = structured_tet_mesh(2, jitter=0.1, seed=p)
    F = tet_faces(m)
    f = int(np.flatnonzero((F.el2 >= 0) == interior)[5])
    owners = [int(e) for e in (F.el1[f], F.el2[f]) if e >= 0]

    def system(nodes):
        F.nodes[f, :3] = nodes
        c = gb.Context(0)
        c.set_mesh(m)
        c.set_coefficients(k=np.ones(m.nel), f=1.0, g=0.3)
        c.dg_set_degrees(np.full(m.nel, p))
        c.dg_set_faces(F, penalty=10.0)
        c.dg_build_structure()
        c.dg_assemble()
        out = c.dg_get_matrix() + tuple(c.dg_get_structure())
        c.close()
        return out

    nodes = F.nodes[f, :3].copy()
    v0, r0, off, bptr, bcol, boff = system(nodes)
    v1, r1 = system(nodes[[0, 0, 2]])[:2]
    for e in range(m.nel):
        touched = e in owners
        assert touched or np.array_equal(r0[off[e]:off[e + 1]], r1[off[e]:off[e + 1]])
        assert not touched or interior or np.all(np.isnan(r1[off[e]:off[e + 1]]))
        for b in range(bptr[e], bptr[e + 1]):
            x, y = v0[boff[b]:boff[b + 1]], v1[boff[b]:boff[b + 1]]
            if touched and bcol[b] in owners:
                assert np.all(np.isnan(y))
            else:
                assert np.array_equal(x, y)
