"""The moment form of the DG prism kernels at the edges of their tiles (GPU),
against the oracle's sums over the quadrature points."""
import numpy as np
import pytest

from _util import REL_TOL, mat_rel_err, vec_rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import modfem_gb300 as g
    g.load_library()
    return g


@pytest.mark.parametrize("p,count", [(1, 1), (1, 31), (1, 33), (2, 11), (2, 13), (3, 1), (3, 5), (4, 1), (4, 3)])
def test_volume_tiles_vs_oracle(gb, p, count):
    """Fewer elements than a tile, one more than a tile, every launch variant:
    blocks and loads within the FP64 tolerance of the oracle and the same bits
    from every variant."""
    import oracle as O
    from modfem_gb300.mesh import anisotropic_tensors, structured_prism_mesh
    m = structured_prism_mesh(3, jitter=0.2, seed=p)
    X = m.coords[m.el_nodes[:count]]
    A = anisotropic_tensors(count, seed=count).reshape(count, 3, 3)
    b = gb.Batch(0)
    b.set(X, A, np.full(count, p), np.zeros((0, 4, 3)), np.zeros((0, 3, 3)), np.zeros(0, np.int32), f=0.7)
    ref = None
    for v in range(3):
        b.set_variants([0] + [v] * 4, None)
        b.run()
        mats, loads = b.blocks()
        out = b.get()
        if ref is None:
            ref = out
        assert np.array_equal(out[0], ref[0]) and np.array_equal(out[1], ref[1])
        for e in range(count):
            K, R = O.dg_prism_element(X[e], A[e], p, 0.7)
            assert mat_rel_err(mats[e], K) < REL_TOL
            assert vec_rel_err(loads[e], R) < REL_TOL
    b.close()


def _system(gb, m, F, p, D, mode=0):
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(D=D, f=1.0, g=0.4)
    c.dg_set_degrees(p)
    c.dg_set_faces(F, penalty=10.0)
    c.dg_build_structure()
    c.dg_set_face_kernel(mode)
    c.dg_assemble()
    vals, rhs = c.dg_get_matrix()
    off, bptr, bcol, boff = c.dg_get_structure()
    A = np.zeros((off[-1], off[-1]))
    for e in range(m.nel):
        ns = off[e + 1] - off[e]
        for b in range(bptr[e], bptr[e + 1]):
            j0, j1 = off[bcol[b]], off[bcol[b] + 1]
            A[off[e]:off[e + 1], j0:j1] = vals[boff[b]:boff[b + 1]].reshape(j1 - j0, ns).T
    c.close()
    return A, rhs


def _oracle_system(m, F, p, D):
    import oracle as O
    rp, ci, val, rhs, off = O.dg_assemble(m, F, p, D, pen=10.0, g=0.4)
    A = np.zeros((off[-1], off[-1]))
    for i in range(off[-1]):
        A[i, ci[rp[i]:rp[i + 1]]] = val[rp[i]:rp[i + 1]]
    return A, rhs


def _check(A, rhs, Ao, ro):
    R, C = np.abs(Ao).max(1), np.abs(Ao).max(0)
    assert np.max(np.abs(A - Ao) / np.sqrt(np.outer(R, C))) < REL_TOL
    assert vec_rel_err(rhs, ro) < REL_TOL


@pytest.mark.parametrize("p1,p2", [(1, 1), (1, 4), (2, 3), (3, 3), (4, 2), (4, 4)])
def test_face_blocks_vs_oracle(gb, p1, p2):
    """Two degrees side by side in both orders (every face bucket, ragged
    blocks), vertices of each prism's triangle rotated and the prism turned
    upside down at random, so that every edge, direction and triangle
    permutation occurs."""
    from modfem_gb300.mesh import anisotropic_tensors, mixed_faces, structured_prism_mesh
    m = structured_prism_mesh(2, jitter=0.2, seed=3 * p1 + p2)
    rng = np.random.default_rng(10 * p1 + p2)
    el = m.el_nodes.copy()
    for e in range(m.nel):
        r = rng.integers(3)
        t = [(i + r) % 3 for i in range(3)]
        # upside down: top and bottom swapped, orientation kept by reversing the triangle
        order = t + [3 + i for i in t] if rng.integers(2) else [3 + i for i in t[::-1]] + t[::-1]
        el[e] = el[e][order]
    m.el_nodes = el
    m.el_nv = np.full(m.nel, 6, np.int32)
    F = mixed_faces(m)
    p = np.where(rng.integers(2, size=m.nel) > 0, p1, p2).astype(np.int32)
    D = anisotropic_tensors(m.nel, seed=p1).reshape(m.nel, 9)
    Ao, ro = _oracle_system(m, F, p, D)
    for mode in (gb.DG_FACE_FP64, gb.DG_FACE_TC_DWORD):
        _check(*_system(gb, m, F, p, D, mode), Ao, ro)


@pytest.mark.parametrize("p1,p2", [(1, 2), (3, 3), (4, 3)])
def test_turned_quadrilateral_vs_oracle(gb, p1, p2):
    """Two prisms sharing a quadrilateral turned by 90 degrees (the edge of one
    triangle is the zeta direction of the other): the moment form does not
    cover it, the sums over the points do, in every face mode."""
    from modfem_gb300.mesh import MixedMesh, anisotropic_tensors, mixed_faces
    X = np.array([[0, 0, 0], [1, 0, 0.1], [0.1, 1, 0], [0, 0, 1], [1, 0, 1.1], [0, 1.1, 1], [0, -1, 0.2], [1, -1.1, 0.3]])
    el = np.array([[0, 1, 2, 3, 4, 5], [0, 3, 6, 1, 4, 7]], np.int32)
    m = MixedMesh(1, X, el, np.full(2, 6, np.int32), 1)
    F = mixed_faces(m)
    assert np.sum(F.el2 >= 0) == 1
    p = np.array([p1, p2], np.int32)
    D = anisotropic_tensors(2, seed=p1).reshape(2, 9)
    Ao, ro = _oracle_system(m, F, p, D)
    for mode in (gb.DG_FACE_FP64, gb.DG_FACE_DWORD):
        _check(*_system(gb, m, F, p, D, mode), Ao, ro)


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_coefficient_that_is_not_finite_shows(gb, p, bad):
    """One prism's coefficient NaN or infinite: nothing finite is left in its
    own block, its neighbours' blocks with it and, on the boundary, its load; all else
    is what it is beside a prism of coefficient 1."""
    from modfem_gb300.mesh import prism_faces, structured_prism_mesh
    m = structured_prism_mesh(3, jitter=0.2, seed=p)
    F = prism_faces(m)

    def system(e, k):
        c = gb.Context(0)
        c.set_mesh(m)
        kk = np.ones(m.nel)
        kk[e] = k
        c.set_coefficients(k=kk, f=1.0, g=0.4)
        c.dg_set_degrees(np.full(m.nel, p))
        c.dg_set_faces(F, penalty=10.0)
        c.dg_build_structure()
        c.dg_assemble()
        out = [np.array(a) for a in c.dg_get_matrix()], c.dg_get_structure()
        c.close()
        return out

    inner = int(np.flatnonzero(~np.isin(np.arange(m.nel), F.el1[F.el2 < 0]))[0])
    for e, boundary in ((inner, False), (int(F.el1[F.el2 < 0][0]), True)):
        (v1, r1), (off, bptr, bcol, boff) = system(e, 1.0)
        (v, r), _ = system(e, bad)
        for i in range(m.nel):
            assert np.array_equal(r[off[i]:off[i + 1]], r1[off[i]:off[i + 1]]) or (i == e and boundary)
            for b in range(bptr[i], bptr[i + 1]):
                x, x1 = v[boff[b]:boff[b + 1]], v1[boff[b]:boff[b + 1]]
                if e in (i, bcol[b]):
                    assert not np.any(np.isfinite(x)), (i, bcol[b])
                else:
                    assert np.array_equal(x, x1)
        assert not boundary or not np.any(np.isfinite(r[off[e]:off[e + 1]]))


@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_a_face_without_a_normal_shows(gb, p):
    """A corner of the mesh moved onto another vertex of its boundary triangle (no
    area, no normal; the element itself keeps a volume): nothing finite in
    that element's own block and load, as from the sums over the points."""
    from modfem_gb300.mesh import prism_faces, structured_prism_mesh
    m = structured_prism_mesh(3)
    F = prism_faces(m)
    m.coords = m.coords.copy()
    m.coords[1] = m.coords[0]
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=np.ones(m.nel), f=1.0, g=0.4)
    c.dg_set_degrees(np.full(m.nel, p))
    c.dg_set_faces(F, penalty=10.0)
    c.dg_build_structure()
    c.dg_assemble()
    v, r = c.dg_get_matrix()
    off, bptr, bcol, boff = c.dg_get_structure()
    c.close()
    flat = [f for f in range(F.n) if F.type[f] == 3 and {0, 1} <= set(F.nodes[f, :3].tolist())]
    assert len(flat) == 1 and F.el2[flat[0]] < 0
    e = int(F.el1[flat[0]])
    d = bptr[e] + int(np.flatnonzero(bcol[bptr[e]:bptr[e + 1]] == e)[0])
    assert not np.any(np.isfinite(v[boff[d]:boff[d + 1]])) and not np.any(np.isfinite(r[off[e]:off[e + 1]]))
    others = np.ones(len(v), bool)
    others[boff[bptr[e]]:boff[bptr[e + 1]]] = False
    assert np.all(np.isfinite(v[others]))
