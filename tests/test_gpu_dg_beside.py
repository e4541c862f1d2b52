"""DG assembly on both sides of the limits of its rules (GPU): the face kernels
beside the volume kernels (up to 16,384 elements), one or two face points a
thread (155,648 points), the two forms of the block SpMV (a CTA a block row,
or eight lanes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import modfem_gb300 as g
    g.load_library()
    return g


def _context(gb, m, p, F, D):
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(D=D, f=1.0, g=0.3)
    c.dg_set_degrees(np.full(m.nel, p))
    c.dg_set_faces(F, penalty=10.0)
    c.dg_build_structure()
    c.dg_assemble()
    return c


@pytest.mark.parametrize("n,p", [(8, 1), (20, 1), (21, 1), (12, 2), (13, 2)])
def test_repeated_assembly_is_the_same(gb, n, p):
    """1,024 to 18,522 prisms: kernels beside one another write disjoint parts
    or wait, so five assemblies give the same bits."""
    from modfem_gb300.mesh import anisotropic_tensors, prism_faces, structured_prism_mesh
    m = structured_prism_mesh(n, jitter=0.1, seed=n)
    c = _context(gb, m, p, prism_faces(m), anisotropic_tensors(m.nel, seed=p).reshape(-1, 9))
    v, r = (a.copy() for a in c.dg_get_matrix())
    for _ in range(5):
        c.dg_set_matrix(np.full(c.dg_nval, np.nan), np.full(c.dg_ndof, np.nan))
        c.dg_assemble()
        w, s = c.dg_get_matrix()
        assert np.array_equal(v, w) and np.array_equal(r, s)


# block rows of one class just below and above the form's limit (prisms of
# degree 1: 512, 2: 6,656; tetrahedra of degree 2: 1,536)
@pytest.mark.parametrize("kind,p,n", [("prism", 1, 6), ("prism", 1, 7), ("prism", 2, 14), ("prism", 2, 15),
                                      ("tet", 1, 3), ("tet", 2, 6), ("tet", 2, 7), ("tet", 3, 5), ("tet", 4, 4)])
def test_block_products(gb, kind, p, n):
    """b - A x against the products of the downloaded blocks: each entry is a sum
    of at most 7 x 75 products, so two orders differ by less than 2 x 525 x 2^-53
    = 1.2e-13 of the sum of magnitudes."""
    from modfem_gb300.mesh import (anisotropic_tensors, prism_faces, structured_prism_mesh, structured_tet_mesh,
                                   tet_faces)
    m = structured_prism_mesh(n, jitter=0.1, seed=n) if kind == "prism" else structured_tet_mesh(n, jitter=0.1, seed=n)
    F = prism_faces(m) if kind == "prism" else tet_faces(m)
    c = _context(gb, m, p, F, anisotropic_tensors(m.nel, seed=p).reshape(-1, 9))
    vals, rhs = c.dg_get_matrix()
    off, bptr, bcol, boff = c.dg_get_structure()
    x = np.random.default_rng(n).standard_normal(c.dg_ndof)
    ref, mag = rhs.copy(), np.abs(rhs)
    ns = off[1]
    X = x.reshape(-1, ns)
    B = vals.reshape(-1, ns, ns)  # column-major blocks: B[k, j, i]
    rows = np.repeat(np.arange(m.nel), np.diff(bptr))
    y = np.einsum("kji,kj->ki", B, X[bcol])
    a = np.einsum("kji,kj->ki", np.abs(B), np.abs(X[bcol]))
    np.subtract.at(ref.reshape(-1, ns), rows, y)
    np.add.at(mag.reshape(-1, ns), rows, a)
    v = c.dg_compute_residual(x)
    assert np.all(np.abs(v - ref) <= 2 * 525 * 2.0**-53 * mag)


@pytest.mark.parametrize("kind,n", [("prism", 6), ("prism", 13), ("tet", 5), ("tet", 12)])
def test_block_products_of_mixed_degrees(gb, kind, n):
    """The same with degrees 1..4 mixed (the forms' limits follow the longest
    row): rows of at most 6 x 75 columns, 2 x 450 x 2^-53 = 1e-13."""
    import scipy.sparse as sp
    from modfem_gb300.mesh import prism_faces, structured_prism_mesh, structured_tet_mesh, tet_faces
    m = structured_prism_mesh(n, jitter=0.1, seed=n) if kind == "prism" else structured_tet_mesh(n, jitter=0.1, seed=n)
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=np.ones(m.nel), f=1.0, g=0.3)
    c.dg_set_degrees(np.random.default_rng(n).integers(1, 5, m.nel))
    c.dg_set_faces(prism_faces(m) if kind == "prism" else tet_faces(m), penalty=10.0)
    c.dg_build_structure()
    c.dg_assemble()
    vals, rhs = c.dg_get_matrix()
    off, bptr, bcol, boff = c.dg_get_structure()
    I, J, V = [], [], []
    for e in range(m.nel):
        ns = off[e + 1] - off[e]
        lo, hi = boff[bptr[e]], boff[bptr[e + 1]]
        cols = np.concatenate([np.arange(off[f], off[f + 1]) for f in bcol[bptr[e]:bptr[e + 1]]])
        I.append(np.tile(np.arange(off[e], off[e + 1]), cols.size))
        J.append(np.repeat(cols, ns))
        V.append(vals[lo:hi])
    A = sp.csr_matrix((np.concatenate(V), (np.concatenate(I), np.concatenate(J))))
    x = np.random.default_rng(n).standard_normal(c.dg_ndof)
    v = c.dg_compute_residual(x)
    assert np.all(np.abs(v - (rhs - A @ x)) <= 2 * 451 * 2.0**-53 * (np.abs(rhs) + abs(A) @ np.abs(x)))
