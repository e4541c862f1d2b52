"""DG block products of classes with more rows than the CTA-a-row form takes (GPU):
groups of eight lanes a row, in FP64, for every block class, with the residual
and with the block Jacobi product, and row counts that do not fill a CTA of 32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import modfem_gb300 as g
    g.load_library()
    return g


def _faces(F, keep):
    class Part:
        pass
    t = Part()
    for a in ("type", "bc", "el1", "el2", "side1", "nodes"):
        setattr(t, a, getattr(F, a)[keep])
    return t


def _context(gb, m, p, F):
    from modfem_gb300.mesh import lognormal_k
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=lognormal_k(m.nel, seed=m.nel), f=1.0, g=0.3)
    c.dg_set_degrees(p)
    c.dg_set_faces(F, penalty=10.0)
    c.dg_build_structure()
    c.dg_assemble()
    return c


# (rows from which the groups take the class: prisms 512, 6,656, 10,000, 13,000; tetrahedra of
# degree 2..4 1,536, 6,144, 8,192, of degree 1 by the longest row).  Prisms of degree 4 with their
# triangles only: 1.8 GB of matrix.
@pytest.mark.parametrize("kind,p,n", [("prism", 1, 7), ("prism", 2, 15), ("prism", 3, 18), ("prism", 4, 19),
                                      ("tet", 1, 7), ("tet", 2, 7), ("tet", 3, 11), ("tet", 4, 13)])
def test_products_by_groups_of_lanes(gb, kind, p, n):
    """b - A x against the downloaded blocks: sums of up to 451 terms in two orders,
    2 x 451 x 2^-53 = 1e-13 of the sum of magnitudes.  And the residual that a GMRES
    cycle reports after its steps is that of the x it returns, Minv (b - A x) with the
    diagonal blocks solved in numpy, to 1e-9 of the first (a few steps lose few digits)."""
    from modfem_gb300.mesh import prism_faces, structured_prism_mesh, structured_tet_mesh, tet_faces
    m = structured_prism_mesh(n, jitter=0.1, seed=n) if kind == "prism" else structured_tet_mesh(n, jitter=0.1, seed=n)
    F = prism_faces(m) if kind == "prism" else tet_faces(m)
    if (kind, p) == ("prism", 4):
        F = _faces(F, F.type == 3)
    c = _context(gb, m, np.full(m.nel, p), F)
    vals, rhs = c.dg_get_matrix()
    off, bptr, bcol, _ = c.dg_get_structure()
    ns, rows = off[1], np.repeat(np.arange(m.nel), np.diff(bptr))
    limit = {"prism": [0, 512, 6656, 10000, 13000], "tet": [0, 0, 1536, 6144, 8192]}[kind][p]
    assert m.nel > limit and m.nel % 32
    B = vals.reshape(-1, ns, ns)  # column-major blocks: B[k, j, i]

    def product(x, mag=False):
        X = (np.abs(x) if mag else x).reshape(-1, ns)[bcol]
        y = np.zeros((m.nel, ns))
        for lo in range(0, len(bcol), 4096):  # (no copy of the whole matrix)
            b = B[lo:lo + 4096]
            np.add.at(y, rows[lo:lo + 4096], np.matmul(X[lo:lo + 4096, None, :], np.abs(b) if mag else b)[:, 0])
        return y.ravel()

    x = np.random.default_rng(n).standard_normal(c.dg_ndof)
    err = np.abs(c.dg_compute_residual(x) - (rhs - product(x)))
    assert np.all(err <= 2 * 451 * 2.0**-53 * (np.abs(rhs) + product(x, True)))
    diag = B[[int(bptr[e] + np.flatnonzero(bcol[bptr[e]:bptr[e + 1]] == e)[0]) for e in range(m.nel)]].transpose(0, 2, 1)
    first = np.linalg.norm(np.linalg.solve(diag, rhs.reshape(-1, ns, 1)))
    for steps in (1, 3):
        x, it, res, _ = c.dg_solve(10, steps, 1e-14)
        r = np.linalg.norm(np.linalg.solve(diag, (rhs - product(x)).reshape(-1, ns, 1)))
        assert it == steps and abs(r - res) <= 1e-9 * first
    c.close()


@pytest.mark.parametrize("p,n,share", [(1, 16, 0.05), (2, 22, 0.03)])
def test_products_by_groups_of_lanes_in_mixed_rows(gb, p, n, share):
    """One class with more rows than its longest one allows the CTA form, a few
    elements of degree 4 among them, so that its rows differ in length; sampled block
    rows, to the same tolerance."""
    from modfem_gb300.mesh import prism_faces, structured_prism_mesh
    m = structured_prism_mesh(n, jitter=0.1, seed=n)
    pd = np.where(np.random.default_rng(n).random(m.nel) < share, 4, p)
    c = _context(gb, m, pd, prism_faces(m))
    vals, rhs = c.dg_get_matrix()
    off, bptr, bcol, boff = c.dg_get_structure()
    width = np.array([np.sum(off[bcol[a:b] + 1] - off[bcol[a:b]]) for a, b in zip(bptr[:-1], bptr[1:])])
    cls = np.flatnonzero(pd == p)
    base, own = {1: (512, 36), 2: (6656, 108)}[p]
    assert cls.size > base * width[cls].max() // own
    x = np.random.default_rng(p).standard_normal(c.dg_ndof)
    v = c.dg_compute_residual(x)
    c.close()
    longest = cls[np.argsort(-width[cls], kind="stable")]
    for e in np.concatenate([longest[:64], longest[-64:], np.random.default_rng(1).choice(m.nel, 400)]):
        r, mag = rhs[off[e]:off[e + 1]].copy(), np.abs(rhs[off[e]:off[e + 1]])
        for b in range(bptr[e], bptr[e + 1]):
            A = vals[boff[b]:boff[b + 1]].reshape(-1, off[e + 1] - off[e]).T
            y = x[off[bcol[b]]:off[bcol[b] + 1]]
            r -= A @ y
            mag += np.abs(A) @ np.abs(y)
        assert np.all(np.abs(v[off[e]:off[e + 1]] - r) <= 2 * 451 * 2.0**-53 * mag)
