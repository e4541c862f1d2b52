"""The block Jacobi inverses of every block class (GPU): blocks that need
their pivots from far rows, group counts that do not fill a CTA, a singular
block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import modfem_gb300 as g
    g.load_library()
    return g


def _context(gb, kind, p, count):
    """A DG context of `count` elements and no faces: a block diagonal matrix."""
    from modfem_gb300.mesh import structured_prism_mesh, structured_tet_mesh
    m = structured_prism_mesh(3) if kind == "prism" else structured_tet_mesh(2)

    class Part:
        coords, el_nodes = m.coords, m.el_nodes[:count]
        nno, nel = len(m.coords), count

    c = gb.Context(0)
    c.set_mesh(Part)
    c.set_coefficients(k=np.ones(count))
    c.dg_set_degrees(np.full(count, p))
    c.dg_build_structure()
    return c


CASES = [("prism", 1, 17), ("prism", 2, 3), ("prism", 2, 5), ("prism", 3, 1), ("prism", 3, 7), ("prism", 4, 1),
         ("prism", 4, 3), ("tet", 1, 33), ("tet", 2, 9), ("tet", 3, 5), ("tet", 4, 1), ("tet", 4, 6)]


def _blocks(c, rng):
    """Permutation + 0.3 / n noise with zeros on the diagonal: condition below
    (1 + 0.3) / (1 - 0.3) = 2 in the 2-norm, no pivot where a plain elimination
    looks first."""
    off, bptr, bcol, boff = c.dg_get_structure()
    vals = np.zeros(c.dg_nval)
    D = []
    for e in range(len(off) - 1):
        n = off[e + 1] - off[e]
        a = np.roll(np.eye(n), 1 + e % (n - 1), axis=0) * rng.choice([-1.0, 1.0], n)
        a += rng.uniform(-0.3 / n, 0.3 / n, (n, n)) * (1 - np.eye(n))
        k = next(k for k in range(bptr[e], bptr[e + 1]) if bcol[k] == e)
        vals[boff[k]:boff[k] + n * n] = a.T.reshape(-1)
        D.append((off[e], k, a))
    return vals, D, boff


@pytest.mark.parametrize("kind,p,count", CASES)
def test_block_diagonal_solve(gb, kind, p, count):
    """A = its diagonal blocks: one iteration gives A^-1 b, to the error of the
    inversion, below n^2 2^-53 cond max|x| < 75^2 x 1.1e-16 x 2 < 2e-12 max|x|."""
    c = _context(gb, kind, p, count)
    rng = np.random.default_rng(p + 10 * count)
    vals, D, _ = _blocks(c, rng)
    b = rng.standard_normal(c.dg_ndof)
    c.dg_set_matrix(vals, b)
    x = c.dg_solve(krylov=5, max_iter=3, tol_rel=1e-10)[0]
    for o, _, a in D:
        n = len(a)
        ref = np.linalg.solve(a, b[o:o + n])
        assert np.max(np.abs(x[o:o + n] - ref)) <= 2e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("kind,p,count", CASES)
def test_singular_block_is_refused(gb, kind, p, count):
    c = _context(gb, kind, p, count)
    vals, D, boff = _blocks(c, np.random.default_rng(1))
    o, k, a = D[count // 2]
    n = len(a)
    a = a.copy()
    a[:, n - 1] = 0.0
    vals[boff[k]:boff[k] + n * n] = a.T.reshape(-1)
    c.dg_set_matrix(vals, np.ones(c.dg_ndof))
    with pytest.raises(Exception, match="singular diagonal block"):
        c.dg_solve(krylov=5, max_iter=3, tol_rel=1e-10)
