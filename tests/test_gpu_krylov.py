"""The vector kernels of the DG Krylov loop at the edges of their tiles (GPU):
row counts on both sides of the 1,024 rows of a block and the 512 of a dot
product, one to nineteen basis vectors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import modfem_gb300 as g
    g.load_library()
    return g


@pytest.fixture(scope="module", params=[(1, 1), (1, 2), (2, 2), (3, 1), (3, 2), (4, 1), (4, 2), (5, 1)])
def system(gb, request):
    from modfem_gb300.mesh import lognormal_k, prism_faces, structured_prism_mesh
    n, p = request.param
    m = structured_prism_mesh(n, jitter=0.1, seed=n)
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=lognormal_k(m.nel, seed=p), f=1.0, g=0.3)
    c.dg_set_degrees(np.full(m.nel, p))
    c.dg_set_faces(prism_faces(m), penalty=10.0)
    c.dg_build_structure()
    c.dg_assemble()
    vals, rhs = c.dg_get_matrix()
    off, bptr, bcol, boff = c.dg_get_structure()
    A = np.zeros((off[-1], off[-1]))
    P = np.zeros_like(A)
    for e in range(m.nel):
        ns = off[e + 1] - off[e]
        for b in range(bptr[e], bptr[e + 1]):
            f = bcol[b]
            B = vals[boff[b]:boff[b] + ns * (off[f + 1] - off[f])].reshape(-1, ns).T
            A[off[e]:off[e + 1], off[f]:off[f + 1]] = B
            if f == e:
                P[off[e]:off[e + 1], off[e]:off[e + 1]] = np.linalg.inv(B)
    return c, P @ A, P @ rhs


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17, 19])
def test_cycle_reaches_the_least_residual(system, k):
    """One cycle of k steps leaves the least |M^-1 (b - A x)| over the Krylov
    space, as numpy's least squares over an orthonormal basis finds it, and the
    x it returns has that residual.  Classical Gram-Schmidt over at most 19
    vectors loses digits with the square of the basis' condition, a few 1e2
    while the residual falls by less than that: 1e5 x 1e-16, held to 1e-9 of the
    first residual."""
    c, MA, Mb = system
    beta = np.linalg.norm(Mb)
    V = [Mb / beta]
    for _ in range(k):
        w = MA @ V[-1]
        for _ in range(2):
            for v in V:
                w = w - (v @ w) * v
        if np.linalg.norm(w) < 1e-10:
            break
        V.append(w / np.linalg.norm(w))
    B = MA @ np.stack(V[:k], 1)
    least = np.linalg.norm(Mb - B @ np.linalg.lstsq(B, Mb, rcond=None)[0])
    x, it, res, rel = c.dg_solve(krylov=k, max_iter=k, tol_rel=1e-12)
    assert it <= k
    assert abs(res - least) <= 1e-9 * beta
    assert abs(np.linalg.norm(Mb - MA @ x) - least) <= 1e-9 * beta
