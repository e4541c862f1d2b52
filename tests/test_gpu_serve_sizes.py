"""The serving engine's step on both sides of its reduction chunks (GPU):
batched requests of one row chunk, of many, and of more rows than chunks of the
smallest size cover; and contexts kept from earlier requests of other sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    from modfem_gb300 import build
    build.build(verbose=False)
    import modfem_gb300
    return modfem_gb300


def _plain(gb, m, k, **kw):
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=k, f=1.0, g=0.0)
    c.build_structure_device()
    c.assemble(gb.SCATTER_GATHER)
    out = c.solve(**kw)
    c.close()
    return out


def test_batched_requests_of_all_sizes(gb):
    """8 to 46,656 unknowns in one mix, none solved alone, twice (the second
    time in contexts that served other sizes): the same bits both times and the plain
    path's x: after the same number of steps both minimise the same residual over the
    same space, and rounding in 20 steps stays far below 1e-8 of x."""
    from modfem_gb300.mesh import lognormal_k, structured_prism_mesh
    from modfem_gb300.serve import STD, Problem, Server, dof_count
    its = 20
    probs = []
    for n in (1, 5, 7, 16, 34, 35):
        m = structured_prism_mesh(n, jitter=0.2, seed=n)
        k = lognormal_k(m.nel, seed=n)
        probs.append((m, k, Problem(m, k, kind=STD, f=1.0, g=0.0, krylov=30, max_iter=its, tol=1e-10)))
    srv = Server(0, max_active=16, prep_threads=2)
    try:
        srv.set_solo_dofs(10**9)
        runs = []
        for order in (range(6), (5, 4, 3, 2, 1, 0)):
            ids = {i: srv.submit(probs[i][2]) for i in order}
            res = {}
            for i, rid in ids.items():
                assert srv.wait(rid, 120.0) == 1
                res[i] = srv.result(rid, dof_count(probs[i][2]))
                srv.release(rid)
            runs.append(res)
    finally:
        srv.close()
    for i, (m, k, pr) in enumerate(probs):
        (xa, ia, _, _), (xb, ib, _, _) = runs[0][i], runs[1][i]
        assert ia == ib and np.array_equal(xa, xb)
        x, it, _, _ = _plain(gb, m, k, krylov=30, max_iter=its, tol_rel=1e-10)
        assert it == ia
        assert np.max(np.abs(x - xa)) <= 1e-8 * np.max(np.abs(x))


@pytest.mark.parametrize("n", [32, 33])
def test_std_gmres_around_the_small_system_limit(gb, n):
    """35,937 and 39,304 rows (dots in the SpMV kernel up to 38,912): the residual
    that one cycle of 30 reports is that of the x it returns, computed
    in numpy, to 1e-9 of the first (30 steps lose a few digits of orthogonality
    at most)."""
    import scipy.sparse as sp
    from modfem_gb300.mesh import lognormal_k, structured_prism_mesh
    m = structured_prism_mesh(n, jitter=0.2, seed=n)
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=lognormal_k(m.nel, seed=n), f=1.0, g=0.0)
    c.build_structure_device()
    c.assemble(gb.SCATTER_GATHER)
    _, rp, ci = c.get_crs_structure()
    val, rhs = c.get_matrix()
    A = sp.csr_matrix((val, ci, rp))
    d = 1.0 / A.diagonal()
    for steps in (1, 2, 7, 8, 9, 15, 16, 17, 30):
        x, it, res, _ = c.solve(30, steps, 1e-12)
        assert it == steps
        r = np.linalg.norm(d * (rhs - A @ x))
        assert abs(r - res) <= 1e-9 * np.linalg.norm(d * rhs)
