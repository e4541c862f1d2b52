"""The serving engine's memory accounting (GPU): what a request is admitted
with against what it then holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import modfem_gb300 as g
    g.load_library()
    return g


def _krylov_bytes(n, m):
    """A lane's Krylov space: x, tmp, m + 1 vectors, Hessenberg matrix, six rows."""
    m1 = m + 1
    return 8 * (n * (m1 + 2) + m1 * m1 + 6 * (m1 + 1))


@pytest.mark.parametrize("krylov", [10, 60])
@pytest.mark.parametrize("n", [1, 5, 20, 40])
def test_std_footprint_covers_what_is_held(gb, n, krylov):
    """In a lane (CRS rows, a Krylov space of its own) and alone (sliced-ELL
    copy and the context's vectors)."""
    from modfem_gb300.mesh import structured_prism_mesh
    from modfem_gb300.serve import STD, Problem
    m = structured_prism_mesh(n, jitter=0.1, seed=n)
    pr = Problem(m, np.ones(m.nel), kind=STD, krylov=krylov)
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=pr.k, f=1.0)
    c.build_structure_device()
    c.assemble(gb.SCATTER_GATHER)
    lane = c.device_bytes() + 8 * m.nno + _krylov_bytes(m.nno, krylov)
    c.solve(krylov, krylov, 1e-12)
    alone = c.device_bytes()
    c.close()
    assert max(lane, alone) <= pr.footprint(), (lane, alone, pr.footprint())


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 4, 12])
def test_dg_footprint_covers_what_is_held(gb, n, p):
    from modfem_gb300.mesh import prism_faces, structured_prism_mesh
    from modfem_gb300.serve import DG, Problem
    m = structured_prism_mesh(n, jitter=0.1, seed=n)
    F = prism_faces(m)
    pr = Problem(m, np.ones(m.nel), kind=DG, p=p, faces=F, krylov=30)
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=pr.k, f=1.0)
    c.dg_set_degrees(np.full(m.nel, p))
    c.dg_set_faces(F, penalty=10.0)
    c.dg_build_structure()
    c.dg_assemble()
    ns = c.dg_ndof // m.nel
    held = c.device_bytes() + 8 * ns * ns * m.nel + _krylov_bytes(c.dg_ndof, 30)
    c.close()
    assert held <= pr.footprint(), (held, pr.footprint())


def test_small_request_in_a_large_context_is_charged_for_it(gb):
    """A solo request of 2,197 unknowns in the context that one of 68,921 has
    left: while it is solved, the charge covers what the larger context holds
    (at least its local matrices, 336 B a prism, and its 31 Krylov vectors)."""
    import time
    from modfem_gb300.mesh import lognormal_k, structured_prism_mesh
    from modfem_gb300.serve import STD, Problem, Server
    big, small = structured_prism_mesh(40), structured_prism_mesh(12)
    held = 336 * big.nel + 8 * 31 * big.nno
    srv = Server(0, prep_threads=1)
    try:
        srv.set_solo_dofs(1000)
        rid = srv.submit(Problem(big, np.ones(big.nel), kind=STD, krylov=30, max_iter=5, tol=1e-10))
        assert srv.wait(rid, 120.0) == 1
        # (20,000 restarts of one vector: some 0.5 s)
        rid = srv.submit(Problem(small, lognormal_k(small.nel, seed=1), kind=STD, krylov=1, max_iter=20000, tol=1e-12))
        end = time.time() + 60.0
        while srv.stats()["active"] == 0 and time.time() < end:
            time.sleep(1e-3)
        st = srv.stats()
        assert srv.wait(rid, 120.0) == 1
    finally:
        srv.close()
    assert st["active"] == 1 and held <= st["bytes"] <= st["budget"]


def _free():
    import ctypes
    cu = ctypes.CDLL("libcuda.so.1")
    free, total = ctypes.c_size_t(), ctypes.c_size_t()
    assert cu.cuMemGetInfo_v2(ctypes.byref(free), ctypes.byref(total)) == 0
    return free.value


def test_a_request_that_must_wait_drops_no_kept_context(gb):
    """A kept DG context (16 MB of matrix and more), a request in flight and one
    that does not fit beside it: the kept context stays while that one waits."""
    import time
    from modfem_gb300.mesh import lognormal_k, prism_faces, structured_prism_mesh
    from modfem_gb300.serve import DG, STD, Problem, Server
    d, m = structured_prism_mesh(8), structured_prism_mesh(48)
    kept = Problem(d, np.ones(d.nel), kind=DG, p=2, faces=prism_faces(d), krylov=10, max_iter=5)
    large = Problem(m, lognormal_k(m.nel, seed=1), kind=STD, krylov=1, max_iter=15000, tol=1e-12)  # over a second
    budget = max(int(1.5 * large.footprint()), 8 * kept.footprint())
    assert 2 * large.footprint() > budget
    srv = Server(0, hbm_budget=budget, prep_threads=1)
    try:
        rid = srv.submit(kept)
        assert srv.wait(rid, 120.0) == 1
        first = srv.submit(large)
        end = time.time() + 60.0
        while srv.stats()["active"] == 0 and time.time() < end:
            time.sleep(1e-3)
        time.sleep(0.2)  # its buffers are there
        before = _free()
        second = srv.submit(large)
        time.sleep(0.2)
        after, st = _free(), srv.stats()
        assert srv.wait(first, 120.0) == 1 and srv.wait(second, 120.0) == 1
    finally:
        srv.close()
    assert st["active"] == 1 and st["queued"] == 1
    assert after - before <= 8 * 2**20


def test_requests_that_need_the_kept_contexts_room_are_served(gb):
    """Std and DG requests of nearly the whole budget in turn, small ones between
    them: each large one waits until the contexts kept from the small ones have been
    freed, is admitted then, and nothing stays charged."""
    from modfem_gb300.mesh import prism_faces, structured_prism_mesh
    from modfem_gb300.serve import DG, STD, Problem, Server
    s, d = structured_prism_mesh(24), structured_prism_mesh(12)
    large = [Problem(s, np.ones(s.nel), kind=STD, krylov=30, max_iter=20, tol=1e-10),
             Problem(d, np.ones(d.nel), kind=DG, p=1, faces=prism_faces(d), krylov=30, max_iter=20, tol=1e-10)]
    t = structured_prism_mesh(6)
    small = [Problem(t, np.ones(t.nel), kind=STD, max_iter=20),
             Problem(t, np.ones(t.nel), kind=DG, p=1, faces=prism_faces(t), max_iter=20)]
    budget = max(p.footprint() for p in large) + min(p.footprint() for p in small)
    srv = Server(0, hbm_budget=budget, prep_threads=2)
    try:
        for _ in range(5):
            ids = [srv.submit(p) for p in small + large]
            for rid in ids:
                assert srv.wait(rid, 60.0) == 1
        st = srv.stats()
    finally:
        srv.close()
    assert st["bytes"] == 0 and st["queued"] == 0 and st["peak_bytes"] <= budget
