"""The gather scatter and the device structure at the edges of their rules:
rows longer than the shared row sums (40 columns), incidence lists longer than
a warp (32), rows at the column limit (256), several penalty faces on an
element, elements that list a vertex twice, tetrahedra.

The reference is the atomic scatter of the same context: the element and face
arithmetic is the same, only the order of the additions differs.  An entry is
a sum of at most m <= 256 contributions, each below sqrt(K_rr K_cc) in sum
(Cauchy-Schwarz over the elements), so two orders differ by at most
2 m 2^-53 = 6e-14 of that.
"""
import numpy as np
import pytest

from _util import energy_scale

pytestmark = pytest.mark.gpu
TOL = 2 * 256 * 2.0**-53


@pytest.fixture(scope="module")
def gb():
    from modfem_gb300 import build
    build.build(verbose=False)
    import modfem_gb300
    return modfem_gb300


class M:
    def __init__(self, coords, el, faces=()):
        self.coords, self.el_nodes = np.asarray(coords, float), np.asarray(el, np.int32)
        self.nno, self.nel = len(self.coords), len(self.el_nodes)
        if faces:
            fa = np.asarray(faces, np.int32)
            self.bc_face_id = np.arange(1, len(fa) + 1, dtype=np.int32)
            self.bc_face_el, self.bc_face_side = fa[:, 0].copy(), fa[:, 1].copy()
            self.bc_face_bc = np.ones(len(fa), np.int32)


def fan(n, kind, faces=()):
    """n prisms (or tetrahedra) around one edge: its vertices have n elements."""
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(a), np.sin(a)], 1) * (1 + 0.1 * np.cos(5 * a))[:, None]
    lo = np.c_[np.vstack([[0, 0], ring]), np.zeros(n + 1)]
    if kind == "prism":
        hi = lo + [0.05, -0.02, 1.0]
        el = [[0, 1 + i, 1 + (i + 1) % n, n + 1, n + 2 + i, n + 2 + (i + 1) % n] for i in range(n)]
        return M(np.vstack([lo, hi]), el, faces)
    return M(np.vstack([lo, [[0.1, 0.0, 1.0]]]), [[0, 1 + i, 1 + (i + 1) % n, n + 1] for i in range(n)])


def check(gb, m, mode, host=True):
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=np.random.default_rng(3).lognormal(size=m.nel), f=1.0, g=0.5 if m.el_nodes.shape[1] == 6 else 0.0,
                       penalty=1e3)
    if host:
        c.build_structure()
        h = c.get_crs_structure() + (c.get_element_tables(),)
    c.build_structure_device()
    d = c.get_crs_structure() + (c.get_element_tables(),)
    if host:
        for x, y in zip(h, d):
            assert np.array_equal(x, y)
    rp, ci = d[1], d[2]
    c.assemble(gb.SCATTER_ATOMIC)
    va, ra = (x.copy() for x in c.get_matrix())
    c.assemble(mode)
    v1, r1 = (x.copy() for x in c.get_matrix())
    c.assemble(mode)
    v2, r2 = c.get_matrix()
    assert np.array_equal(v1, v2) and np.array_equal(r1, r2)
    assert np.all(np.abs(v1 - va) <= TOL * energy_scale(rp, ci, va))
    assert np.all(np.abs(r1 - ra) <= TOL * np.abs(ra))


@pytest.mark.parametrize("n", [3, 19, 20, 32, 33, 126])
def test_prism_fans(gb, n):
    check(gb, fan(n, "prism", [(0, s) for s in (4, 0, 2, 1, 3)] + [(e, 3) for e in range(1, n)]), gb.SCATTER_GATHER)


@pytest.mark.parametrize("n", [3, 32, 33, 100])
def test_tet_fans_colour(gb, n):
    check(gb, fan(n, "tet"), gb.SCATTER_COLOR)


def test_one_element(gb):
    check(gb, M(fan(5, "prism").coords, [[0, 1, 2, 6, 7, 8]], [(0, 1)]), gb.SCATTER_GATHER)
    check(gb, M(fan(5, "tet").coords, [[0, 1, 2, 6]]), gb.SCATTER_COLOR)


def test_element_with_a_vertex_twice(gb):
    """Prisms whose upper triangle shares a vertex with the lower one."""
    m = fan(6, "prism", [(0, 0), (0, 1), (0, 4), (2, 2)])
    el = m.el_nodes.copy()
    el[:, 3] = el[:, 0]
    check(gb, M(m.coords, el, [(0, 0), (0, 1), (0, 4), (2, 2)]), gb.SCATTER_GATHER, host=False)


def test_too_many_neighbours_are_refused(gb):
    c = gb.Context(0)
    m = fan(128, "prism")
    c.set_mesh(m)
    c.set_coefficients(k=np.ones(m.nel))
    with pytest.raises(Exception, match="more neighbours"):
        c.build_structure_device()
