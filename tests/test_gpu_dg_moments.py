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
