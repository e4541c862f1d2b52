"""DG systems whose prism faces are sums over the points (GPU): one quadrilateral turned
by 90 degrees between its two prisms keeps the whole mesh off the moment
form, so these are the face kernels in FP64, in double words and on the
tensor cores, each on its own arithmetic, with neighbours, boundary and all
degrees around them."""
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


def _mesh(n, turned=True, seed=0):
    """2 n^3 jittered prisms, and beside them two that share a turned
    quadrilateral."""
    from modfem_gb300.mesh import MixedMesh, mixed_faces, structured_prism_mesh
    m = structured_prism_mesh(n, jitter=0.2, seed=seed)
    X = np.array([[0, 0, 0], [1, 0, 0.1], [0.1, 1, 0], [0, 0, 1], [1, 0, 1.1], [0, 1.1, 1], [0, -1, 0.2], [1, -1.1, 0.3]])
    pair = np.array([[0, 1, 2, 3, 4, 5], [0, 3, 6, 1, 4, 7]], np.int32) + len(m.coords)
    if not turned:
        X, pair = np.zeros((0, 3)), np.zeros((0, 6), np.int32)
    el = np.concatenate([m.el_nodes, pair]).astype(np.int32)
    t = MixedMesh(1, np.concatenate([m.coords, X / n + 2.0]), el, np.full(len(el), 6, np.int32), 1)
    return t, mixed_faces(t)


def _system(gb, m, F, p, volume, face, **kw):
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(f=1.0, g=0.3, **kw)
    c.dg_set_degrees(p)
    c.dg_set_faces(F, penalty=10.0)
    c.dg_build_structure()
    c.dg_set_volume_kernel(volume)
    c.dg_set_face_kernel(face)
    out = []
    for _ in range(2):  # again over a matrix of NaN: nothing is left from before
        c.dg_assemble()
        out.append([np.array(a) for a in c.dg_get_matrix()])
        c.dg_set_matrix(np.full(c.dg_nval, np.nan), np.full(c.dg_ndof, np.nan))
    s = c.dg_get_structure()
    c.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    return out[0][0], out[0][1], s


def _modes(gb):
    return [(v, f) for v in (gb.DG_VOLUME_FP64, gb.DG_VOLUME_TC_DWORD)
            for f in (gb.DG_FACE_FP64, gb.DG_FACE_DWORD, gb.DG_FACE_TC, gb.DG_FACE_TC_DWORD)]


def _coefficients(m, aniso, seed):
    from modfem_gb300.mesh import anisotropic_tensors, lognormal_k
    return {"D": anisotropic_tensors(m.nel, seed=seed).reshape(m.nel, 9)} if aniso else {"k": lognormal_k(m.nel, seed=seed)}


@pytest.mark.parametrize("pmax,aniso", [(1, True), (2, False), (3, True), (4, True), (4, False)])
def test_every_face_mode_vs_oracle(gb, pmax, aniso):
    m, F = _mesh(2, seed=pmax)
    p = np.random.default_rng(pmax).integers(1, pmax + 1, m.nel).astype(np.int32)
    kw = _coefficients(m, aniso, pmax)
    D = kw.get("D")
    if D is None:
        D = (kw["k"][:, None, None] * np.eye(3)).reshape(m.nel, 9)
    rp, ci, val, rhs, off = O.dg_assemble(m, F, p, D, pen=10.0, g=0.3)
    for volume, face in _modes(gb):
        v, r, s = _system(gb, m, F, p, volume, face, **kw)
        rp2, ci2, v = dg_blocks_to_crs(*s, v)
        assert np.array_equal(rp, rp2) and np.array_equal(ci, ci2)
        assert sparse_rel_err(rp, ci, v, val) < REL_TOL, (volume, face)
        assert vec_rel_err(r, rhs) < REL_TOL


@pytest.mark.parametrize("n,pmax,aniso", [(6, 1, False), (6, 2, True), (7, 3, True), (8, 4, False), (7, 4, True)])
def test_every_face_mode_vs_fp64_point_sums(gb, n, pmax, aniso):
    """Hundreds of prisms, mixed and uniform degrees: double words and tensor
    cores against the FP64 sums over the points (1e-13 and the FP64 tolerance,
    as their own statements have it), and those against the moment form of
    the same prisms without the turned pair."""
    m, F = _mesh(n, seed=n + pmax)
    p = (np.full(m.nel, pmax) if n % 2 else np.random.default_rng(n).integers(1, pmax + 1, m.nel)).astype(np.int32)
    kw = _coefficients(m, aniso, n)
    v0, r0, s = _system(gb, m, F, p, gb.DG_VOLUME_FP64, gb.DG_FACE_FP64, **kw)
    rp, ci, c0 = dg_blocks_to_crs(*s, v0)
    for face, tol in ((gb.DG_FACE_DWORD, 1e-13), (gb.DG_FACE_TC, REL_TOL), (gb.DG_FACE_TC_DWORD, REL_TOL)):
        v, r, _ = _system(gb, m, F, p, gb.DG_VOLUME_FP64, face, **kw)
        assert sparse_rel_err(rp, ci, dg_blocks_to_crs(*s, v)[2], c0) < tol, face
        assert vec_rel_err(r, r0) < tol
    q, G = _mesh(n, turned=False, seed=n + pmax)
    v, r, t = _system(gb, q, G, p[:q.nel], gb.DG_VOLUME_FP64, gb.DG_FACE_FP64, **{k: a[:q.nel] for k, a in kw.items()})
    rp, ci, c = dg_blocks_to_crs(*t, v)
    assert sparse_rel_err(rp, ci, c0[:len(c)], c) < REL_TOL
    assert vec_rel_err(r0[:len(r)], r) < REL_TOL
