"""What the performance of this library is measured on: passes through its public entry points, from the smallest
systems a program assembles to the largest, on seeded structured meshes with jittered nodes.

A case is a dict of plain values; `prepare` makes what a program holds before the call (mesh, structure, tables, page-locked
buffers), `run` is one pass and returns its outputs, `exact` gives the same outputs from plain torch in 64 bits.
"""
import ctypes
import functools

import numpy as np
import torch

import modfem_gb300 as gb
from modfem_gb300 import serve
from modfem_gb300.mesh import (anisotropic_tensors, lognormal_k, mixed_faces, structured_mixed_mesh,
                               structured_prism_mesh, structured_tet_mesh)

JITTER = 0.2
NS = {1: 6, 2: 18, 3: 40, 4: 75}        # functions of a DG prism of degree p
TET_NS = {1: 4, 2: 10, 3: 20, 4: 35}
NQ = {1: 6, 2: 18, 3: 48, 4: 80}        # volume points of a DG prism
FAST = ("fp64", "fast")                 # DG kernels: the FP64 defaults, or double word and tensor cores


def listed():
    return [
        # the call that stands in for the host code's assembly, host arrays in and out, default options
        # (tables go up with every call): a small model problem
        {"name": "dropin_16k", "kind": "dropin", "n": 20, "arith": "fp64", "cache": False},
        # the same at production size as a time loop uses it: tables kept, double-word elements
        {"name": "dropin_2m_dword", "kind": "dropin", "n": 100, "arith": "dword", "cache": True},
        # assemble and 60 GMRES(30) iterations: one nonlinear step of a small model, bound by latency
        {"name": "solve_std_16k", "kind": "std_solve", "n": 20, "arith": "fp64", "iters": 60},
        # the same at production size
        {"name": "solve_std_2m", "kind": "std_solve", "n": 100, "arith": "fp64", "iters": 60},
        # a new mesh each time, as after remeshing or for a served request: upload, structure on the device,
        # deterministic assembly, one restart cycle
        {"name": "new_mesh_315k", "kind": "std_new_mesh", "n": 54, "iters": 30},
        # linear tetrahedra, colour scatter, matrix and rhs back to the host
        {"name": "std_tet_162k", "kind": "std_tet", "n": 30},
        # the smallest DG systems: degree 2, whole block matrix to the host
        {"name": "dg_p2_2k_matrix", "kind": "dg_matrix", "n": 10, "p": 2, "aniso": False, "mode": "fp64"},
        # every degree in one mesh (hp), whole block matrix to the host
        {"name": "dg_p1to4_8k_matrix", "kind": "dg_matrix", "n": 16, "p": 0, "aniso": False, "mode": "fp64"},
        # degree 3 with full tensors: assembly and one short GMRES cycle, the DG production step
        {"name": "dg_p3_54k_solve", "kind": "dg_solve", "n": 30, "p": 3, "aniso": True, "mode": "fp64", "iters": 20},
        # prisms and tetrahedra in one hp system with the fast kernels, and its residual at a given state
        {"name": "dg_prism_tet_fast", "kind": "dg_mixed", "n": 16, "layers": 10, "mode": "fast"},
        # element matrices of a mixed batch of prisms and tetrahedra, degrees 1..4, to the host
        {"name": "batch_35k", "kind": "batch", "np": 20000, "nt": 15000, "arith": "fp64"},
        # a burst of small independent problems at the server
        {"name": "serve_burst", "kind": "serve", "std": 6, "dg": 2, "nmin": 10, "nmax": 20, "iters": 60},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["dropin", "std_solve", "std_new_mesh", "std_tet", "dg_matrix", "dg_solve", "dg_mixed", "batch",
                       "serve"])
    if kind == "dropin":
        return {"kind": kind, "n": _log(rng, 5, 95), "arith": rng.choice(["fp64", "dword"]),
                "cache": rng.random() < 0.5}
    if kind == "std_solve":
        return {"kind": kind, "n": _log(rng, 8, 95), "arith": rng.choice(["fp64", "dword"]), "iters": rng.randint(20, 60)}
    if kind == "std_new_mesh":
        return {"kind": kind, "n": _log(rng, 8, 60), "iters": rng.randint(10, 30)}
    if kind == "std_tet":
        return {"kind": kind, "n": _log(rng, 4, 40)}
    if kind == "dg_matrix":
        p = rng.randint(0, 4)
        return {"kind": kind, "n": _log(rng, 3, {0: 15, 1: 30, 2: 22, 3: 16, 4: 12}[p]), "p": p,
                "aniso": rng.random() < 0.5, "mode": rng.choice(FAST)}
    if kind == "dg_solve":  # (a block-Jacobi iterate of degree 4, or of a double-word matrix, magnifies its rounding too far)
        p = rng.randint(1, 3)
        return {"kind": kind, "n": _log(rng, 4, {1: 36, 2: 32, 3: 27}[p]), "p": p, "aniso": rng.random() < 0.5,
                "mode": "fp64", "iters": rng.randint(8, 20)}
    if kind == "dg_mixed":
        n = _log(rng, 4, 16)
        return {"kind": kind, "n": n, "layers": rng.randint(1, n - 1), "mode": rng.choice(FAST)}
    if kind == "batch":
        return {"kind": kind, "np": _log(rng, 100, 20000), "nt": _log(rng, 100, 15000),
                "arith": rng.choice(["fp64", "dword"])}
    return {"kind": kind, "std": rng.randint(2, 8), "dg": rng.randint(0, 2), "nmin": rng.randint(6, 9),
            "nmax": rng.randint(12, 20), "iters": rng.randint(30, 60)}


# ---------------------------------------------------------------------------
# inputs (the topology of a structured mesh is the same for every seed)
# ---------------------------------------------------------------------------
class _Mesh:
    """A mesh of structured_prism_mesh / _tet_mesh / _mixed_mesh with other node positions."""

    def __init__(self, base, coords):
        self.__dict__.update(base.__dict__)
        self.coords = coords
        self.nno, self.nel = coords.shape[0], self.el_nodes.shape[0]


@functools.lru_cache(maxsize=4)
def _prism_base(n):
    return structured_prism_mesh(n)


@functools.lru_cache(maxsize=4)
def _prism_faces(n):
    m = _prism_base(n)
    m.el_nv = np.full(m.nel, 6, np.int32)
    return mixed_faces(m)


@functools.lru_cache(maxsize=4)
def _mixed_base(n, layers):
    m = structured_mixed_mesh(n, layers)
    return m, mixed_faces(m)


def _jittered(base, n, seed):
    x = base.coords
    d = np.random.default_rng(seed).uniform(-JITTER / n, JITTER / n, size=x.shape)
    d[(np.abs(x) < 1e-12) | (np.abs(x - 1.0) < 1e-12)] = 0.0
    return _Mesh(base, x + d)


def _prisms(n, seed):
    return _jittered(_prism_base(n), n, seed)


def _tets(n, seed):
    m = structured_tet_mesh(n, jitter=JITTER, seed=seed)
    return _Mesh(m, m.coords)


def _degrees(case, nel):
    """The element degrees (p = 0: 1..4 in turn at random); they fix the size of the system, so no seed changes them."""
    if case.get("p", 0):
        return np.full(nel, case["p"], np.int32)
    return np.random.default_rng(nel).integers(1, 5, nel).astype(np.int32)


def _coeff(case, nel, seed):
    """(k, D): a lognormal isotropic coefficient or rotated full tensors."""
    if case.get("aniso"):
        return None, anisotropic_tensors(nel, seed=seed)
    return lognormal_k(nel, seed=seed), None


def _host(n):
    """A page-locked output buffer (the array keeps it alive)."""
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _pinned(a):
    return torch.as_tensor(a).pin_memory().numpy()


def _serve_sizes(case):
    std = [int(round(v)) for v in np.geomspace(case["nmin"], case["nmax"], case["std"])]
    return std[::2] + std[1::2][::-1], [4 + i % 3 for i in range(case["dg"])]


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "serve":
        return _prepare_serve(case, seed)
    s = {"kind": kind, "case": case}
    c = s["ctx"] = gb.Context(0)
    if kind in ("dg_matrix", "dg_solve", "dg_mixed"):
        if kind == "dg_mixed":
            base, faces = _mixed_base(case["n"], case["layers"])
            m = _jittered(base, case["n"], seed)
            X = m.coords[m.el_nodes[m.el_nv == 4][:, :4]]
            assert np.all(np.einsum("ij,ij->i", X[:, 1] - X[:, 0], np.cross(X[:, 2] - X[:, 0], X[:, 3] - X[:, 0])) > 0)
            c.set_mesh_mixed(m)
        else:
            m, faces = _prisms(case["n"], seed), _prism_faces(case["n"])
            c.set_mesh(m)
        k, D = _coeff(case, m.nel, seed)
        c.set_coefficients(k=k, D=D, f=1.0, g=0.3)
        c.dg_set_degrees(_degrees(case, m.nel))
        c.dg_set_faces(faces, penalty=10.0)
        if case["mode"] == "fast":
            c.dg_set_volume_kernel(gb.DG_VOLUME_DWORD)
            c.dg_set_face_kernel(gb.DG_FACE_TC_DWORD)
        nd, nv = c.dg_build_structure()
        if kind == "dg_matrix":
            s["val"], s["rhs"] = _host(nv), _host(nd)
        if kind == "dg_mixed":
            s["x"] = np.random.default_rng(seed + 5).standard_normal(nd)
        return s
    if kind == "std_tet":
        m = _tets(case["n"], seed)
        c.set_mesh(m)
        c.set_coefficients(k=lognormal_k(m.nel, seed=seed), f=1.0)
        nd, nnz, _ = c.build_structure()
        s["val"], s["rhs"] = _host(nnz), _host(nd)
        return s
    m = s["mesh"] = _prisms(case["n"], seed)
    k = s["k"] = lognormal_k(m.nel, seed=seed)
    if case.get("arith") == "dword":
        c.set_option(gb.OPT_STD_ARITH, gb.STD_DWORD)
    if kind == "std_new_mesh":
        return s
    c.set_mesh(m)
    nd, nnz = c.build_structure_device()
    if kind == "std_solve":
        return s
    tables = c.get_element_tables()
    nbf = m.bc_face_id.size
    ids = np.concatenate([np.arange(1, m.nel + 1), m.bc_face_id]).astype(np.int32)
    lists = (np.concatenate([np.full(m.nel, gb.ELEMENT), np.full(nbf, gb.FACE)]).astype(np.int32), ids,
             np.array([0, m.nel], np.int32), np.array([m.nel, ids.size], np.int32),
             (np.arange(ids.size) * 42).astype(np.int32),
             np.concatenate([tables, tables.reshape(m.nel, 42)[m.bc_face_el].reshape(-1)]).astype(np.int32))
    s["keep"] = [_pinned(a) for a in (m.coords, k) + lists]
    s["val"], s["rhs"] = _host(nnz), _host(nd)
    if case["cache"]:
        c.set_option(gb.OPT_CACHE_TABLES, 1)
    return s


def _batch_inputs(case, seed):
    n = next(i for i in range(2, 100) if 2 * i ** 3 >= case["np"])
    t = next(i for i in range(2, 100) if 6 * i ** 3 >= case["nt"])
    pm, tm = _prisms(n, seed), _tets(t, seed)
    pp, tp = _degrees({}, case["np"]), _degrees({}, case["nt"])
    A = lognormal_k(case["np"] + case["nt"], seed=seed)[:, None] * np.eye(3).reshape(1, 9)
    return (pm.coords[pm.el_nodes[:case["np"]]], A[:case["np"]], pp, tm.coords[tm.el_nodes[:case["nt"]]],
            A[case["np"]:], tp)


def _prepare_batch(case, seed):
    b = gb.Batch(0)
    nval, nrhs = b.set(*_batch_inputs(case, seed))
    b.set_arith(case["arith"] == "dword")
    return {"kind": "batch", "case": case, "batch": b, "val": _host(nval), "rhs": _host(nrhs)}


def _serve_meshes(case, seed):
    std, dg = _serve_sizes(case)
    return [(serve.STD, _prisms(n, seed + i), 1, None) for i, n in enumerate(std)] + \
           [(serve.DG, _prisms(n, seed + 50 + i), 1 + i % 2, _prism_faces(n)) for i, n in enumerate(dg)]


def _prepare_serve(case, seed):
    probs = [serve.Problem(m, lognormal_k(m.nel, seed=seed + i), kind=kd, p=p, faces=fa, krylov=30,
                           max_iter=case["iters"], tol=1e-14)
             for i, (kd, m, p, fa) in enumerate(_serve_meshes(case, seed))]
    return {"kind": "serve", "case": case, "problems": probs,
            "server": serve.Server(0, hbm_budget=16 << 30, max_active=16, prep_threads=4)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "batch":
        b = s["batch"]
        b.run()
        if b.L.gbfem_batch_get(b._h, _ptr(s["val"]), _ptr(s["rhs"])) < 0:
            raise gb.GbFemError(b.L.gbfem_last_error().decode())
        return {"val": s["val"], "rhs": s["rhs"]}
    if kind == "serve":
        ids = [s["server"].submit(p) for p in s["problems"]]
        out = []
        for i, p in zip(ids, s["problems"]):
            s["server"].wait(i)
            out.append(s["server"].result(i, serve.dof_count(p))[0])
            s["server"].release(i)
        return out
    c = s["ctx"]
    if kind == "dropin":
        xyz, k, *lists = s["keep"]
        c.set_node_coords(xyz)
        c.set_coefficients(k=k, f=1.0, g=0.0, penalty=1e7)
        c.create_assemble_stiff_mat(*lists, crs_val=s["val"], rhs=s["rhs"])
        return {"val": s["val"], "rhs": s["rhs"]}
    if kind == "std_solve":
        c.set_coefficients(k=s["k"], f=1.0, g=0.0, penalty=1e7)
        c.assemble(gb.SCATTER_ATOMIC)
        return c.solve(30, case["iters"], 1e-14)[0]
    if kind == "std_new_mesh":
        c.set_mesh(s["mesh"])
        c.build_structure_device()
        c.set_coefficients(k=s["k"], f=1.0, g=0.0, penalty=1e7)
        c.assemble(gb.SCATTER_GATHER)
        return c.solve(30, case["iters"], 1e-14)[0]
    if kind == "std_tet":
        c.assemble(gb.SCATTER_COLOR)
        c.get_matrix(s["val"], s["rhs"])
        return {"val": s["val"], "rhs": s["rhs"]}
    c.dg_assemble()
    if kind == "dg_matrix":
        if c.L.gbfem_dg_get_matrix(c._h, _ptr(s["val"]), _ptr(s["rhs"])) < 0:
            raise gb.GbFemError(c.L.gbfem_last_error().decode())
        return {"val": s["val"], "rhs": s["rhs"]}
    if kind == "dg_mixed":
        return c.dg_compute_residual(s["x"])
    return c.dg_solve(30, case["iters"], 1e-14)[0]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _gmres_bytes(nnz_bytes, n, iters, m=30):
    """Matrix once and the Krylov basis twice (dots, update) an iteration."""
    return sum(nnz_bytes + 16 * n + 16 * n * (i % m + 2) for i in range(iters))


def _dg_work(nel, ns, nq, faces):
    val = 8 * nel * (1 + faces) * ns * ns
    return val, nel * 2 * (nq * 80 + 8 * ns * ns * (1 + faces))


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    std = lambda n: (2 * n ** 3, (n + 1) ** 3, 21 * (n + 1) ** 3)  # noqa: E731  elements, nodes, stored values
    if kind in ("dropin", "std_solve", "std_new_mesh"):
        nel, nno, nnz = std(n)
        inp, out, fl = 24 * nno + 32 * nel, 8 * nnz + 8 * nno, 791 * nel
        if kind == "dropin":
            return {"bytes": inp + out + (0 if case["cache"] else 168 * nel), "flops": fl}
        return {"bytes": inp + out + _gmres_bytes(12 * nnz, nno, case["iters"]),
                "flops": fl + case["iters"] * (2 * nnz + 64 * nno)}
    if kind == "std_tet":
        nel, nno = 6 * n ** 3, (n + 1) ** 3
        return {"bytes": 24 * nno + 24 * nel + 8 * 15 * nno, "flops": 150 * nel}
    if kind in ("dg_matrix", "dg_solve", "dg_mixed"):
        p = case.get("p", 0)
        nel = 2 * n ** 3 if kind != "dg_mixed" else 2 * n * n * case["layers"] + 6 * n * n * (n - case["layers"])
        ns = {**NS, 0: 43}[p] if kind != "dg_mixed" else 30
        val, fl = _dg_work(nel, ns, {**NQ, 0: 40}[p], 4.5)
        if kind == "dg_solve":
            it = case["iters"]
            return {"bytes": val + _gmres_bytes(val + 8 * nel * ns * ns, nel * ns, it), "flops": fl + it * val / 4}
        return {"bytes": val if kind == "dg_matrix" else 2 * val, "flops": fl}
    if kind == "batch":
        np_, nt = case["np"], case["nt"]
        return {"bytes": 8 * (np_ * 1896 + nt * 435) + 216 * (np_ + nt), "flops": 2 * (np_ * 16000 + nt * 3000)}
    std_n, dg_n = _serve_sizes(case)
    b = f = 0
    for m in std_n:
        w = work({"kind": "std_solve", "n": m, "iters": case["iters"]})
        b, f = b + w["bytes"], f + w["flops"]
    for i, m in enumerate(dg_n):
        w = work({"kind": "dg_solve", "n": m, "p": 1 + i % 2, "iters": case["iters"]})
        b, f = b + w["bytes"], f + w["flops"]
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same outputs from plain torch in 64 bits
# ---------------------------------------------------------------------------
# symmetric triangle rules (points in orbits of permuted barycentric coordinates, weights summing to 1/2): 3, 6, 12
# and 16 points, exact to degree 2, 4, 6 and 8
_T3 = lambda a, w: [(a, a, w), (a, 1 - 2 * a, w), (1 - 2 * a, a, w)]  # noqa: E731
_T6 = lambda a, b, w: [(x, y, w) for x, y in  # noqa: E731
                       ((a, b), (b, 1 - a - b), (1 - a - b, a), (a, 1 - a - b), (b, a), (1 - a - b, b))]
_TRI = {1: _T3(1 / 6, 1 / 6),
        2: _T3(0.445948490915965, 0.1116907948390055) + _T3(0.091576213509771, 0.054975871827661),
        3: _T3(0.24928674517091, 0.0583931378631895) + _T3(0.063089014491502, 0.0254224531851035)
        + _T6(0.310352451033784, 0.636502499121399, 0.041425537809187),
        4: [(1 / 3, 1 / 3, 0.0721578038388935)] + _T3(0.459292588292723, 0.0475458171336425)
        + _T3(0.17056930775176, 0.051608685267359) + _T3(0.050547228317031, 0.016229248811599)
        + _T6(0.263112829634638, 0.728492392955404, 0.0136151570872175)}


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_dev())


def _volume_rule(p):
    g, w = np.polynomial.legendre.leggauss(p + 1)
    pts = [(x, y, z, wt * wz) for z, wz in zip(g, w) for x, y, wt in _TRI[p]]
    return np.array([q[:3] for q in pts]), np.array([q[3] for q in pts])


def _prism_shape(e):
    """Values (q, 6) and local gradients (q, 6, 3) of the linear prism at local points e (q, 3)."""
    x, y, z = e[:, 0], e[:, 1], e[:, 2]
    L = np.stack([1 - x - y, x, y], 1)
    dL = np.array([[-1.0, -1.0], [1.0, 0.0], [0.0, 1.0]])
    lo, hi = (1 - z) / 2, (1 + z) / 2
    N = np.concatenate([L * lo[:, None], L * hi[:, None]], 1)
    G = np.zeros((len(e), 6, 3))
    for i in range(3):
        G[:, i, :2], G[:, i + 3, :2] = dL[i] * lo[:, None], dL[i] * hi[:, None]
        G[:, i, 2], G[:, i + 3, 2] = -0.5 * L[:, i], 0.5 * L[:, i]
    return N, G


_SIDES = ((0, 2, 1), (3, 4, 5), (0, 1, 4, 3), (1, 2, 5, 4), (2, 0, 3, 5))
_LOCAL = np.array([[0, 0, -1], [1, 0, -1], [0, 1, -1], [0, 0, 1], [1, 0, 1], [0, 1, 1]], float)


def _face_weights(nv, p):
    """Vertex weights (q, nv), their (s, t) derivatives and quadrature weights of the face rule of degree p."""
    if nv == 3:
        q = np.array(_TRI[p])
        s, t, w = q.T
        one = np.ones_like(s)
        return (np.stack([1 - s - t, s, t], 1), np.stack([-one, one, 0 * one], 1), np.stack([-one, 0 * one, one], 1), w)
    g, wg = np.polynomial.legendre.leggauss(p + 1)
    s, t = [a.ravel() for a in np.meshgrid((g + 1) / 2, (g + 1) / 2, indexing="ij")]
    w = np.outer(wg, wg).ravel()
    if nv == 4:
        return (np.stack([(1 - s) * (1 - t), s * (1 - t), s * t, (1 - s) * t], 1),
                np.stack([t - 1, 1 - t, t, -t], 1) / 2, np.stack([s - 1, -s, s, 1 - s], 1) / 2, w)
    raise ValueError(nv)


def _std_system(m, k, tet=False):
    """(rows, cols, values) of the element and penalty-face entries by node, and the rhs by node."""
    X, el, k = _t(m.coords)[_t(m.el_nodes).long()], _t(m.el_nodes).long(), _t(k)
    nv = el.shape[1]
    if tet:
        G = np.array([[[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]], float)
        N, w = np.full((1, 4), 0.25), np.array([1 / 6])
    else:
        e, w = _volume_rule(1)
        N, G = _prism_shape(e)
    K = torch.zeros(el.shape[0], nv, nv, dtype=torch.float64, device=X.device)
    R = torch.zeros(el.shape[0], nv, dtype=torch.float64, device=X.device)
    for q in range(len(w)):
        J = torch.einsum("eia,ib->eab", X, _t(G[q]))
        det = torch.linalg.det(J).abs() * w[q]
        g = torch.linalg.solve(J.transpose(1, 2), _t(G[q]).T.expand(el.shape[0], 3, nv)).transpose(1, 2)
        K += (det * k)[:, None, None] * (g @ g.transpose(1, 2))
        R += det[:, None] * _t(N[q])
    rows, cols = [el[:, :, None].expand_as(K).reshape(-1)], [el[:, None, :].expand_as(K).reshape(-1)]
    vals = [K.reshape(-1)]
    rhs = torch.zeros(m.nno, dtype=torch.float64, device=X.device).index_add_(0, el.reshape(-1), R.reshape(-1))
    for side, loc in enumerate(_SIDES if not tet else ()):
        f = _t(m.bc_face_el[m.bc_face_side == side]).long()
        nd = el[f][:, list(loc)]
        Y = _t(m.coords)[nd]
        M = torch.zeros(len(f), len(loc), len(loc), dtype=torch.float64, device=X.device)
        W, Ws, Wt, wq = _face_weights(len(loc), 1)
        for q in range(len(wq)):
            a = torch.linalg.norm(torch.linalg.cross(torch.einsum("eia,i->ea", Y, _t(Ws[q])),
                                                     torch.einsum("eia,i->ea", Y, _t(Wt[q]))), dim=1) * wq[q]
            M += 1e7 * a[:, None, None] * _t(np.outer(W[q], W[q]))
        rows.append(nd[:, :, None].expand_as(M).reshape(-1))
        cols.append(nd[:, None, :].expand_as(M).reshape(-1))
        vals.append(M.reshape(-1))
    return torch.cat(rows), torch.cat(cols), torch.cat(vals), rhs


def _dof_of_node(m):
    """Degrees of freedom in the order in which the elements first meet their vertices."""
    u, first = np.unique(m.el_nodes.ravel(), return_index=True)
    d = np.full(m.nno, -1, np.int64)
    d[u[np.argsort(first, kind="stable")]] = np.arange(u.size)
    return d


def _std_crs(m, k, tet=False):
    d = _t(_dof_of_node(m))
    r, c, v, b = _std_system(m, k, tet)
    n = int(d.max()) + 1
    key, inv = torch.unique(d[r] * n + d[c], return_inverse=True)
    val = torch.zeros(key.numel(), dtype=torch.float64, device=v.device).index_add_(0, inv, v)
    rhs = torch.zeros(n, dtype=torch.float64, device=v.device)
    rhs[d[d >= 0]] = b[d >= 0]
    return key // n, key % n, val, rhs


def _gmres(mv, b, iters, m=30):
    """x after `iters` iterations of GMRES(m) from zero on the (preconditioned) operator mv."""
    x = torch.zeros_like(b)
    while iters > 0:
        r = b - mv(x)
        beta = float(torch.linalg.norm(r))
        k = min(m, iters)
        V, H = [r / beta], np.zeros((k + 1, k))
        for j in range(k):
            w = mv(V[j])
            B = torch.stack(V)
            for _ in range(2):
                h = B @ w
                w = w - B.T @ h
                H[:j + 1, j] += h.cpu().numpy()
            H[j + 1, j] = float(torch.linalg.norm(w))
            V.append(w / H[j + 1, j])
        e = np.zeros(k + 1)
        e[0] = beta
        y = np.linalg.lstsq(H, e, rcond=None)[0]
        x = x + torch.stack(V[:k]).T @ _t(y)
        iters -= k
    return x


def _std_solve(m, k, iters):
    r, c, v, b = _std_crs(m, k)
    n = b.numel()
    dinv = torch.ones_like(b)
    dinv[r[r == c]] = 1.0 / v[r == c]
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=b.device)
    ptr[1:] = torch.cumsum(torch.bincount(r, minlength=n), 0)
    A = torch.sparse_csr_tensor(ptr, c, v * dinv[r], (n, n))
    return _gmres(lambda x: (A @ x[:, None])[:, 0], dinv * b, iters)


def _exps(p):
    """Monomial exponents of the tensor basis: the linear prism first, then level by level in zeta."""
    rest = [(1, 1)] * (p > 1) + [(a, b) for b in range(p + 1) for a in range(p - b + 1)
                                 if a + b > 1 and (a, b) != (1, 1)]
    lin = [(0, 0), (1, 0), (0, 1)]
    out = [(a, b, c) for c in (0, 1) for a, b in lin] + [(a, b, c) for c in (0, 1) for a, b in rest]
    return np.array(out + [(a, b, c) for c in range(2, p + 1) for a, b in lin + rest])


def _tet_exps(p):
    return np.array([(a, b, d - a - b) for d in range(p + 1) for a in range(d, -1, -1) for b in range(d - a, -1, -1)])


def _monomials(E, e):
    """Values (q, ns) and local gradients (q, ns, 3) of monomials E at points e."""
    pw = e[:, None, :] ** E[None]
    G = np.zeros((len(e), len(E), 3))
    for a in range(3):
        d = E.copy()
        d[:, a] = np.maximum(d[:, a] - 1, 0)
        G[:, :, a] = E[:, a] * np.prod(e[:, None, :] ** d[None], axis=2)
    return np.prod(pw, axis=2), G


def _volume(X, A, E, e, w, shape_grad):
    """Stiffness (n, ns, ns) and unit load (n, ns) of elements with vertices X and tensors A."""
    phi, dphi = _monomials(E, e)
    K = torch.zeros(X.shape[0], len(E), len(E), dtype=torch.float64, device=X.device)
    R = torch.zeros(X.shape[0], len(E), dtype=torch.float64, device=X.device)
    for q in range(len(w)):
        J = torch.einsum("eia,ib->eab", X, _t(shape_grad[q]))
        det = torch.linalg.det(J).abs() * w[q]
        g = torch.linalg.solve(J.transpose(1, 2), _t(dphi[q]).T.expand(X.shape[0], 3, len(E)))
        K += g.transpose(1, 2) @ (det[:, None, None] * (A @ g))
        R += det[:, None] * _t(phi[q])
    return K, R


def _dg_system(m, F, deg, k, D, g=0.3, pen=10.0):
    """The DG system of a prism mesh: {(row degree, column degree): [(rows, cols, blocks), ...]} and the rhs list."""
    X = _t(m.coords)[_t(m.el_nodes).long()]
    A = _t(D).reshape(-1, 3, 3) if D is not None else _t(k)[:, None, None] * torch.eye(3, dtype=torch.float64, device=_dev())
    blocks, rhs = [], {}
    dev = X.device
    for p in range(1, 5):
        es = _t(np.nonzero(deg == p)[0])
        if not len(es):
            continue
        e, w = _volume_rule(p)
        K, R = _volume(X[es], A[es], _exps(p), e, w, _prism_shape(e)[1])
        rhs[p] = torch.zeros(m.nel, NS[p], dtype=torch.float64, device=dev)
        rhs[p][es] += R
        blocks.append((p, p, es, es, K))
    nf = F.el1.size
    loc = np.full((2, nf, 4), -1)
    for s, el in enumerate((F.el1, F.el2)):
        loc[s] = np.argmax(m.el_nodes[el][:, None, :] == F.nodes[:, :, None], axis=2)
    d2 = np.where(F.el2 >= 0, deg[F.el2], 0)
    key = np.stack([F.type, deg[F.el1], d2, *(loc[0].T * (F.nodes >= 0).T), *(loc[1].T * (F.nodes >= 0).T * (F.el2 >= 0))])
    for u in np.unique(key, axis=1).T:
        fs = np.nonzero((key == u[:, None]).all(0))[0]
        nv, p1, p2 = int(u[0]), int(u[1]), int(u[2])
        W, Ws, Wt, wq = _face_weights(nv, max(p1, p2))
        Y = _t(m.coords)[_t(F.nodes[fs][:, :nv]).long()]
        cr = lambda i, j: torch.linalg.norm(torch.linalg.cross(Y[:, (i + 1) % nv] - Y[:, i], Y[:, (j + 1) % nv] - Y[:, j]), dim=1)  # noqa: E731,E501
        area = 0.5 * cr(0, 1) if nv == 3 else 0.5 * (cr(0, 1) + cr(2, 3))
        c = pen * (min(p1, p2) if p2 else p1) / torch.sqrt(area)
        els = [_t(F.el1[fs]).long()] + ([_t(F.el2[fs]).long()] if p2 else [])
        ps = [p1, p2][:len(els)]
        at = [W @ _LOCAL[u[3 + 4 * s:3 + 4 * s + nv]] for s in range(len(els))]
        mon, geo = [_monomials(_exps(p), a) for p, a in zip(ps, at)], [_prism_shape(a)[1] for a in at]
        cen = X[els[0]].mean(1)
        acc = [[torch.zeros(len(fs), NS[p], NS[r], dtype=torch.float64, device=dev) for r in ps] for p in ps]
        for q in range(len(wq)):
            n = torch.linalg.cross(torch.einsum("eia,i->ea", Y, _t(Ws[q])), torch.einsum("eia,i->ea", Y, _t(Wt[q])))
            n = n * torch.sign(((Y.mean(1) - cen) * n).sum(1))[:, None]
            a = torch.linalg.norm(n, dim=1)
            n, a = n / a[:, None], a * wq[q]
            ph, gr = [], []
            for s, el in enumerate(els):
                J = torch.einsum("eia,ib->eab", X[el], _t(geo[s][q]))
                v = torch.linalg.solve(J, torch.einsum("eji,ej->ei", A[el], n))
                ph.append(_t(mon[s][0][q]))
                gr.append(v @ _t(mon[s][1][q]).T)
            fac = 0.5 if p2 else 1.0
            for i, si in enumerate((1.0, -1.0)[:len(els)]):
                L = a[:, None] * (fac * gr[i] + si * c[:, None] * ph[i])
                for j, sj in enumerate((1.0, -1.0)[:len(els)]):
                    acc[i][j] += L[:, :, None] * (sj * ph[j]) - (si * fac * a)[:, None, None] * ph[i][:, None] * gr[j][:, None, :]
                if not p2:
                    rhs[p1].index_add_(0, els[0], g * L)
        for i, p in enumerate(ps):
            for j, r in enumerate(ps):
                blocks.append((p, r, els[i], els[j], acc[i][j]))
    return blocks, rhs


def _dg_matrix(m, F, deg, blocks, rhs):
    """The stored values: block rows in element order, blocks ascending, each column-major."""
    r = np.concatenate([np.arange(m.nel), F.el1[F.el2 >= 0], F.el2[F.el2 >= 0]])
    c = np.concatenate([np.arange(m.nel), F.el2[F.el2 >= 0], F.el1[F.el2 >= 0]])
    ns = np.array([NS[int(p)] for p in deg], np.int64)
    key = np.sort(r.astype(np.int64) * m.nel + c)
    off = np.concatenate([[0], np.cumsum(ns[key // m.nel] * ns[key % m.nel])])
    val = torch.zeros(int(off[-1]), dtype=torch.float64, device=_dev())
    off, key = _t(off), _t(key)
    for p, q, rows, cols, B in blocks:
        o = off[torch.searchsorted(key, rows * m.nel + cols)]
        at = o[:, None] + torch.arange(NS[p] * NS[q], device=o.device)
        val.index_add_(0, at.reshape(-1), B.transpose(1, 2).reshape(-1))
    doff = _t(np.concatenate([[0], np.cumsum(ns)]))
    return val, _dg_vector(m, deg, doff, rhs)


def _dg_vector(m, deg, doff, rhs):
    out = torch.zeros(int(doff[-1]), dtype=torch.float64, device=_dev())
    for p, v in rhs.items():
        es = _t(np.nonzero(deg == p)[0])
        out[(doff[es][:, None] + torch.arange(NS[p], device=out.device)).reshape(-1)] = v[es].reshape(-1)
    return out


def _dg_solve(m, deg, blocks, rhs, iters):
    ns = np.array([NS[int(p)] for p in deg], np.int64)
    doff = _t(np.concatenate([[0], np.cumsum(ns)]))
    at = {p: (lambda es, p=p: doff[es][:, None] + torch.arange(NS[p], device=doff.device)) for p in rhs}
    b = _dg_vector(m, deg, doff, rhs)
    diag = {p: torch.zeros(m.nel, NS[p], NS[p], dtype=torch.float64, device=_dev()) for p in rhs}
    for p, q, rows, cols, B in blocks:
        if rows is cols or bool((rows == cols).all()):
            diag[p].index_add_(0, rows, B)
    inv = {p: torch.linalg.inv(diag[p][_t(np.nonzero(deg == p)[0])]) for p in rhs}

    def prec(v):
        out = torch.zeros_like(v)
        for p in rhs:
            i = at[p](_t(np.nonzero(deg == p)[0]))
            out[i.reshape(-1)] = (inv[p] @ v[i][:, :, None]).reshape(-1)
        return out

    where = [(at[p](rows).reshape(-1), at[q](cols), B) for p, q, rows, cols, B in blocks]

    def mv(x):
        y = torch.zeros_like(x)
        for i, j, B in where:
            y.index_add_(0, i, (B @ x[j][:, :, None]).reshape(-1))
        return prec(y)
    return _gmres(mv, prec(b), iters)


def _batch_exact(case, seed):
    PX, PA, pp, TX, TA, tp = _batch_inputs(case, seed)
    vals, loads = [None] * (len(pp) + len(tp)), [None] * (len(pp) + len(tp))
    for p in range(1, 5):
        e, w = _volume_rule(p)
        g, wg = np.polynomial.legendre.leggauss(p + 3)
        g, wg = (g + 1) / 2, wg / 2
        U, V, Z = [a.ravel() for a in np.meshgrid(g, g, g, indexing="ij")]
        te = np.stack([U, V * (1 - U), Z * (1 - U) * (1 - V)], 1)
        tw = np.prod(np.stack([a.ravel() for a in np.meshgrid(wg, wg, wg, indexing="ij")]), 0) * (1 - U) ** 2 * (1 - V)
        tg = np.broadcast_to(np.array([[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float), (len(tw), 4, 3))
        for X, A, deg, E, at, wt, sg, base in ((PX, PA, pp, _exps(p), e, w, _prism_shape(e)[1], 0),
                                               (TX, TA, tp, _tet_exps(p), te, tw, tg, len(pp))):
            es = np.nonzero(deg == p)[0]
            if len(es):
                K, R = _volume(_t(X[es]), _t(A[es]).reshape(-1, 3, 3), E, at, wt, sg)
                K, R = K.cpu().numpy(), R.cpu().numpy()
                for i, x in enumerate(es):
                    vals[base + x], loads[base + x] = K[i].T.ravel(), R[i]
    return {"val": np.concatenate(vals), "rhs": np.concatenate(loads)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "dg_mixed":  # faces between prisms and tetrahedra: no short plain form
        return None
    if kind == "batch":
        return _batch_exact(case, seed)
    if kind == "serve":
        out = []
        for i, (kd, m, p, fa) in enumerate(_serve_meshes(case, seed)):
            k = lognormal_k(m.nel, seed=seed + i)
            if kd == serve.STD:
                out.append(_std_solve(m, k, case["iters"]))
            else:
                deg = np.full(m.nel, p)
                out.append(_dg_solve(m, deg, *_dg_system(m, fa, deg, k, None, g=0.0), case["iters"]))
        return [x.cpu().numpy() for x in out]
    if kind == "std_tet":
        m = _tets(case["n"], seed)
        _, _, val, rhs = _std_crs(m, lognormal_k(m.nel, seed=seed), tet=True)
        return {"val": val.cpu().numpy(), "rhs": rhs.cpu().numpy()}
    m = _prisms(case["n"], seed)
    if kind == "dropin":
        _, _, val, rhs = _std_crs(m, lognormal_k(m.nel, seed=seed))
        return {"val": val.cpu().numpy(), "rhs": rhs.cpu().numpy()}
    if kind in ("std_solve", "std_new_mesh"):
        return _std_solve(m, lognormal_k(m.nel, seed=seed), case["iters"]).cpu().numpy()
    F, deg = _prism_faces(case["n"]), _degrees(case, m.nel)
    blocks, rhs = _dg_system(m, F, deg, *_coeff(case, m.nel, seed))
    if kind == "dg_matrix":
        val, b = _dg_matrix(m, F, deg, blocks, rhs)
        return {"val": val.cpu().numpy(), "rhs": b.cpu().numpy()}
    return _dg_solve(m, deg, blocks, rhs, case["iters"]).cpu().numpy()
