"""The device tables that the first call builds, built by several threads at
once (GPU): in a process of its own, whose first calls they are."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import threading
import numpy as np
import modfem_gb300 as gb
from modfem_gb300.mesh import mixed_faces, structured_mixed_mesh, structured_prism_mesh, structured_tet_mesh
gb.load_library()
pm, tm, mm = structured_prism_mesh(2), structured_tet_mesh(2), structured_mixed_mesh(3, 1)
F = mixed_faces(mm)
out, start = [None] * 8, threading.Barrier(8)


def batch():
    b = gb.Batch(0)
    X, T = pm.coords[pm.el_nodes], tm.coords[tm.el_nodes]
    b.set(X, np.tile(np.eye(3), (len(X), 1, 1)), np.arange(len(X)) % 4 + 1, T, np.tile(np.eye(3), (len(T), 1, 1)),
          np.arange(len(T)) % 4 + 1)
    b.run()
    v = [np.array(a) for a in b.get()]
    b.close()
    return v


def system():
    c = gb.Context(0)
    c.set_mesh_mixed(mm)
    c.set_coefficients(k=np.ones(mm.nel), f=1.0)
    c.dg_set_degrees(np.arange(mm.nel) % 4 + 1)
    c.dg_set_faces(F, penalty=10.0)
    c.dg_build_structure()
    c.dg_assemble()
    v = [np.array(a) for a in c.dg_get_matrix()]
    c.close()
    return v


def work(i):
    start.wait()
    out[i] = (batch, system)[i % 2]()


t = [threading.Thread(target=work, args=(i,)) for i in range(8)]
[a.start() for a in t]
[a.join() for a in t]
ref = [batch(), system()]
for i in range(8):
    assert out[i] is not None and all(np.array_equal(a, b) for a, b in zip(out[i], ref[i % 2])), i
    assert all(np.all(np.isfinite(a)) for a in out[i])
print("same")
"""


@pytest.mark.parametrize("run", range(3))
def test_tables_built_by_eight_threads(run):
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]
