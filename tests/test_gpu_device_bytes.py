"""gbfem_device_bytes against the device's own free memory (GPU)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import modfem_gb300 as g
    g.load_library()
    return g


def _free():
    cu = ctypes.CDLL("libcuda.so.1")
    free, total = ctypes.c_size_t(), ctypes.c_size_t()
    assert cu.cuMemGetInfo_v2(ctypes.byref(free), ctypes.byref(total)) == 0
    return free.value


def _std(gb):
    """686,000 prisms: gather scatter (230 MB of local matrices), GMRES in both
    arithmetics (75 MB a sliced-ELL copy)."""
    from modfem_gb300.mesh import structured_prism_mesh
    m = structured_prism_mesh(70)
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=np.ones(m.nel), f=1.0)
    c.build_structure_device()
    c.assemble(gb.SCATTER_GATHER)
    c.solve(30, 2, 1e-12)
    c.set_option(gb.OPT_STD_SPMV_ARITH, gb.STD_DWORD)
    c.solve(30, 2, 1e-12)
    return c


def _dg(gb):
    """8,192 cubic prisms (0.5 GB of matrix): assembly, GMRES with the double-word
    operator (as much again), refinement around FP32 (half)."""
    from modfem_gb300.mesh import prism_faces, structured_prism_mesh
    m = structured_prism_mesh(16)
    c = gb.Context(0)
    c.set_mesh(m)
    c.set_coefficients(k=np.ones(m.nel), f=1.0)
    c.dg_set_degrees(np.full(m.nel, 3))
    c.dg_set_faces(prism_faces(m), penalty=10.0)
    c.dg_build_structure()
    c.dg_assemble()
    c.set_option(gb.OPT_DG_SPMV_ARITH, gb.STD_DWORD)
    c.dg_solve(20, 2, 1e-12)
    c.dg_solve_ir(20, 20, 1e-3, 1e-2)
    return c


@pytest.mark.parametrize("make", [_std, _dg])
def test_device_bytes_are_what_the_device_lost(gb, make):
    """Every buffer is an allocation of its own, rounded up to 2 MB at most:
    under a hundred of them.  The same work once before, so that
    modules, local memory and pools are there."""
    make(gb).close()
    before = _free()
    c = make(gb)
    held, lost = c.device_bytes(), before - _free()
    c.close()
    assert abs(lost - held) <= 100 * 2**21, (lost, held)
    assert abs(before - _free()) <= 2**26
