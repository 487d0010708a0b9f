"""The FP64 block CG reports the residual of the x that it returns: it confirms
its verdict on b - A x, read back from the memory that it has just written, in the
slice form and in the global form.  The sums' order inside a row differs from the
oracle's, by 1e-13 of |b| against a residual of 1e-9: 1e-3 bounds the difference."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(31, 2), (64, 32), (152, 128), (400, 206)])
@pytest.mark.parametrize("planned", [1, 0])
def test_reported_residual_is_that_of_x(nx, ny, planned):
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.device import DeviceArray
    from nbots_gb300.fem import FemSystem
    p = W.cantilever_q4(nx, ny, top_traction=0.01)
    p.E = W.lognormal_E(p.n_elems, 0.3, 5)
    s = FemSystem(p)
    assert s.assemble() == 0
    s.apply_bcs()
    lib, A, r = L.lib(), s.block_layout(), L.CgResult()
    n = (lib.nbg_cg_bsr_layout_workspace_bytes(C.byref(A)) if planned
         else lib.nbg_cg_bsr_workspace_bytes(s.N))
    # from a start far from the solution: a stale x would show
    u, ws = DeviceArray(np.sin(np.arange(s.N))), DeviceArray(np.zeros(n, np.uint8))
    rc = lib.nbg_cg_bsr_f64(C.byref(A), s.dptr(L.FEM_F), u.ptr, 8 * s.N, 1e-9,
                            L.CG_JACOBI | L.CG_RELATIVE, C.byref(r), ws.ptr, n, None)
    F = s.get(L.FEM_F)
    res = np.linalg.norm(F - O.spmv(s.get(L.FEM_ROW_PTR), s.get(L.FEM_COL_IDX), s.get(L.FEM_K),
                                    u.numpy()))
    assert rc == 0 and r.tol_reached <= 1e-9 * r.bnorm
    assert abs(r.tol_reached - res) <= 1e-3 * res
    s.close()
