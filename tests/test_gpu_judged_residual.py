"""The residual that a mixed solve reports is nbots' own in every form of the
solver: that of the oracle's SpMV, to the rounding of the norms (1e-12), also past
the slice form's sizes, and also where the start already meets the tolerance."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-7


# 156,417 nodes: past the slice form; 617,671: past the own rows in shared memory
@pytest.mark.parametrize("nx,ny,planned,form", [(64, 32, 1, 2), (660, 236, 1, 2), (660, 236, 0, 1),
                                                (1120, 550, 1, 2), (1120, 550, 0, 0)])
def test_reported_residual_is_nbots_own(nx, ny, planned, form):
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.device import DeviceArray
    from nbots_gb300.fem import FemSystem
    p = W.cantilever_q4(nx, ny, top_traction=0.01)
    p.E = W.lognormal_E(p.n_elems, 0.3, 5)
    s = FemSystem(p)
    assert s.assemble() == 0
    s.apply_bcs()
    lib, A, u, r = L.lib(), s.block_layout(), DeviceArray(np.zeros(s.N)), L.MixedResult()
    n = (lib.nbg_cg_mixed_layout_workspace_bytes(C.byref(A)) if planned
         else lib.nbg_cg_mixed_workspace_bytes(s.N))
    ws = DeviceArray(np.zeros(n, np.uint8))
    rp, ci, K, F = (s.get(w) for w in (L.FEM_ROW_PTR, L.FEM_COL_IDX, L.FEM_K, L.FEM_F))
    for again in range(2):  # the second from the first one's solution
        rc = lib.nbg_cg_mixed(C.byref(A), s.dptr(L.FEM_F), u.ptr, 8 * s.N, TOL * (1 + 1e-9 * again),
                              0.1, L.CG_JACOBI | L.CG_RELATIVE, C.byref(r), ws.ptr, n, None)
        assert rc == 0 and lib.nbg_cg_mixed_last_form() == form
        assert (r.niter == 0) == bool(again)
        rel = np.linalg.norm(F - O.spmv(rp, ci, K, u.numpy())) / np.linalg.norm(F)
        assert abs(rel - r.relres) <= 1e-12 * rel
    s.close()
