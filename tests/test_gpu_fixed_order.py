"""The FP64 CG with NBG_CG_FIXED_ORDER: the same bits with the workspace of
the slice form as without it, at sizes where the two forms' blocks differ (one
row, one slice, 16 slices and a block of 9 slices per SM)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 2), (15, 2), (84, 6), (96, 48), (300, 138)])
@pytest.mark.parametrize("jacobi", [0, 1])
def test_fixed_order_bits(nx, ny, jacobi):
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.device import DeviceArray
    from nbots_gb300.fem import FemSystem
    p = W.cantilever_q4(nx, ny, top_traction=0.01)
    p.E = W.lognormal_E(p.n_elems, 0.3, 5)
    s = FemSystem(p)
    assert s.assemble() == 0
    s.apply_bcs()
    lib, A = L.lib(), s.block_layout()
    got = []
    for n in (lib.nbg_cg_bsr_layout_workspace_bytes(C.byref(A)),
              lib.nbg_cg_bsr_workspace_bytes(s.N)):
        u, r = DeviceArray(np.zeros(s.N)), L.CgResult()
        ws = DeviceArray(np.full(n, 0xff, np.uint8))  # stale records must not count
        rc = lib.nbg_cg_bsr_f64(C.byref(A), s.dptr(L.FEM_F), u.ptr, 300, 1e-8, jacobi | 4 | 8,
                                C.byref(r), ws.ptr, n, None)
        assert rc in (0, 1)
        got.append((r.niter, r.status, r.tol_reached, r.bnorm, u.numpy()))
    assert got[0][:4] == got[1][:4]
    assert np.array_equal(got[0][4].view(np.uint64), got[1][4].view(np.uint64))
    s.close()
