"""The workspace's size chooses the form of the mixed solver, not its iterates:
with the ghost plan and without it the same bits, past the slice form's sizes,
on both sides of the size from which the own rows no longer fit in shared memory
(110 slices per block), and up to the largest ghost-node systems.  Updates are made
frequent (delta 0.5) so that a short budget has several."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# slices per block: 33, 101, 110, 116, 127, 172
@pytest.mark.parametrize("nx,ny", [(660, 236), (980, 500), (1060, 504), (1100, 510), (1120, 550),
                                   (1300, 640)])
def test_same_bits_with_and_without_the_plan(nx, ny):
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.device import DeviceArray
    from nbots_gb300.fem import FemSystem
    p = W.cantilever_q4(nx, ny, top_traction=0.01)
    p.E = W.lognormal_E(p.n_elems, 0.3, 5)
    s = FemSystem(p)
    assert s.assemble() == 0
    s.apply_bcs()
    lib, A, out = L.lib(), s.block_layout(), []
    for n in (lib.nbg_cg_mixed_layout_workspace_bytes(C.byref(A)),
              lib.nbg_cg_mixed_workspace_bytes(s.N)):
        u, r, ws = DeviceArray(np.zeros(s.N)), L.MixedResult(), DeviceArray(np.zeros(n, np.uint8))
        rc = lib.nbg_cg_mixed(C.byref(A), s.dptr(L.FEM_F), u.ptr, 400, 1e-9, 0.5,
                              L.CG_JACOBI | L.CG_RELATIVE, C.byref(r), ws.ptr, n, None)
        assert rc == 1 and r.niter == 400 and r.n_updates > 2
        out.append((r.n_updates, r.relres, u.numpy().view(np.uint64),
                    lib.nbg_cg_mixed_last_form()))
    assert out[0][3] == 2 and out[1][3] != 2
    assert out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2])
    s.close()
