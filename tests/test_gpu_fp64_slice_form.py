"""The FP64 block CG's slice form at the sizes where its launch changes: one
slice, a last slice with one row, one and two blocks, a lane per dof up to
four slices per block and a lane per row above, more than 512 and 896 threads
per block, the largest size and the first one past it.  A workspace without
the ghost plan runs the global form: same iteration counts to rounding (2 %,
at least 2), both with a true residual (the oracle's SpMV) that meets the
tolerance."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def solve(L, s, ws_bytes, tol, flags, x0):
    from nbots_gb300.device import DeviceArray
    lib = L.lib()
    A = s.block_layout()
    u = DeviceArray(x0)
    ws = DeviceArray(np.full(ws_bytes, 0xff, np.uint8))  # stale records must not count
    r = L.CgResult()
    rc = lib.nbg_cg_bsr_f64(C.byref(A), s.dptr(L.FEM_F), u.ptr, 8 * s.N, tol, flags, C.byref(r),
                            ws.ptr, ws_bytes, None)
    return rc, r, u.numpy()


@pytest.mark.parametrize("nx,ny,mesh", [(15, 2, "q4"), (10, 2, "t3"), (31, 2, "q4"),
                                        (84, 228, "q4"), (151, 127, "t3"), (152, 128, "q4"),
                                        (400, 206, "q4"), (550, 256, "t3"), (575, 268, "q4"),
                                        (660, 236, "q4")])
@pytest.mark.parametrize("rule", ["true", "nbots", "plain"])
def test_fp64_slice_form_sizes(nx, ny, mesh, rule):
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.fem import FemSystem
    if rule == "plain" and nx > 100:
        pytest.skip("the unpreconditioned rule is the same code; small sizes cover it")
    p = W.cantilever_q4(nx, ny + ny % 2, top_traction=0.01)
    if mesh == "t3":
        c = p.conn
        p.elem = "t3"
        p.conn = np.stack([c[:, [0, 1, 2]], c[:, [0, 2, 3]]], 1).reshape(-1, 3)
        p.edges = np.concatenate([p.edges, c[:, [0, 2]]])
    p.E = W.lognormal_E(p.n_elems, 0.3, 5)
    s = FemSystem(p)
    assert s.assemble() == 0
    s.apply_bcs()
    lib, A = L.lib(), s.block_layout()
    F = s.get(L.FEM_F)
    rel = 1e-9 if p.n_nodes < 20_000 else 1e-4
    # a start other than zero: a tenth of a smooth field
    x0 = 0.1 * np.repeat(np.sin(p.nod[:, 0]), 2)
    x0[2 * p.sgm[4].astype(np.int64)] = x0[2 * p.sgm[4].astype(np.int64) + 1] = 0.0
    if rule == "nbots":
        flags, tol = L.CG_JACOBI | L.CG_NBOTS_STOP, rel * np.linalg.norm(F)
    else:
        flags, tol = (L.CG_JACOBI if rule == "true" else 0) | L.CG_RELATIVE, rel
    rc1, r1, u1 = solve(L, s, lib.nbg_cg_bsr_layout_workspace_bytes(C.byref(A)), tol, flags, x0)
    rc0, r0, u0 = solve(L, s, lib.nbg_cg_bsr_workspace_bytes(s.N), tol, flags, x0)
    assert rc0 == rc1 == 0
    assert abs(int(r1.niter) - int(r0.niter)) <= max(2, 0.02 * r0.niter)
    for u in (u0, u1):
        res = F - O.spmv(s.get(L.FEM_ROW_PTR), s.get(L.FEM_COL_IDX), s.get(L.FEM_K), u)
        # the oracle's products are rounded, the solver's fused
        assert np.linalg.norm(res) <= 1.01 * rel * np.linalg.norm(F)
    s.close()
