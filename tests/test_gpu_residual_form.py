"""The residual that the mixed solver iterates on is b - A u with fused
multiply-adds, the more accurate of the two that it computes.  One iteration from
a nearly converged x0 moves x by alpha z, z = r / Aii, and r is mostly the rounding of
A x0 there: a least-squares fit of the step on the z of both residuals tells which
one it was.  (Each dof's step is rounded like its entry of A x0, so over the
4,290 dofs the fitted share of the other residual scatters by a few hundredths
about 0, or about 1; the bound is 0.3.)"""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def fused(rp, ci, K, x):
    """A x row by row with fused multiply-adds, columns ascending."""
    fx = [Fraction(v) for v in x]
    y = np.zeros(x.size)
    for i in range(x.size):
        t = 0.0
        for k in range(int(rp[i]), int(rp[i + 1])):
            t = float(Fraction(K[k]) * fx[ci[k]] + Fraction(t))
        y[i] = t
    return y


@pytest.mark.parametrize("planned", [1, 0])
def test_iterates_on_the_fused_residual(planned):
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.device import DeviceArray
    from nbots_gb300.fem import FemSystem
    p = W.cantilever_q4(64, 32, top_traction=0.01)
    p.E = W.lognormal_E(p.n_elems, 1.0, 3)
    s = FemSystem(p)
    assert s.assemble() == 0
    s.apply_bcs()
    assert s.solve_mixed(tol=1e-12).status == 0
    rp, ci, K, F, x0 = (s.get(w) for w in (L.FEM_ROW_PTR, L.FEM_COL_IDX, L.FEM_K, L.FEM_F, L.FEM_U))
    lib, A, u, r = L.lib(), s.block_layout(), DeviceArray(x0), L.MixedResult()
    n = (lib.nbg_cg_mixed_layout_workspace_bytes(C.byref(A)) if planned
         else lib.nbg_cg_mixed_workspace_bytes(s.N))
    ws = DeviceArray(np.zeros(n, np.uint8))
    rc = lib.nbg_cg_mixed(C.byref(A), s.dptr(L.FEM_F), u.ptr, 1, 0.0, 0.1, L.CG_JACOBI, C.byref(r),
                          ws.ptr, n, None)
    assert rc == 1 and r.niter == 1
    step = u.numpy() - x0
    s.close()
    diag = np.array([K[rp[i] + np.searchsorted(ci[rp[i]:rp[i + 1]], i)] for i in range(x0.size)])
    zf = (F - fused(rp, ci, K, x0)) / diag
    zn = (F - O.spmv(rp, ci, K, x0)) / diag
    assert np.linalg.norm(zn - zf) > 0.1 * np.linalg.norm(zf)  # the rounding shows
    alpha, other = np.linalg.lstsq(np.stack([zf, zn - zf], 1), step, rcond=None)[0]
    assert abs(other / alpha) < 0.3, (alpha, other)
