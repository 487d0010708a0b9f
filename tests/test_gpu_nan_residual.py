"""A mixed solve whose residual is not a number has not converged: status 1, from
a load that holds one and from an iteration that breaks down (a singular matrix
and a direction that it maps to zero: p.w = 0, infinite steps), in every form of
the solver."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_sum_range import block_diagonal, solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nn,planned,form", [(40, 1, 2), (5000, 0, 1), (156_000, 1, 2),
                                             (156_000, 0, 1), (600_000, 0, 0)])
@pytest.mark.parametrize("what", ["load", "breakdown"])
def test_nan_is_not_converged(what, Nn, planned, form):
    from nbots_gb300 import _lib as L
    off = 1.0 if what == "breakdown" else 0.5
    A, keep = block_diagonal(np.tile(np.array([[1.0, off], [off, 1.0]]), (Nn, 1, 1)))
    b = np.tile([1.0, -1.0], (Nn, 1))
    if what == "load":
        b[Nn // 2, 1] = np.nan
    n = (L.lib().nbg_cg_mixed_layout_workspace_bytes(C.byref(A)) if planned
         else L.lib().nbg_cg_mixed_workspace_bytes(A.N))
    rc, r, u, f = solve(A, b, n, 1e-9, max_iter=20)
    assert f == form
    assert rc == 1 and r.status == 1 and not r.relres <= 1e-9
    assert r.niter <= 20


def test_nan_is_not_converged_in_a_batch():
    from nbots_gb300 import _lib as L
    from nbots_gb300.device import DeviceArray
    lib = L.lib()
    A, keep = block_diagonal(np.tile(np.array([[1.0, 0.5], [0.5, 1.0]]), (128, 1, 1)))
    b = np.tile([1.0, -1.0], (128, 1))
    b[70, 0] = np.nan  # of the second system
    F, u, m = DeviceArray(b.ravel()), DeviceArray(np.zeros(A.N)), C.c_void_p()
    ptr = np.array([0, 2, 4], np.uint32)
    assert lib.nbg_mixed_batch_create(C.byref(m), C.byref(A), F.ptr, u.ptr, 2, ptr.ctypes.data, 20,
                                      1e-9, 0.1, L.CG_JACOBI | L.CG_RELATIVE, None) == 0
    assert lib.nbg_mixed_batch_launch(m) == 0
    res = (L.MixedResult * 2)()
    assert lib.nbg_mixed_batch_results(m, res, None) == 1
    assert (res[0].status, res[1].status) == (0, 1)
    lib.nbg_mixed_batch_destroy(m)
