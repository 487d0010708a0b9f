"""nbg_solver_multiply (the drop-in's product) around the size where x goes to
the device by a kernel: even and odd offsets of the caller's vectors, bit for
bit the oracle's."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(8, 4), (62, 128), (63, 127), (64, 126), (200, 150)])
@pytest.mark.parametrize("offset", [0, 1])
def test_multiply_sizes(nx, ny, offset):
    from nbots_gb300 import _lib as L, workloads as W
    p = W.cantilever_q4(nx, ny + ny % 2)
    fl = O.Flat(p)
    rp, ci = O.pattern(fl)
    st, K, F = O.assemble(fl, rp, ci)
    assert st == 0
    lib, h = L.lib(), C.c_void_p()
    N = F.shape[0]
    assert lib.nbg_solver_create(C.byref(h), None) == 0
    assert lib.nbg_solver_set_matrix(h, N, rp.ctypes.data, ci.ctypes.data, K.ctypes.data, 0) == 0
    lib.nbg_solver_multiply.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p]
    x = np.random.default_rng(N).standard_normal(N + offset)
    y = np.zeros(N + offset)
    for k in range(2):  # new values behind the same address
        x[:] = np.roll(x, 3) * (k + 1)
        assert lib.nbg_solver_multiply(h, x.ctypes.data + 8 * offset, y.ctypes.data + 8 * offset) == 0
        ref = O.spmv(rp, ci, K, np.ascontiguousarray(x[offset:]))
        assert np.array_equal(y[offset:].view(np.uint64), ref.view(np.uint64))
    lib.nbg_solver_destroy(h)
