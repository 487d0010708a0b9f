"""nbg_solver_multiply and vectors that do not start on a double (a numpy view into
a byte buffer): no kernel reads or writes them in place.  The host code against
stand-ins of the device calls (tests/c/solver_unaligned.c) on the CPU; the product
itself on the GPU."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_kernels_get_aligned_vectors_only(tmp_path):
    from nbots_gb300 import _lib as L
    L.lib()  # built
    pkg, exe = os.path.dirname(L.GPU_SO), tmp_path / "solver_unaligned"
    subprocess.run(["gcc", "-std=c99", "-Wall", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "nbots_gb300", "host"),
                    os.path.join(ROOT, "tests", "c", "solver_unaligned.c"), "-o", str(exe),
                    "-L" + pkg, "-lnbots_gpu", "-lnbots_host", "-Wl,-rpath," + pkg], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.returncode


@pytest.mark.gpu
@pytest.mark.parametrize("n", [100, 16384, 20001])
def test_product_of_unaligned_vectors(n):
    import ctypes as C
    from nbots_gb300 import _lib as L
    lib, rng = L.lib(), np.random.default_rng(n)
    rp, ci = np.arange(n + 1, dtype=np.uint32), np.arange(n, dtype=np.uint32)[::-1].copy()
    val, x = rng.standard_normal(n), rng.standard_normal(n)
    want = val * x[ci]  # one entry in a row: the product has one rounding
    s = C.c_void_p()
    L.check(lib.nbg_solver_create(C.byref(s), None), "create")
    L.check(lib.nbg_solver_set_matrix(s, n, rp.ctypes.data, ci.ctypes.data, val.ctypes.data, 0), "matrix")
    for pi, po in ((0, 0), (4, 0), (0, 4), (3, 5)):
        bi, bo = np.zeros(8 * n + 8, np.uint8), np.zeros(8 * n + 8, np.uint8)
        bi[pi:pi + 8 * n] = x.view(np.uint8)
        L.check(lib.nbg_solver_multiply(s, C.c_void_p(bi.ctypes.data + pi),
                                        C.c_void_p(bo.ctypes.data + po)), "multiply")
        assert np.array_equal(bo[po:po + 8 * n], want.view(np.uint8)), (pi, po)
    lib.nbg_solver_destroy(s)
