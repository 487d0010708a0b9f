"""What a solve needs of memory.  The FP64 block CG asks for the ghost plan's only
for systems that its slice form can take (32 slices per SM): a larger one needs what
it needed without that form, and runs in just that.  Where the plan's memory
cannot be had (here: for a layout that says that it has 2^38 entries, 550 GB of
local columns), the solver that allocates its own workspace and the batch run
without it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_systems_need_no_plan():
    import torch
    from nbots_gb300 import _lib as L
    lib, nsm = L.lib(), torch.cuda.get_device_properties(0).multi_processor_count
    for S, more in ((1, True), (32 * nsm, True), (32 * nsm + 1, False), (400_000, False)):
        A = L.Bsr(64 * S, 32 * S, S, 32 * 9 * S)
        plain = lib.nbg_cg_bsr_workspace_bytes(A.N)
        assert (lib.nbg_cg_bsr_layout_workspace_bytes(C.byref(A)) > plain) == more


def test_a_large_system_solves_in_the_plain_workspace():
    from nbots_gb300 import _lib as L
    from nbots_gb300.device import DeviceArray
    from test_gpu_sum_range import block_diagonal, two_values
    blocks, b, want = two_values(160_000, 0.5, 0.25, 0)
    A, keep = block_diagonal(blocks)
    n, r = L.lib().nbg_cg_bsr_layout_workspace_bytes(C.byref(A)), L.CgResult()
    assert n == L.lib().nbg_cg_bsr_workspace_bytes(A.N)
    u, F, ws = DeviceArray(np.zeros(A.N)), DeviceArray(b.ravel()), DeviceArray(np.zeros(n, np.uint8))
    for w, m in ((ws.ptr, n), (None, 0)):
        u.upload(np.zeros(A.N))
        assert L.lib().nbg_cg_bsr_f64(C.byref(A), F.ptr, u.ptr, 50, 1e-12, L.CG_JACOBI | L.CG_RELATIVE,
                                      C.byref(r), w, m, None) == 0
        assert np.linalg.norm(u.numpy() - want) <= 3e-12 * np.linalg.norm(want)


def test_the_plan_is_dropped_when_its_memory_is_not_there():
    from nbots_gb300 import _lib as L
    from nbots_gb300.device import DeviceArray
    from test_gpu_sum_range import block_diagonal, two_values
    lib = L.lib()
    blocks, b, want = two_values(640, 0.5, 0.25, 0)
    A, keep = block_diagonal(blocks)
    A.n_entries = 1 << 38
    u, F, r = DeviceArray(np.zeros(A.N)), DeviceArray(b.ravel()), L.CgResult()
    assert lib.nbg_cg_bsr_f64(C.byref(A), F.ptr, u.ptr, 50, 1e-12, L.CG_JACOBI | L.CG_RELATIVE,
                              C.byref(r), None, 0, None) == 0
    assert np.linalg.norm(u.numpy() - want) <= 3e-12 * np.linalg.norm(want)
    m, ptr, res = C.c_void_p(), np.array([0, 4, 20], np.uint32), (L.MixedResult * 2)()
    assert lib.nbg_mixed_batch_create(C.byref(m), C.byref(A), F.ptr, u.ptr, 2, ptr.ctypes.data, 50,
                                      1e-9, 0.1, L.CG_JACOBI | L.CG_RELATIVE, None) == 0
    assert lib.nbg_mixed_batch_launch(m) == 0
    assert lib.nbg_mixed_batch_results(m, res, None) == 0
    assert np.linalg.norm(u.numpy() - want) <= 3e-9 * np.linalg.norm(want)
    lib.nbg_mixed_batch_destroy(m)
