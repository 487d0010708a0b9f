"""Mixed solves whose sums fall far in one iteration, in every form of the
solver.  A matrix of node blocks d [[1, c], [c, 1]] has two eigenvalues after
scaling, and a right-hand side that is one eigenvector plus `eps` of the other
makes p.w, r.z and |r|^2 fall by eps^2 from the first iteration to the second,
after which the solve is done: at 2^-60 to 2^-80 that crosses the least sum that
the fixed-point form gives as a float-float number (2^-97).  Then small models
whose own sums do the same.  The error bound of the first: the second iteration
is exact but for rounding, and the tolerance (1e-9 of the load) bounds the rest
times the condition number, 3."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def block_diagonal(blocks):
    """Device layout of one 2x2 block per node row; keeps its arrays alive."""
    from nbots_gb300 import _lib as L
    from nbots_gb300.device import DeviceArray
    Nn = len(blocks)
    S = (Nn + 31) // 32
    rp = np.arange(2 * Nn + 1, dtype=np.uint32) * 2
    ci = np.repeat(np.arange(Nn, dtype=np.uint32), 4) * 2 + np.tile([0, 1, 0, 1], Nn).astype(np.uint32)
    n = 32 * S
    keep = [DeviceArray(np.arange(S + 1, dtype=np.uint32)), DeviceArray(rp), DeviceArray(ci),
            DeviceArray(np.ascontiguousarray(blocks, np.float64).ravel())]
    keep += [DeviceArray(np.zeros(k, t)) for k, t in
             ((n, np.uint32), (4 * n, np.float64), (4 * n, np.float32), (4 * n, np.uint16),
              (4 * n, np.uint8), (2 * Nn, np.float64), (2 * Nn, np.float32))]
    A = L.Bsr(2 * Nn, Nn, S, n, keep[0].ptr, *(k.ptr for k in keep[4:]), None, None)
    assert L.lib().nbg_bsr_fill(C.byref(A), keep[1].ptr, keep[2].ptr, keep[3].ptr, None) == 0
    return A, keep


def two_values(Nn, c, eps, ex, d=1.0):
    """d [[1, c], [c, 1]] on every node and a load whose first p.w is near 2^ex."""
    rng = np.random.default_rng(Nn)
    v = rng.uniform(0.5, 1.0, Nn)
    b = np.stack([v + eps * v[::-1], v - eps * v[::-1]], 1)
    b *= np.sqrt(2.0 ** ex * d / (2.0 * (1.0 + c) * np.sum(v * v)))
    blocks = d * np.tile(np.array([[1.0, c], [c, 1.0]]), (Nn, 1, 1))
    return blocks, b, np.linalg.solve(blocks, b[:, :, None])[:, :, 0].ravel()


def solve(A, b, ws_bytes, tol, max_iter=50):
    from nbots_gb300 import _lib as L
    from nbots_gb300.device import DeviceArray
    u, F = DeviceArray(np.zeros(A.N)), DeviceArray(np.ascontiguousarray(b, np.float64).ravel())
    ws, r = DeviceArray(np.zeros(ws_bytes, np.uint8)), L.MixedResult()
    rc = L.lib().nbg_cg_mixed(C.byref(A), F.ptr, u.ptr, max_iter, tol, 0.1,
                              L.CG_JACOBI | L.CG_RELATIVE, C.byref(r), ws.ptr, ws_bytes, None)
    return rc, r, u.numpy(), L.lib().nbg_cg_mixed_last_form()


# 40 nodes: one block; 5,000: 40 blocks; 156,000: past the slice form
@pytest.mark.parametrize("Nn,planned,form", [(40, 1, 2), (5000, 1, 2), (5000, 0, 1),
                                             (156_000, 1, 2), (156_000, 0, 1)])
@pytest.mark.parametrize("ex,drop", [(-60, 18), (-76, 18), (-76, 24), (-78, 28), (-79, 20),
                                     (-79, 28), (-81, 20)])
def test_sums_that_fall(Nn, planned, form, ex, drop):
    from nbots_gb300 import _lib as L
    blocks, b, want = two_values(Nn, 0.5, 2.0 ** (-drop / 2), ex)
    A, keep = block_diagonal(blocks)
    n = (L.lib().nbg_cg_mixed_layout_workspace_bytes(C.byref(A)) if planned
         else L.lib().nbg_cg_mixed_workspace_bytes(A.N))
    rc, r, u, f = solve(A, b, n, 1e-9)
    assert rc == 0 and f == form and r.relres <= 1e-9
    assert np.linalg.norm(u - want) <= 3e-9 * np.linalg.norm(want)


@pytest.mark.parametrize("ex,drop", [(-60, 18), (-79, 20), (-79, 28)])
def test_sums_that_fall_in_a_batch(ex, drop):
    from nbots_gb300 import _lib as L
    from nbots_gb300.device import DeviceArray
    lib, sizes = L.lib(), (64, 320, 32, 4800)
    parts = [two_values(n, 0.5, 2.0 ** (-drop / 2), ex) for n in sizes]
    A, keep = block_diagonal(np.concatenate([p[0] for p in parts]))
    b = DeviceArray(np.concatenate([p[1].ravel() for p in parts]))
    u = DeviceArray(np.zeros(A.N))
    ptr = (np.cumsum((0,) + sizes) // 32).astype(np.uint32)
    m = C.c_void_p()
    assert lib.nbg_mixed_batch_create(C.byref(m), C.byref(A), b.ptr, u.ptr, len(sizes),
                                      ptr.ctypes.data, 50, 1e-9, 0.1,
                                      L.CG_JACOBI | L.CG_RELATIVE, None) == 0
    assert lib.nbg_mixed_batch_launch(m) == 0
    res = (L.MixedResult * len(sizes))()
    assert lib.nbg_mixed_batch_results(m, res, None) == 0
    got = np.split(u.numpy(), 2 * np.cumsum(sizes)[:-1])
    for r, g, (_, _, want) in zip(res, got, parts):
        assert r.status == 0 and r.relres <= 1e-9
        assert np.linalg.norm(g - want) <= 3e-9 * np.linalg.norm(want)
    lib.nbg_mixed_batch_destroy(m)


@pytest.mark.parametrize("nx,ny,E,load", [(3, 2, 2.1e11, 1.0), (3, 2, 1.0, 1e-6), (2, 6, 1e6, 1e-5)])
def test_small_models_in_their_own_units(nx, ny, E, load):
    """The relative residual of the oracle's SpMV meets the tolerance (with its
    rounding of A u, 1e-12 for these conditions), and so does an error bounded by
    the condition number of the scaled matrix."""
    from oracle import oracle as O
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.fem import FemSystem
    s = FemSystem(W.cantilever_q4(nx, ny, E=E, point_load=-load))
    assert s.assemble() == 0
    s.apply_bcs()
    r = s.solve_mixed(tol=1e-10)
    rp, ci, K, F = (s.get(w) for w in (L.FEM_ROW_PTR, L.FEM_COL_IDX, L.FEM_K, L.FEM_F))
    u = s.get(L.FEM_U)
    s.close()
    assert r.status == 0 and r.relres <= 1e-10
    assert np.linalg.norm(F - O.spmv(rp, ci, K, u)) <= 1.02e-10 * np.linalg.norm(F)
    D = np.zeros((F.size, F.size))
    D[np.repeat(np.arange(F.size), np.diff(rp.astype(np.int64))), ci] = K
    want = np.linalg.solve(D, F)
    assert np.linalg.norm(u - want) <= 1.1e-10 * np.linalg.norm(F) * np.linalg.norm(np.linalg.inv(D), 2)
