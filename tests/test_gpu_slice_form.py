"""The mixed solver's slice form (one 32-row slice per warp, sums in fixed
point) at the sizes where its launch changes: one slice, a last slice with
one row, one block, the grid's last block short, more than 512 and 896 threads
per block, and the first size past the form.  With the layout-sized workspace
it keeps its block's ghosts in shared memory, with the minimal one it gathers
p from global memory; both give the same bits.  It judges the solve on nbots'
own residual, so the relative residual of the oracle's SpMV is the one it
reports, to the rounding of the norms (1e-12)."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-9


def solve(L, s, ws_bytes, tol=TOL, F=None):
    from nbots_gb300.device import DeviceArray
    lib = L.lib()
    A = s.block_layout()
    u = DeviceArray(np.zeros(s.N))
    ws = DeviceArray(np.full(ws_bytes, 0xff, np.uint8))  # stale records must not count
    r = L.MixedResult()
    rc = lib.nbg_cg_mixed(C.byref(A), s.dptr(L.FEM_F) if F is None else F.ptr, u.ptr, 8 * s.N,
                          tol, 0.1, L.CG_JACOBI | L.CG_RELATIVE, C.byref(r), ws.ptr, ws_bytes,
                          None)
    return rc, r, u.numpy(), lib.nbg_cg_mixed_last_form()


# nodes (nx + 1)(ny + 1): 32 (one slice), 33 (a last slice with one row),
# 128 and 129 (one and two blocks), 19,465 (a short last block), 66,049 (1 of
# 152 blocks short), 80,143 (17 slices, 544 threads), 141,511 (30 slices, 960
# threads), 155,520 (the largest with 32), 156,333 (past the form)
@pytest.mark.parametrize("nx,ny,shuffle", [(15, 1, 0), (10, 2, 0), (31, 3, 0), (42, 2, 0),
                                           (84, 228, 0), (256, 256, 0), (256, 256, 1),
                                           (576, 138, 0), (550, 256, 0), (550, 256, 1), (575, 269, 0),
                                           (660, 236, 0)])
def test_slice_form_sizes(nx, ny, shuffle):
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.fem import FemSystem
    p = W.cantilever_q4(nx, ny + ny % 2, top_traction=0.01) if ny % 2 == 0 else None
    if p is None:  # an odd height has no middle node: load the corner
        nod, conn, edges = W.q4_grid(nx, ny)
        w = nx + 1
        p = W.Problem("odd", "q4", nod, conn, edges, np.array([nx], np.uint32),
                      [(np.arange(ny + 1) * w).astype(np.uint32)],
                      [W.BC(W.DIRICHLET, W.ON_SEGMENT, 0, (1, 1)),
                       W.BC(W.NEUMANN, W.ON_POINT, 0, (1, 1), (0.1, -1.0))],
                      np.ones(conn.shape[0]))
    p.E = W.lognormal_E(p.n_elems, 0.3, 5)
    if shuffle:  # a numbering without locality: at 141,511 nodes more ghosts than fit
        rank = np.random.default_rng(1).permutation(p.n_nodes).astype(np.uint32)
        nod = np.empty_like(p.nod)
        nod[rank] = p.nod
        p.nod, p.conn, p.edges = nod, rank[p.conn], rank[p.edges]
        p.vtx, p.sgm = rank[p.vtx], [rank[g] for g in p.sgm]
    s = FemSystem(p)
    assert s.assemble() == 0
    s.apply_bcs()
    lib, A = L.lib(), s.block_layout()
    # the largest sizes: a loose tolerance keeps the test short
    tol = TOL if p.n_nodes < 20_000 else 1e-4
    rc1, r1, u1, form1 = solve(L, s, lib.nbg_cg_mixed_layout_workspace_bytes(C.byref(A)), tol)
    rc0, r0, u0, form0 = solve(L, s, lib.nbg_cg_mixed_workspace_bytes(s.N), tol)
    assert rc0 == rc1 == 0
    assert form0 != 2 and form1 == (1 if shuffle and nx == 550 else 2)
    assert (r1.niter, r1.n_updates) == (r0.niter, r0.n_updates)
    assert np.array_equal(u1.view(np.uint64), u0.view(np.uint64))
    F = s.get(L.FEM_F)
    res = F - O.spmv(s.get(L.FEM_ROW_PTR), s.get(L.FEM_COL_IDX), s.get(L.FEM_K), u1)
    rel = np.linalg.norm(res) / np.linalg.norm(F)
    assert rel <= tol * (1 + 1e-6)
    if (p.n_nodes + 31) // 32 <= 32 * 152:
        assert abs(rel - r1.relres) <= 1e-12 * r1.relres + 1e-16
    s.close()


@pytest.mark.parametrize("scale", [1e-11, 1e-8, 1e15])
def test_scaled_load_scales_the_solution(scale):
    """The windows of the fixed-point sums follow the values; sums outside
    2^-80 .. 2^80 go to the records.  A scaled load (the solver keeps |r|^2 in
    FP32 pairs: 1e-11 is near the least that its range allows) takes as many iterations,
    give or take the rounding, to the same relative residual."""
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.device import DeviceArray
    from nbots_gb300.fem import FemSystem
    s = FemSystem(W.config_c1())
    assert s.assemble() == 0
    s.apply_bcs()
    n = L.lib().nbg_cg_mixed_layout_workspace_bytes(C.byref(s.block_layout()))
    _, r, u, _ = solve(L, s, n)
    rc, rs, us, _ = solve(L, s, n, F=DeviceArray(s.get(L.FEM_F) * scale))
    assert rc == 0 and rs.relres <= TOL
    assert abs(int(rs.niter) - int(r.niter)) <= 0.02 * r.niter + 2
    # both within TOL's error of the same solution
    assert np.linalg.norm(us / scale - u) <= 1e-6 * np.linalg.norm(u)
    s.close()
