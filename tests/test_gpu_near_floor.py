"""Mixed solves of large systems close to their FP64 floor (about 3e-11 of the load
here), in the ghost-node form and, past what its shared memory holds, with the own rows
in global memory: they converge, and the residual is the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,form,tol", [(1120, 550, 2, 5e-11), (1500, 760, 0, 1e-10)])
def test_converges_near_the_floor(nx, ny, form, tol):
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.fem import FemSystem
    p = W.cantilever_q4(nx, ny, top_traction=0.01)
    p.E = W.lognormal_E(p.n_elems, 0.3, 5)
    s = FemSystem(p)
    assert s.assemble() == 0
    s.apply_bcs()
    r = s.solve_mixed(tol=tol, max_iter=25_000)
    assert r.status == 0 and r.relres <= tol and L.lib().nbg_cg_mixed_last_form() == form
    F = s.get(L.FEM_F)
    res = F - O.spmv(s.get(L.FEM_ROW_PTR), s.get(L.FEM_COL_IDX), s.get(L.FEM_K), s.get(L.FEM_U))
    rel = np.linalg.norm(res) / np.linalg.norm(F)
    assert abs(rel - r.relres) <= 1e-12 * rel
    s.close()
