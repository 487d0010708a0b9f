"""The batched solver's slice form (one block per SM, a warp per slice): many
small systems, blocks of 16 slices and of more, systems that fill one launch
(152 blocks of 16) and one system more, several launches, and a numbering whose
ghosts do not fit.  Each system's reported residual is that of the oracle's SpMV (the form
judges on nbots' arithmetic, so to 1e-12), its iterations those of the single solve within 2 %, and replays have the same
bits."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-6


def shuffled(p, seed):
    rank = np.random.default_rng(seed).permutation(p.n_nodes).astype(np.uint32)
    nod = np.empty_like(p.nod)
    nod[rank] = p.nod
    p.nod, p.conn, p.edges = nod, rank[p.conn], rank[p.edges]
    p.vtx, p.sgm = rank[p.vtx], [rank[g] for g in p.sgm]
    return p


# slices of a system of nx by ny elements: 2 (8, 4); 149 (96, 48); 263 (128, 64);
# 586 (192, 96); 1,037 (256, 128); 603 (190, 100), 4 of which take 152 blocks; 2,321
# (384, 192)
@pytest.mark.parametrize("sizes", [
    ((8, 4),) * 40 + ((3, 2), (96, 48)),
    ((256, 128), (96, 48), (192, 96), (192, 96), (8, 4)),
    ((190, 100),) * 4,
    ((190, 100),) * 4 + ((3, 2),),
    ((384, 192), (450, 224)),
    ((96, 48),) * 3 + ((256, 128),) * 7 + ((64, 32), (128, 64)),
    ((192, 96), (96, 48), -192)])
def test_batch_slices(sizes):
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.batch import Batch
    from nbots_gb300.fem import FemSystem
    probs, rho = [], []
    for k, sz in enumerate(sizes):
        if isinstance(sz, tuple):
            p = W.cantilever_q4(*sz)
        else:
            p = shuffled(W.cantilever_q4(-sz, -sz // 2), 7)
        probs.append(p)
        rho.append(np.random.Generator(np.random.PCG64(k)).uniform(0.3, 0.7, size=p.n_elems))
    b = Batch(probs)
    b.assemble_simp(rho, probs[0].nu)
    b.setup(max_iter=20000, tol=TOL)
    _, blocks, _ = b.blocks()
    slices = np.diff(b.node_off.astype(np.int64)) // 32
    assert np.all(slices <= 32 * blocks)
    b.launch()
    res, _ = b.results()
    rp, ci, K, F, u, E = (b.merged(w) for w in (L.FEM_ROW_PTR, L.FEM_COL_IDX, L.FEM_K, L.FEM_F,
                                                L.FEM_U, L.FEM_E))
    seen = {}
    for k, p in enumerate(probs):
        assert res[k].status == 0 and res[k].relres <= TOL
        r0, r1 = 2 * int(b.node_off[k]), 2 * int(b.node_off[k]) + p.n_dof
        seg = slice(int(rp[r0]), int(rp[r1]))
        y = O.spmv(rp[r0:r1 + 1] - rp[r0], (ci[seg] - r0).astype(np.uint32), K[seg], u[r0:r1])
        rel = np.linalg.norm(F[r0:r1] - y) / np.linalg.norm(F[r0:r1])
        assert abs(rel - res[k].relres) <= 1e-12 * rel + 1e-16
        if sizes[k] not in seen:  # one single solve per size is enough
            seen[sizes[k]] = True
            p.E = E[int(b.elem_off[k]):int(b.elem_off[k + 1])].copy()
            s = FemSystem(p)
            assert s.assemble() == 0
            s.apply_bcs()
            r = s.solve_mixed(tol=TOL)
            assert abs(int(r.niter) - int(res[k].niter)) <= 0.02 * r.niter + 2
            s.close()
    b.launch()
    b.results()
    assert np.array_equal(u.view(np.uint64), b.merged(L.FEM_U).view(np.uint64))
    b.close()
