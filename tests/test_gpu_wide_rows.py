"""Assembly of rows of more than 12 node blocks (a fan of elements around one
node), which the gather takes another way than the others, with and without self
weight: K and F are the oracle's bits, before and after the boundary conditions."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def fan(n, quads):
    """n triangles around node 0, or n quadrilaterals 0, a, b, c with a ring of
    corner nodes between the spokes."""
    from nbots_gb300 import workloads as W
    t = 2 * np.pi * np.arange(n) / n
    spoke = np.stack([np.cos(t), np.sin(t)], 1) * (1.0 + 0.05 * np.sin(3 * t))[:, None]
    i = np.arange(n)
    j = (i + 1) % n
    if quads:
        corner = 1.5 * np.stack([np.cos(t + np.pi / n), np.sin(t + np.pi / n)], 1)
        nod = np.concatenate([[[0.0, 0.0]], spoke, corner])
        conn = np.stack([0 * i, 1 + i, 1 + n + i, 1 + j], 1)
        edges = np.concatenate([np.stack([0 * i, 1 + i], 1), np.stack([1 + i, 1 + n + i], 1),
                                np.stack([1 + n + i, 1 + j], 1)])
    else:
        nod = np.concatenate([[[0.0, 0.0]], spoke])
        conn = np.stack([0 * i, 1 + i, 1 + j], 1)
        edges = np.concatenate([np.stack([0 * i, 1 + i], 1), np.stack([1 + i, 1 + j], 1)])
    rng = np.random.default_rng(n)
    return W.Problem("fan", "q4" if quads else "t3", nod, conn.astype(np.uint32),
                     edges.astype(np.uint32), np.array([1, 2], np.uint32),
                     [np.array([1, 2], np.uint32)],
                     [W.BC(W.DIRICHLET, W.ON_SEGMENT, 0, (1, 1)),
                      W.BC(W.NEUMANN, W.ON_POINT, 1, (1, 1), (0.1, -1.0))],
                     rng.uniform(0.5, 2.0, len(conn)))


@pytest.mark.parametrize("n,quads", [(11, 0), (12, 0), (30, 0), (5, 1), (6, 1), (14, 1)])
@pytest.mark.parametrize("weight", [False, True])
@pytest.mark.parametrize("thickness", [1.0, 0.3])
def test_wide_rows(n, quads, weight, thickness):
    from nbots_gb300 import _lib as L
    from nbots_gb300.fem import FemSystem
    p = fan(n, quads)
    p.self_weight, p.density, p.gravity, p.thickness = weight, 7.8, (0.3, -9.81), thickness
    fl = O.Flat(p)
    rp, ci = O.pattern(fl)
    st, K, F = O.assemble(fl, rp, ci)
    assert st == 0 and np.diff(rp.astype(np.int64)).max() // 2 == (2 * n + 1 if quads else n + 1)
    s = FemSystem(p)
    for _ in range(2):
        assert s.assemble() == 0
        assert np.array_equal(s.get(L.FEM_K).view(np.uint64), K.view(np.uint64))
        assert np.array_equal(s.get(L.FEM_F).view(np.uint64), F.view(np.uint64))
    O.set_bconditions(fl, rp, ci, K, F)
    s.apply_bcs()
    assert np.array_equal(s.get(L.FEM_K).view(np.uint64), K.view(np.uint64))
    assert np.array_equal(s.get(L.FEM_F).view(np.uint64), F.view(np.uint64))
    s.close()
