"""Which form a batch takes: in waves of the slice form, its ghosts in shared memory
but for a numbering whose ghosts do not fit, or all systems side by side; and the
solutions stay those of the tolerance when the plan changes while waves are in
use (nbg_mixed_batch_plan and _tune with other gammas)."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_batch_slices import shuffled

pytestmark = pytest.mark.gpu
GLOBAL, RESIDENT, GHOST = 0, 1, 2


def batch(sizes, tol):
    from nbots_gb300 import workloads as W
    from nbots_gb300.batch import Batch
    probs = [W.cantilever_q4(*sz) if isinstance(sz, tuple)
             else shuffled(W.cantilever_q4(-sz, -sz // 2), 7) for sz in sizes]
    rho = [np.random.Generator(np.random.PCG64(k)).uniform(0.3, 0.7, size=p.n_elems)
           for k, p in enumerate(probs)]
    b = Batch(probs)
    b.assemble_simp(rho, probs[0].nu)
    b.setup(max_iter=20000, tol=tol)
    return b


def forms(b):
    from nbots_gb300 import _lib as L
    f = L.lib().nbg_mixed_batch_form
    f.argtypes, f.restype = [C.c_void_p, C.c_void_p], C.c_int
    out = np.full(len(b.problems), -1, np.int32)
    return f(b.solver, out.ctypes.data), out.tolist()


# 2,323 slices: 384 x 192, each a wave of its own, which costs more than all side by
# side; the rows of six (2 KB per slice, 29 MB) fit in the shared memory of 152 SMs (34
# MB), those of nine of 4,112 slices do not
@pytest.mark.parametrize("sizes,waves,form", [
    (((8, 4),) * 40 + ((3, 2), (96, 48)), 1, [GHOST] * 42),
    (((190, 100),) * 4, 1, [GHOST] * 4),
    (((190, 100),) * 4 + ((3, 2),), 2, [GHOST] * 5),
    (((192, 96), (96, 48), -192), 1, [GHOST] * 3),
    (((512, 256), -512), 2, [GHOST, RESIDENT]),
    (((384, 192),) * 6, 0, [RESIDENT] * 6),
    (((512, 256),) * 9, 0, [GLOBAL] * 9)])
def test_batch_form(sizes, waves, form):
    b = batch(sizes, 1e-2)
    b.launch()
    res, _ = b.results()
    assert all(r.status == 0 for r in res)
    assert forms(b) == (waves, form)
    b.close()


def test_other_plans_while_waves_are_in_use():
    sizes = ((256, 128), (96, 48), (192, 96), (64, 32), (128, 64), (8, 4))
    b = batch(sizes, 1e-9)
    b.launch()
    assert forms(b)[0] > 0
    first, res = b.displacements(), b.results()[0]
    for gamma in (0.0, 1.0, 3.0, 1.5):
        b.plan(gamma)
        b.launch()
        got, again = b.displacements(), b.results()[0]
        assert forms(b)[0] > 0
        for u, v, r, q in zip(first, got, res, again):
            # the sums do not depend on the shares: the same iterates
            assert q.status == 0 and q.niter == r.niter
            assert np.array_equal(u.view(np.uint64), v.view(np.uint64))
    b.tune((0.5, 2.0))
    b.launch()
    assert all(r.status == 0 and r.relres <= 1e-9 for r in b.results()[0])
    b.close()
