"""Solves of different sizes from several host threads at once: each kernel
form asks for as much shared memory as its system needs, and the bits are
those of the solve alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_concurrent_solves():
    from nbots_gb300 import _lib as L, workloads as W
    from nbots_gb300.fem import FemSystem
    systems = []
    for nx, ny in ((24, 12), (96, 48), (150, 80), (250, 126)):
        s = FemSystem(W.cantilever_q4(nx, ny, top_traction=0.01))
        assert s.assemble() == 0
        s.apply_bcs()
        systems.append(s)

    def solve(s):
        out = []
        for run in (s.solve_mixed, s.solve_fast, s.solve):
            r = run(tol=1e-6)
            out.append((r.status, r.niter, s.get(L.FEM_U).view(np.uint64)))
        return out

    alone = [solve(s) for s in systems]
    wrong = []

    def work(s, want):
        for _ in range(8):
            try:
                got = solve(s)
            except Exception as e:
                wrong.append((s.N, e))
                return
            wrong.extend((s.N, k) for k, (g, w) in enumerate(zip(got, want))
                         if g[:2] != w[:2] or not np.array_equal(g[2], w[2]))

    threads = [threading.Thread(target=work, args=a) for a in zip(systems, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    for s in systems:
        s.close()
