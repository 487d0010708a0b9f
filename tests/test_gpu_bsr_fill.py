"""nbg_bsr_fill against the layout's definition written in numpy, word for
word: node counts around a slice, rows of up to 12 blocks (staged through
shared memory) and more, with and without a node order, and values whose
remainder counts are hard (ties, zeros, the ends of FP32's range)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def counts(a):
    """rint((a - hi) / (2^-46 hi)) + 2^22 of FP64 values."""
    hi = a.astype(np.float32).astype(np.float64)
    with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
        q = np.rint((a - hi) / (hi * 2.0 ** -46))
    q = np.where(hi == 0.0, 0.0, np.clip(q, -(2.0 ** 22 - 1), 2.0 ** 22 - 1))
    return (q + 2 ** 22).astype(np.uint32)


def values(rng, n):
    v = rng.standard_normal(n) * 10.0 ** rng.integers(-12, 12, n)
    v[rng.random(n) < 0.05] = 0.0
    tie = rng.random(n) < 0.1  # few significant bits: exact counts and ties
    v[tie] = v[tie].astype(np.float32) * (1.0 + 2.0 ** -30 * rng.integers(-64, 64, tie.sum()))
    edge = rng.random(n) < 0.05  # FP32 subnormals, tiny and large normal numbers
    v[edge] = rng.choice([1e-45, 3e-40, 1.2e-38, 3.3e38, -2.1e-39], edge.sum()) * \
        (1.0 + 1e-3 * rng.random(edge.sum()))
    return v


@pytest.mark.parametrize("Nn,widest,order", [(1, 1, 0), (31, 5, 0), (33, 9, 0), (160, 12, 0),
                                             (129, 13, 0), (500, 16, 0), (129, 9, 1),
                                             (300, 14, 1)])
def test_fill_matches_definition(Nn, widest, order):
    from nbots_gb300 import _lib as L
    from nbots_gb300.device import DeviceArray
    lib = L.lib()
    rng = np.random.default_rng(Nn + widest)
    rows = []
    for v in range(Nn):
        n = min(Nn, int(rng.integers(1, widest + 1)))
        rows.append(np.unique(np.concatenate([[v], rng.choice(Nn, n - 1, replace=False)]
                                             if n > 1 else [[v]])).astype(np.int64))
    rp = np.zeros(2 * Nn + 1, np.uint32)
    ci = []
    for v, r in enumerate(rows):
        c = np.stack([2 * r, 2 * r + 1], 1).ravel()
        ci += [c, c]
        rp[2 * v + 1] = rp[2 * v] + c.size
        rp[2 * v + 2] = rp[2 * v + 1] + c.size
    ci = np.concatenate(ci).astype(np.uint32)
    val = values(rng, ci.size)
    for v, r in enumerate(rows):  # a diagonal to divide by
        k = int(np.searchsorted(r, v))
        val[rp[2 * v] + 2 * k], val[rp[2 * v + 1] + 2 * k + 1] = 2.0 + v, 3.0 - 7.0 * v
    perm = rng.permutation(Nn).astype(np.uint32) if order else np.arange(Nn, dtype=np.uint32)
    iperm = np.argsort(perm).astype(np.uint32)
    S = (Nn + 31) // 32
    so = np.zeros(S + 1, np.uint32)
    for s in range(S):
        so[s + 1] = so[s] + max(len(rows[perm[i]]) for i in range(32 * s, min(Nn, 32 * s + 32)))
    n = 32 * int(so[-1])
    dev = dict(so=DeviceArray(so), rp=DeviceArray(rp), ci=DeviceArray(ci), val=DeviceArray(val),
               perm=DeviceArray(perm), iperm=DeviceArray(iperm))
    out = dict(bcol=(n, np.uint32), b64=(4 * n, np.float64), b32=(4 * n, np.float32),
               blo=(4 * n, np.uint16), bxt=(4 * n, np.uint8), d64=(2 * Nn, np.float64),
               d32=(2 * Nn, np.float32))
    o = {k: DeviceArray(np.zeros(*s)) for k, s in out.items()}
    A = L.Bsr(2 * Nn, Nn, S, n, dev["so"].ptr, o["bcol"].ptr, o["b64"].ptr, o["b32"].ptr,
              o["blo"].ptr, o["bxt"].ptr, o["d64"].ptr, o["d32"].ptr,
              dev["perm"].ptr if order else None, dev["iperm"].ptr if order else None)
    assert lib.nbg_bsr_fill(C.byref(A), dev["rp"].ptr, dev["ci"].ptr, dev["val"].ptr, None) == 0
    bcol, b64 = np.zeros(n, np.uint32), np.zeros((n, 4))
    d64 = np.zeros(2 * Nn)
    for i in range(Nn):
        v, s, r = int(perm[i]), i // 32, i % 32
        for k in range(int(so[s + 1] - so[s])):
            e = (int(so[s]) + k) * 32 + r
            bcol[e] = i
            if k < len(rows[v]):
                bcol[e] = iperm[rows[v][k]]
                a, b = rp[2 * v] + 2 * k, rp[2 * v + 1] + 2 * k
                b64[e] = val[a], val[a + 1], val[b], val[b + 1]
                if rows[v][k] == v:
                    d64[2 * i], d64[2 * i + 1] = 1.0 / val[a], 1.0 / val[b + 1]
    written = np.zeros(n, bool)  # rows past Nn in the last slice stay as they were
    for s in range(S):
        lanes = np.arange(32) + 32 * s < Nn
        written[32 * so[s]:32 * so[s + 1]] = np.tile(lanes, int(so[s + 1] - so[s]))
    cm = b64[:, [0, 2, 1, 3]]  # column by column
    q = counts(cm)
    q[~written] = 0
    assert np.array_equal(o["bcol"].numpy(), bcol)
    assert np.array_equal(o["b64"].numpy().view(np.uint64), b64.ravel().view(np.uint64))
    assert np.array_equal(o["b32"].numpy().view(np.uint32),
                          cm.astype(np.float32).ravel().view(np.uint32))
    assert np.array_equal(o["blo"].numpy(), (q & 0xFFFF).astype(np.uint16).ravel())
    assert np.array_equal(o["bxt"].numpy(), (q >> 16).astype(np.uint8).ravel())
    assert np.array_equal(o["d64"].numpy().view(np.uint64), d64.view(np.uint64))
    assert np.array_equal(o["d32"].numpy(), d64.astype(np.float32))
