"""Draws from short rows: warps in which every draw, many of them, or a few have a
row of fewer than 32 totals, against the reference's walk
(matom_deactivation_from_matrix, macro_accelerate.c:995-1008)."""
import numpy as np
import pytest

from python_b200 import workloads as wl


@pytest.mark.gpu
@pytest.mark.parametrize("orders", [(1,), (2,), (10,), (30,), (31,), (32,), (3, 31, 32, 33), (5, 200, 200, 200, 200),
                                    (7, 100, 150, 200)])
@pytest.mark.parametrize("nq", [3, 400, 400003])
def test_draws_from_short_rows(engine, orders, nq):
    rng = np.random.default_rng([nq, *orders])
    n = rng.permutation(np.repeat(np.array(orders, np.int32), 3))
    offA = wl.offsets(n, True)
    rows = []
    for k in n:
        w = rng.random((k, k)) + 1e-3
        c = np.cumsum(w / w.sum(1, keepdims=True), 1) * rng.choice([1.0, 0.9], (k, 1))   # some end below z
        c[rng.random((k, k)) < 0.01] = np.nan              # a total that is not below anything
        rows.append(c)
    C = np.concatenate([r.ravel() for r in rows])
    sys = rng.integers(-1, n.size + 1, nq).astype(np.int32)
    inside = (sys >= 0) & (sys < n.size)
    lev = np.full(nq, 1, np.int32)
    lev[inside] = (rng.random(inside.sum()) * n[sys[inside]]).astype(np.int32)
    bad = rng.random(nq) < 0.02
    lev[bad] = rng.choice([-1, 300], bad.sum())
    z = rng.uniform(-0.05, 1.05, nq)
    z[rng.random(nq) < 0.02] = np.nan
    got = engine.matom_sample(n, offA, C, sys, lev, z)
    want = np.full(nq, -2)
    for s, k in enumerate(n):
        q = np.flatnonzero((sys == s) & (lev >= 0) & (lev < k))
        hit = ~(rows[s][lev[q]] < z[q, None])
        want[q] = np.where(0.0 < z[q], np.where(hit.any(1), hit.argmax(1), -1), 0)
    assert np.array_equal(got, want), np.flatnonzero(got != want)[:5]
