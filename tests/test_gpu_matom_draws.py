"""Draws at the edges of the draw kernel: fewer draws than slots or lanes, rows
around its 32-column rounds, totals that never reach z, NaN totals, z outside
(0, 1) and out-of-range cells and levels, against the reference's walk
(matom_deactivation_from_matrix, macro_accelerate.c:995-1008)."""
import numpy as np
import pytest

from python_b200 import workloads as wl


@pytest.mark.gpu
@pytest.mark.parametrize("nq", [1, 3, 5, 31, 33, 257, 5000, 60000])
def test_draws_match_the_walk(engine, nq):
    rng = np.random.default_rng(nq)
    n = np.array([1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 200], np.int32)
    offA = wl.offsets(n, True)
    rows = []
    for k in n:
        w = rng.random((k, k)) + 1e-3
        c = np.cumsum(w / w.sum(1, keepdims=True), 1)
        if k == 33:
            c[::2] = c[::2, ::-1]          # totals that fall: the first hit still decides
        if k == 64:
            c[3, 5] = np.nan               # a total that is not below anything
        rows.append(c.ravel())
    C = np.concatenate(rows)
    sys = rng.integers(-1, n.size + 1, nq).astype(np.int32)
    lev = rng.integers(-1, 201, nq).astype(np.int32)
    inside = (sys >= 0) & (sys < n.size) & (rng.random(nq) < 0.9)
    lev[inside] = (rng.random(inside.sum()) * n[sys[inside]]).astype(np.int32)
    z = rng.uniform(-0.05, 1.05, nq)
    z[rng.random(nq) < 0.02] = np.nan
    got = engine.matom_sample(n, offA, C, sys, lev, z)
    for i in range(nq):
        s, u = int(sys[i]), int(lev[i])
        if s < 0 or s >= n.size or u < 0 or u >= n[s]:
            want = -2
        elif not 0.0 < z[i]:
            want = 0
        else:
            row = C[offA[s] + u * n[s]:offA[s] + (u + 1) * n[s]]
            hit = np.flatnonzero(~(row < z[i]))
            want = int(hit[0]) if hit.size else -1
        assert got[i] == want, (i, s, u, z[i])
