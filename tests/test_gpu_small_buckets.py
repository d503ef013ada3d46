"""Batches of small systems whose buckets do not all run the same way: some fill the
GPU and run in turn, others are forked beside them, as enqueued and as captured in
a CUDA graph; and mixed-mode warps of which some groups fall back to the exact
solve while the others do not."""
import numpy as np
import pytest

from oracle import oracle
from python_b200 import workloads as wl
from helpers import same_values

# order: systems.  Four systems a block above 16: 9,000 and 6,000 fill the GPU twice over; the others do not.
COUNTS = {27: 9000, 20: 6000, 14: 500, 5: 200, 40: 50, 70: 20}


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["solve", "invert"])
@pytest.mark.parametrize("mode", ["FP64", "MIXED", "FAST"])
def test_filling_and_forked_buckets_captured(engine, kind, mode):
    import torch
    rng = np.random.default_rng(23)
    base = {n: [(rng.standard_normal((n, n)) + np.eye(n) * n, rng.standard_normal(n)) for _ in range(5)]
            for n in COUNTS}
    which = [(n, i % 5) for n, k in COUNTS.items() for i in range(k)]
    which = [which[i] for i in rng.permutation(len(which))]
    b = wl.from_matrices(kind, [base[n][i][0] for n, i in which], [base[n][i][1] for n, i in which])
    dev = torch.device("cuda", 0)
    A = torch.from_numpy(b.A).to(dev)
    rhs = torch.from_numpy(b.b).to(dev) if kind == "solve" else None
    out = torch.zeros_like(A if kind == "invert" else rhs)
    st = torch.full((b.nsys,), -9, dtype=torch.int32, device=dev)
    plan = engine.Plan(b, getattr(engine, mode))
    plan.execute(A, out, st, b=rhs)
    torch.cuda.synchronize()
    want, codes = out.cpu().numpy(), st.cpu().numpy()
    assert (codes == 0).all()
    if kind == "solve" and mode != "MIXED":
        few = wl.from_matrices("solve", [m for n in COUNTS for m, _ in base[n]], [v for n in COUNTS for _, v in base[n]])
        xr, _ = oracle.solve(few, "port")
        at = {n: 5 * j for j, n in enumerate(COUNTS)}
        for s, (n, i) in enumerate(which):
            o, r = int(b.offv[s]), int(few.offv[at[n] + i])
            assert same_values(want[o:o + n], xr[r:r + n]).all(), n
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        with torch.cuda.graph(g, stream=s):
            plan.execute(A, out, st, b=rhs, stream=s)
    for _ in range(2):
        out.zero_()
        st.fill_(-9)
        g.replay()
        torch.cuda.synchronize()
        assert same_values(out.cpu().numpy(), want).all() and np.array_equal(st.cpu().numpy(), codes)
    del g
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 4, 6, 8, 11, 12, 15, 16, 20, 27, 32])
def test_mixed_groups_that_fall_back_beside_others(engine, n):
    import torch
    rng = np.random.default_rng(n)
    mats, rhs, hard = [], [], []
    for i in range(203):
        a = rng.standard_normal((n, n)) + 2.0 * n * np.eye(n)
        kind = rng.integers(0, 5)
        if kind == 0:                     # rank one apart from 1e-12: its FP32 factors say nothing
            v = 1.0 + rng.random(n)
            a = np.outer(v, v) + 1e-12 * a
        elif kind == 1:                   # a repeated row: code 4
            a[n - 1] = a[0]
        hard.append(kind <= 1)
        mats.append(a)
        rhs.append(rng.standard_normal(n))
    b = wl.from_matrices("solve", mats, rhs)
    xr, sr = oracle.solve(b, "port")
    dev = torch.device("cuda", 0)
    A, db = torch.from_numpy(b.A).to(dev), torch.from_numpy(b.b).to(dev)
    x = torch.zeros_like(db)
    st, diag = (torch.full((b.nsys,), -9, dtype=torch.int32, device=dev) for _ in range(2))
    plan = engine.Plan(b, engine.MIXED)
    plan.execute(A, x, st, b=db, diag=diag)
    torch.cuda.synchronize()
    plan.close()
    x, st, diag = x.cpu().numpy(), st.cpu().numpy(), diag.cpu().numpy()
    exact = (diag & 256) != 0
    assert np.array_equal(st, sr)
    assert exact[np.array(hard)].all() and not exact.all()
    for s in np.flatnonzero(sr != 4):
        v, r = x[s * n:s * n + n], xr[s * n:s * n + n]
        if exact[s]:
            assert same_values(v, r).all(), s
        else:
            assert np.max(np.abs(v - r)) <= 1e-10 * np.max(np.abs(r)), s
