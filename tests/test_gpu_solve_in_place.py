"""Device solves whose x is the same buffer as b, in every kernel family that
serves a solve: x and status are those of a solve into a buffer of its own.  The
reference's residual check (matrix_cpu.c:155-187) compares A x with b, so a
kernel has to read b for the last time before it stores x."""
import ctypes

import numpy as np
import pytest

from oracle import oracle
from python_b200 import workloads as wl
from helpers import same_values

ORDERS = (1, 4, 7, 16, 27, 32, 33, 40, 48, 49, 64, 65, 96, 97, 128, 150, 192, 200, 256, 257, 320, 384, 400, 512, 600)


def _batch(rng):
    mats, rhs = [], []
    for rep in range(3):
        for n in ORDERS:
            a, b = rng.standard_normal((n, n)), rng.standard_normal(n)
            if rep == 1:                    # rows of very different size: some fail the residual check
                a *= np.exp2(rng.integers(-40, 41, (n, 1)).astype(float))
                b = np.abs(b) * np.exp2(rng.integers(-40, 41, n).astype(float))
            if rep == 2 and n > 1:          # a repeated row: code 4
                a = rng.integers(-3, 4, (n, n)).astype(float)
                a[n - 1] = a[0]
            mats.append(a)
            rhs.append(b)
    return wl.from_matrices("solve", mats, rhs)


@pytest.mark.gpu
@pytest.mark.parametrize("entry", ["plan", "batched"])
@pytest.mark.parametrize("mode", ["FP64", "MIXED"])
def test_solve_in_place(engine, entry, mode):
    import torch
    b = _batch(np.random.default_rng(17))
    mode = getattr(engine, mode)
    dev = torch.device("cuda", 0)
    A = torch.from_numpy(b.A).to(dev)
    n = np.ascontiguousarray(b.n, np.int32)

    def run(rhs, x):
        st = torch.full((b.nsys,), -99, dtype=torch.int32, device=dev)
        if entry == "plan":
            plan = engine.Plan(b, mode)
            plan.execute(A, x, st, b=rhs)
            torch.cuda.synchronize()
            plan.close()
        else:
            h = lambda a: a.ctypes.data_as(ctypes.c_void_p)
            d = lambda t: ctypes.c_void_p(t.data_ptr())
            torch.cuda.synchronize()
            engine.set_precision(mode)
            rc = engine.load().solve_matrix_batched(b.nsys, h(n), h(b.offA), d(A), h(b.offv), d(rhs), d(x), d(st))
            engine.set_precision(engine.FP64)
            assert rc == 0, engine.last_error()
        return x.cpu().numpy(), st.cpu().numpy()

    rhs = torch.from_numpy(b.b).to(dev)
    x, st = run(rhs, torch.zeros_like(rhs))
    assert np.array_equal(rhs.cpu().numpy(), b.b)
    xi, sti = run(rhs, rhs)
    if mode == engine.FP64:
        xr, sr = oracle.solve(b, "port")
        assert np.array_equal(st, sr) and {0, 2, 3, 4} <= set(sr.tolist())
    assert np.array_equal(sti, st), [(int(b.n[s]), int(sti[s]), int(st[s])) for s in np.flatnonzero(sti != st)]
    for s in np.flatnonzero(st != 4):
        o, k = int(b.offv[s]), int(b.n[s])
        assert same_values(xi[o:o + k], x[o:o + k]).all(), k
        if mode == engine.FP64:
            assert same_values(xi[o:o + k], xr[o:o + k]).all(), k
