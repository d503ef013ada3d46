"""The certified macro-atom epilogue on several matrices in a row per CTA and per
cluster: the next matrix's first pivot inverse, written into every CTA of a
cluster, must not meet the running totals of the one before.  B and C against the
plain certified inverse: B = N^-1 diag(R), one rounding per product, and C its
running totals from left to right, so every bit is determined."""
import ctypes

import numpy as np
import pytest

from python_b200 import workloads as wl


@pytest.mark.gpu
@pytest.mark.parametrize("n", [36, 48, 64, 96, 127, 128, 139, 144, 153, 160, 161, 176, 187, 192, 200, 208, 217, 224])
@pytest.mark.parametrize("totals", [True, False])
def test_epilogue_over_many_matrices(engine, n, totals):
    import torch
    k = 1200 if n < 100 else 500            # at least three a CTA or cluster where few of them fit the GPU
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(n)
    q = torch.rand((k, n, n), generator=g, dtype=torch.float64, device=dev)
    q *= torch.rand((k, n, n), generator=g, dtype=torch.float64, device=dev) < 0.3
    q[1, 0, 1] = 40.0                        # rows of very different size
    q.diagonal(dim1=1, dim2=2).zero_()
    N = torch.eye(n, dtype=torch.float64, device=dev) - q / (q.sum(2, keepdim=True) * 1.05 + 1e-3)
    N[5] = torch.rand((n, n), generator=g, dtype=torch.float64, device=dev)   # not an M-matrix: the exact path
    N = N.contiguous()
    R = torch.rand((k, n), generator=g, dtype=torch.float64, device=dev)
    ns = np.full(k, n, np.int32)
    offA, offv = wl.offsets(ns, True), wl.offsets(ns, False)
    inv, B = torch.empty_like(N), torch.full_like(N, np.nan)
    C = torch.full_like(N, np.nan) if totals else None
    st = torch.full((k,), -9, dtype=torch.int32, device=dev)
    st2 = torch.full_like(st, -9)
    plan = engine.Plan(wl.Batch("invert", ns, offA, np.empty(0)), engine.FAST)
    plan.execute(N, inv, st)
    torch.cuda.synchronize()
    h = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    d = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None
    engine.set_precision(engine.FAST)
    rc = engine.load().matom_matrices_batched(k, h(ns), h(offA), h(offv), d(N), d(R), d(B), d(C), d(st2))
    engine.set_precision(engine.FP64)
    assert rc == 0, engine.last_error()
    plan.close()
    assert int((st != 0).sum()) == 0 and int((st2 != 0).sum()) == 0
    want = inv * R[:, None, :]
    assert torch.equal(B, want)
    if totals:
        total = torch.zeros((k, n), dtype=torch.float64, device=dev)
        for c in range(n):
            total = total + want[:, :, c]
            assert torch.equal(C[:, :, c], total), c
