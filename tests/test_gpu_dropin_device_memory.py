"""The drop-in calls with buffers that are not plain host memory: device and
page-locked ones, alone and mixed, on both sides of the orders that a warp
solves and of the page-locked path's bound."""
import ctypes

import numpy as np
import pytest

from oracle import oracle
from python_b200 import workloads as wl
from helpers import same_values


@pytest.fixture(scope="module")
def lib(engine):
    lib = engine.load()
    solve, invert = lib.gpu_solve_matrix, lib.gpu_invert_matrix
    saved = solve.argtypes, invert.argtypes
    solve.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    invert.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]
    yield lib
    solve.argtypes, invert.argtypes = saved


def _place(a, where):
    import torch
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t.cuda() if where == "device" else t.pin_memory() if where == "pinned" else t.clone()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5, 32, 33, 100, 400])
@pytest.mark.parametrize("where", ["device device device", "host host device", "device host host", "host device host",
                                   "pinned pinned pinned", "pinned device host"])
def test_drop_in_buffers(lib, n, where):
    import torch
    wa, wb, wx = where.split()
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal((n, n)) + n * np.eye(n), rng.standard_normal(n)
    sx, ss = oracle.solve(wl.from_matrices("solve", [a], [b]), "port")
    A, B, X = _place(a, wa), _place(b, wb), _place(np.full(n, np.nan), wx)
    inv = _place(np.full((n, n), np.nan), wx)
    torch.cuda.synchronize()
    assert lib.gpu_solve_matrix(A.data_ptr(), B.data_ptr(), n, X.data_ptr()) == ss[0] == 0
    assert same_values(X.cpu().numpy(), sx).all()
    assert lib.gpu_invert_matrix(A.data_ptr(), inv.data_ptr(), n) == 0
    assert np.max(np.abs(inv.cpu().numpy() @ a - np.eye(n))) < 1e-10
    assert np.array_equal(A.cpu().numpy(), a) and np.array_equal(B.cpu().numpy(), b)
    # a singular system leaves x and the inverse alone
    sing = _place(np.ones((n, n)), wa)
    X, inv = _place(np.full(n, 7.0), wx), _place(np.full((n, n), 7.0), wx)
    torch.cuda.synchronize()
    assert lib.gpu_solve_matrix(sing.data_ptr(), B.data_ptr(), n, X.data_ptr()) == 4
    assert lib.gpu_invert_matrix(sing.data_ptr(), inv.data_ptr(), n) == 1
    assert (X.cpu().numpy() == 7.0).all() and (inv.cpu().numpy() == 7.0).all()
