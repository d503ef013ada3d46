"""rcp_markstein and div_markstein (ss_common.cuh) against correctly rounded
division, bit for bit, wherever the solves use them: over the whole range, at its
ends, at significands next to 1 and to 2, with signed zeros, and with quotients on
either side of 2^+-900, where div_markstein hands over to a division."""
import ctypes

import numpy as np
import pytest

COUNT = 1 << 22


def _significands(rng, k):
    m = rng.integers(0, 1 << 52, k, dtype=np.uint64)
    edge = np.array([0, 1, 2, 3, (1 << 52) - 1, (1 << 52) - 2, (1 << 32) - 1, 1 << 32, ((1 << 20) - 1) << 32, 1 << 51,
                     (1 << 51) - 1], np.uint64)
    near = rng.random(k) < 0.3
    m[near] = rng.choice(edge, near.sum())
    low = rng.random(k) < 0.1               # low word all ones: not covered
    m[low] |= np.uint64(0xffffffff)
    return m


def _values(rng, k, lo, hi):
    e = (rng.integers(lo, hi + 1, k) + 1023).astype(np.uint64)
    s = rng.integers(0, 2, k, dtype=np.uint64)
    return ((s << np.uint64(63)) | (e << np.uint64(52)) | _significands(rng, k)).view(np.float64)


def _run(lib, u, d):
    import torch
    dev = torch.device("cuda", 0)
    du, dd = torch.from_numpy(u).to(dev), torch.from_numpy(d).to(dev)
    r, q = torch.empty_like(du), torch.empty_like(du)
    c, f = (torch.empty(u.size, dtype=torch.int32, device=dev) for _ in range(2))
    torch.cuda.synchronize()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    assert lib.sirocco_check_rounding(u.size, p(du), p(dd), p(r), p(c), p(q), p(f)) == 0
    return r.cpu().numpy(), c.cpu().numpy() != 0, q.cpu().numpy(), f.cpu().numpy().view(np.uint32)


def _bits(a):
    return a.view(np.uint64)


@pytest.fixture(scope="module")
def lib(engine):
    from python_b200 import build
    lib = ctypes.CDLL(str(build.build_rounding_check()))
    lib.sirocco_check_div_far.restype = ctypes.c_uint
    lib.sirocco_check_rounding.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 6
    return lib


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["all", "ends", "one"])
def test_reciprocals(lib, case):
    rng = np.random.default_rng(len(case))
    if case == "all":
        d = _values(rng, COUNT, -1022, 1023)
    elif case == "ends":
        d = _values(rng, COUNT, -1022, -1019)
        d[::2] = _values(rng, d[::2].size, 1018, 1023)
        d[:6] = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324]
    else:
        d = _values(rng, COUNT, -2, 2)
    r, covers, _, _ = _run(lib, np.ones_like(d), d)
    ex = np.abs(d)
    low = (_bits(d) & np.uint64(0xffffffff)) == np.uint64(0xffffffff)
    assert np.array_equal(covers, (ex >= 2.0 ** -1021) & (ex < 2.0 ** 1021) & ~low)
    assert covers.sum() > COUNT // 4
    want = 1.0 / d[covers]
    bad = np.flatnonzero(_bits(r[covers]) != _bits(want))
    assert bad.size == 0, (bad.size, d[covers][bad[:4]])


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["all", "near one", "edge of the range", "zeros and others"])
def test_quotients(lib, case):
    rng = np.random.default_rng(10 + len(case))
    far_at = lib.sirocco_check_div_far()
    if case == "all":
        u, d = _values(rng, COUNT, -1022, 1023), _values(rng, COUNT, -1022, 1023)
    elif case == "near one":
        u, d = _values(rng, COUNT, -3, 3), _values(rng, COUNT, -3, 3)
        d[::3] = np.nextafter(u[::3], 0.0)
    elif case == "edge of the range":       # quotients, and numerators, next to 2^+-900
        d = _values(rng, COUNT, -120, 120)
        u = _values(rng, COUNT, -1, 1)
        e = (_bits(d) >> np.uint64(52) & np.uint64(0x7ff)).astype(int) - 1023
        with np.errstate(over="ignore"):
            u = np.ldexp(u, np.where(rng.random(COUNT) < 0.5, 900, -900) + np.where(rng.random(COUNT) < 0.5, e, 0))
    else:
        u, d = _values(rng, COUNT, -1022, 1023), _values(rng, COUNT, -1022, 1023)
        u[::2] = rng.choice([0.0, -0.0], u[::2].size)
        u[1::8] = rng.choice([np.inf, -np.inf, np.nan, 5e-324, -1e-310], u[1::8].size)
        d[2::16] = rng.choice([0.0, np.inf, np.nan, -5e-324], d[2::16].size)
    _, covers, q, far = _run(lib, u, d)
    with np.errstate(all="ignore"):
        want = u / d
    use = far < far_at
    # in use exactly where the reciprocal is, and u is zero or both u and the
    # quotient lie in [2^-900, 2^900)
    au, aq = np.abs(u), np.abs(want)
    inside = covers & ((u == 0.0) | ((au >= 2.0 ** -900) & (au < 2.0 ** 900) & (aq >= 2.0 ** -900) & (aq < 2.0 ** 900)))
    assert np.array_equal(use, inside), np.flatnonzero(use != inside)[:4]
    assert use.sum() > COUNT // 16
    bad = np.flatnonzero(_bits(q[use]) != _bits(want[use]))
    assert bad.size == 0, (bad.size, u[use][bad[:4]], d[use][bad[:4]])
