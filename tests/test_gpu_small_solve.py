"""The warp-group solves (orders 1-32) where their fast paths end: group and row
edges, pivots whose reciprocal or quotients leave the range of the branch-free
forms, equal magnitudes, and warps holding several orders.  Bits against the
oracle; its loops are GSL's, so nothing but equality is a pass."""
import numpy as np
import pytest

from oracle import oracle
from python_b200 import workloads as wl
from helpers import same_values

ORDERS = (1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 15, 16, 17, 20, 21, 24, 25, 27, 28, 29, 31, 32)


def _systems(kind, rng):
    mats, rhs = [], []
    for rep in range(5):
        for n in ORDERS:
            a = rng.standard_normal((n, n))
            b = rng.standard_normal(n)
            if kind == "ties":              # small integers: equal magnitudes, zero pivots, singular systems
                a = rng.integers(-2, 3, (n, n)).astype(float)
            elif kind == "wide":            # quotients beyond 2^+-900, so the sweep is done over by divisions
                a *= np.exp2(rng.integers(-30, 31, (n, 1)).astype(float))
                b *= np.exp2(rng.choice([-1000.0, -940.0, 0.0, 940.0], n))
            elif kind == "tiny":            # pivots below 2^-1021 and subnormal: divided by, not scaled
                a *= np.exp2(rng.choice([-1022.0, -1030.0, -1060.0], (n, 1)))
            elif kind == "huge":
                a *= 2.0 ** 1021
            elif kind == "ones":            # pivots whose significand is all ones
                a = np.where(rng.random((n, n)) < 0.3, np.nextafter(2.0, 0.0) * np.exp2(rng.integers(-3, 3, (n, n))),
                             a * 1e-3)
            elif kind == "ion":
                a, b = wl.ion_matrix(rng, n)
            elif kind == "zero":            # right-hand sides with exact and negative zeros
                b = np.where(rng.random(n) < 0.7, rng.choice([0.0, -0.0], n), b)
                a = np.triu(a) if rep % 2 else a
            mats.append(a)
            rhs.append(b)
    order = rng.permutation(len(mats))
    return wl.from_matrices("solve", [mats[i] for i in order], [rhs[i] for i in order])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["dense", "ties", "wide", "tiny", "huge", "ones", "ion", "zero"])
def test_small_solves_bit_identical(engine, kind):
    b = _systems(kind, np.random.default_rng([11, len(kind), ord(kind[0])]))
    x, st = engine.solve_batched(b)
    xr, sr = oracle.solve(b, "port")
    assert np.array_equal(st, sr), np.flatnonzero(st != sr)[:5]
    for s in range(b.nsys):
        if sr[s] != 4:
            o, n = int(b.offv[s]), int(b.n[s])
            assert same_values(x[o:o + n], xr[o:o + n]).all(), (s, n)
