"""Solves of the CTA family at the edges of its upper sweep and residual check:
8-column pieces, 32-row check tiles, 256-column sweep pieces, the class edges,
with codes 0, 2, 3 and 4.  Bits against the oracle."""
import numpy as np
import pytest

from oracle import oracle
from python_b200 import workloads as wl
from helpers import same_values

ORDERS = (33, 39, 40, 41, 47, 48, 49, 63, 64, 65, 79, 80, 81, 95, 96, 97, 127, 128, 129, 160, 161, 192, 193, 207, 208, 209, 223,
          224, 225, 255, 256, 257, 263, 264, 320, 321, 384, 385, 448, 449, 511, 512, 513)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["dense", "graded", "integers"])
def test_cta_solves_bit_identical(engine, kind):
    rng = np.random.default_rng([3, len(kind)])
    mats, rhs = [], []
    for n in ORDERS:
        a, b = rng.standard_normal((n, n)), rng.standard_normal(n)
        if kind == "graded":            # rows of very different size: rows failing the residual check
            a *= np.exp2(rng.integers(-40, 41, (n, 1)).astype(float))
            b = np.abs(b) * np.exp2(rng.integers(-40, 41, n).astype(float))
        elif kind == "integers":        # ties, and a repeated row in every third system: code 4
            a = rng.integers(-3, 4, (n, n)).astype(float)
            if n % 3 == 0:
                a[n - 1] = a[0]
        mats.append(a)
        rhs.append(b)
    b = wl.from_matrices("solve", mats, rhs)
    x, st = engine.solve_batched(b)
    xr, sr = oracle.solve(b, "port")
    assert np.array_equal(st, sr)
    for s in range(b.nsys):
        if sr[s] != 4:
            o, n = int(b.offv[s]), int(b.n[s])
            assert same_values(x[o:o + n], xr[o:o + n]).all(), n
