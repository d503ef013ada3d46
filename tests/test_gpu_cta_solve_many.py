"""Solves of the CTA family in a batch of more systems than the inverse's shapes run
at once, where the classes of many solves (cta_solve_classes.inc) take over: every
class, both sides of its edges, in memory of its own and in place, with codes 0,
2, 3 and 4.  Bits against the oracle."""
import re
from pathlib import Path

import numpy as np
import pytest

from oracle import oracle
from python_b200 import workloads as wl
from helpers import same_values

CSRC = Path(__file__).resolve().parent.parent / "python_b200" / "csrc"


def _tops(name, macro):
    return [int(m) for m in re.findall(rf"^{macro}\(\d+, (\d+),", (CSRC / name).read_text(), re.M)]


TOPS = _tops("cta_solve_classes.inc", "SS_CTA_SOLVE_CLASS")
ORDERS = sorted({33, 34, 39, 44, 57, 73, 1023} | {t + d for t in TOPS for d in (-1, 0, 1) if t + d <= 513} | set(TOPS))
PAD = 4000      # systems of order 33: several times what any shape runs at once


def test_classes_cover_the_family():
    assert TOPS == sorted(TOPS) and TOPS[-1] == 1024 == _tops("cta_classes.inc", "SS_CTA_CLASS")[-1]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["dense", "graded", "integers"])
def test_many_solves_bit_identical(engine, kind):
    import torch
    rng = np.random.default_rng([5, len(kind)])
    mats, rhs = [], []
    for n in ORDERS:
        if kind != "dense" and n > 520:
            continue
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
    few = wl.from_matrices("solve", mats, rhs)
    xr, sr = oracle.solve(few, "port")
    at = len(mats)
    pads = [(rng.standard_normal((33, 33)), rng.standard_normal(33)) for _ in range(7)]
    for i in range(PAD):
        mats.append(pads[i % 7][0])
        rhs.append(pads[i % 7][1])
    order = rng.permutation(len(mats))
    b = wl.from_matrices("solve", [mats[i] for i in order], [rhs[i] for i in order])
    pad = wl.from_matrices("solve", [p[0] for p in pads], [p[1] for p in pads])
    xp, sp = oracle.solve(pad, "port")

    dev = torch.device("cuda", 0)
    A, db = torch.from_numpy(b.A).to(dev), torch.from_numpy(b.b).to(dev)
    plan = engine.Plan(b, engine.FP64)
    if kind == "dense":
        # a launch per class: the table of many solves has one class more than the inverse's
        assert plan.launches == len(TOPS) == len(_tops("cta_classes.inc", "SS_CTA_CLASS")) + 1
    for x in (torch.zeros_like(db), db):        # the second time in place
        st = torch.full((b.nsys,), -9, dtype=torch.int32, device=dev)
        plan.execute(A, x, st, b=db)
        torch.cuda.synchronize()
        xh, sh = x.cpu().numpy(), st.cpu().numpy()
        for pos, i in enumerate(order):
            ref, rx, code = (few, xr, sr) if i < at else (pad, xp, sp)
            j = i if i < at else (i - at) % 7
            n = int(ref.n[j])
            assert sh[pos] == code[j], (n, sh[pos], code[j])
            if code[j] != 4:
                o, r = int(b.offv[pos]), int(ref.offv[j])
                assert same_values(xh[o:o + n], rx[r:r + n]).all(), n
    plan.close()
    if kind == "integers":
        assert (sr == 4).any()
    if kind == "graded":
        assert {2, 3} & set(sr.tolist())
