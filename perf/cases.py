"""The timed workloads of the batched dense-solve engine.

Each case is one call, or one plan execution, that a Sirocco-like host program
makes per ionisation cycle (or per photon batch), through the engine's public
entry points: the drop-in calls, the batched host calls, device plans in their
precision modes, the macro-atom epilogue and draws, and the lock-step n_e
iteration.  Inputs follow the repository's own generators
(python_b200/workloads.py), formed on the GPU where they are large.
"""
import ctypes
import math

import numpy as np
import torch

from python_b200 import engine
from python_b200 import workloads as wl

# orders of the ion-balance systems one cell carries: H, He and eight metals
CELL_ORDERS = (2, 3, 7, 8, 9, 11, 13, 15, 17, 27)
MODES = {"fp64": engine.FP64, "fast": engine.FAST}
# lock-step tables: hydrogen first, the abundances of its elements
ZS = (1, 2, 6, 8, 26)
ABUND = np.array([1.0, 0.1, 3e-4, 5e-4, 3e-5])


def listed():
    return [
        # a host that calls solve_matrix cell by cell (matrix_ion.c:276): one iron-sized system in host memory
        {"name": "solve one 27", "do": "one", "kind": "solve", "n": 27},
        # one element's systems of every cell of a wind grid, resident on the GPU
        {"name": "ion solves 4096x27", "do": "ion", "cells": 4096, "n": 27},
        # all ten elements of every cell, shuffled, one plan per cycle
        {"name": "ion solves mixed", "do": "ion", "cells": 20000, "n": 0},
        # the same systems handed over in pinned host memory by a C host
        {"name": "ion solves from host", "do": "host", "cells": 4096},
        # level populations of macro elements (macro_gov.c:444): general solves above 32 levels
        {"name": "level solves 33-200", "do": "levels", "nsys": 4096, "lo": 33, "hi": 200},
        # the default precision mode's inverses of the macro-atom matrices: GSL-exact
        {"name": "exact inverses 20-200", "do": "inverse", "mode": "fp64", "nsys": 8192, "lo": 20, "hi": 200,
         "density": 0.25},
        # one macro-atom model in every cell: all matrices of one order, certified mode
        {"name": "inverses 8192x61", "do": "inverse", "mode": "fast", "nsys": 8192, "lo": 61, "hi": 61,
         "density": 0.25},
        # mixed models over a 50,000-cell grid, certified mode
        {"name": "inverses 50000x20-200", "do": "inverse", "mode": "fast", "nsys": 50000, "lo": 20, "hi": 200,
         "density": 0.25},
        # large macro atoms
        {"name": "inverses 2048x256-1024", "do": "inverse", "mode": "fast", "nsys": 2048, "lo": 256, "hi": 1024,
         "density": 0.10},
        # a cycle's jumping matrices left on the GPU: B = N^-1 diag(R) and its running totals
        {"name": "matom B and C", "do": "matom", "mode": "fast", "nsys": 8192, "lo": 20, "hi": 200},
        # a photon batch's macro-atom activations drawn from those totals
        {"name": "matom draws", "do": "draws", "nq": 1 << 20, "nsys": 4096, "lo": 20, "hi": 200},
        # the n_e iteration of every cell, rate matrices assembled on the GPU
        {"name": "ion lock-step", "do": "lockstep", "cells": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges."""
    do = rng.choice(["one", "ion", "ion", "host", "levels", "inverse", "inverse", "inverse", "matom", "draws",
                     "lockstep"])
    if do == "one":
        return {"do": do, "kind": rng.choice(["solve", "invert"]), "n": _log(rng, 2, 200)}
    if do == "ion":
        n = rng.choice([0, 0] + list(range(2, 33)))
        return {"do": do, "cells": _log(rng, 256, 20000 if n == 0 else 100000), "n": n}
    if do == "host":
        return {"do": do, "cells": _log(rng, 100, 10000)}
    if do == "levels":
        lo = _log(rng, 33, 200)
        return {"do": do, "nsys": _log(rng, 256, 6000), "lo": lo, "hi": min(256, lo + rng.choice([0, 7, 50, 167]))}
    if do == "inverse":
        mode = rng.choice(["fast", "fast", "fp64"])
        lo = _log(rng, 20, 1000 if mode == "fast" else 300)
        hi = min(1024, lo + rng.choice([0, 0, 5, lo // 2, 180]))
        most = 4e11 if mode == "fast" else 1e11   # flops
        nsys = _log(rng, 64, max(128, min(50000, int(most / (2.0 * ((lo + hi) / 2) ** 3)))))
        return {"do": do, "mode": mode, "nsys": nsys, "lo": lo, "hi": hi, "density": rng.choice([0.10, 0.25])}
    if do == "matom":
        lo = _log(rng, 20, 200)
        hi = min(400, lo + rng.choice([0, 5, lo // 2, 180]))
        nsys = _log(rng, 64, max(128, min(20000, int(8e10 / (2.0 * ((lo + hi) / 2) ** 3)))))
        return {"do": do, "mode": rng.choice(["fast", "fast", "fp64"]), "nsys": nsys, "lo": lo, "hi": hi}
    if do == "draws":
        lo = _log(rng, 10, 300)
        return {"do": do, "nq": _log(rng, 1000, 4000000), "nsys": _log(rng, 16, 4096), "lo": lo,
                "hi": lo + rng.choice([0, 40, 180])}
    return {"do": do, "cells": _log(rng, 64, 16384)}


# ------------------------------------------------------------------ layouts --
def _orders(case):
    """The orders of a case's systems: the layout a program keeps from cycle to cycle."""
    do = case["do"]
    if do == "one":
        return np.array([case["n"]], np.int32)
    if do in ("ion", "host"):
        if case.get("n", 0):
            return np.full(case["cells"], case["n"], np.int32)
        o = np.tile(np.array(CELL_ORDERS, np.int32), case["cells"])
        np.random.RandomState(case["cells"]).shuffle(o)
        return o
    r = np.random.RandomState([case["nsys"], case["lo"], case["hi"]])
    return r.randint(case["lo"], case["hi"] + 1, case["nsys"]).astype(np.int32)


def _groups(n, chunk=1 << 24):
    """(order, systems of that order), in pieces of at most `chunk` matrix elements."""
    order = np.argsort(n, kind="stable")
    vals, first = np.unique(n[order], return_index=True)
    for v, part in zip(vals, np.split(order, first[1:])):
        k = max(1, chunk // (int(v) * int(v)))
        for i in range(0, part.size, k):
            yield int(v), part[i:i + k]


def _at(off, part, k, dev):
    """Positions of the k packed elements of each listed system."""
    return torch.from_numpy(off[part]).to(dev)[:, None] + torch.arange(k, device=dev)[None, :]


def _lu(g, lo, hi, *shape):
    r = torch.rand(*shape, generator=g, dtype=torch.float64, device=g.device)
    return torch.exp(math.log(lo) + r * (math.log(hi) - math.log(lo)))


def _bern(g, p, *shape):
    return torch.rand(*shape, generator=g, device=g.device) < p


# ------------------------------------------------------------------- inputs --
def _ion_matrices(g, m, n):
    """m ion-balance systems of order n (workloads.ion_matrix): last row ones, b = e_last.  The few that
    meet a zero pivot (code 4: no solution is written) are replaced by another one."""
    a = torch.zeros(m, n, n, dtype=torch.float64, device=g.device)
    for d in (1, 2, 3, 4):
        if n > d:
            down = _lu(g, 1e-14, 1e2, m, n - 1) if d == 1 else \
                torch.where(_bern(g, 0.1, m, n - d), _lu(g, 1e-16, 1e-6, m, n - d), 0.0)
            a.diagonal(-d, 1, 2).copy_(down)
    if n > 1:
        a.diagonal(1, 1, 2).copy_(_lu(g, 1e-14, 1e2, m, n - 1))
    a.diagonal(0, 1, 2).copy_(-a.sum(1))
    a[:, n - 1, :] = 1.0
    b = torch.zeros(m, n, dtype=torch.float64, device=g.device)
    b[:, n - 1] = 1.0
    bad = (_factor(a.clone(), b.clone()) == 0.0).any(1)
    return torch.where(bad[:, None, None], a[torch.argmin(bad.int())], a), b


def _level_matrices(g, m, n):
    """m macro-atom level systems of order n: rates between about a third of the level pairs and
    between neighbours, first row ones, b = e_0 (macro_gov.c:401-431)."""
    a = torch.where(_bern(g, 0.35, m, n, n), _lu(g, 1e-4, 1e4, m, n, n), 0.0)
    if n > 1:
        a.diagonal(-1, 1, 2).copy_(_lu(g, 1e-2, 1e4, m, n - 1))
        a.diagonal(1, 1, 2).copy_(_lu(g, 1e-2, 1e4, m, n - 1))
    a.diagonal(0, 1, 2).zero_()
    a.diagonal(0, 1, 2).copy_(-a.sum(1))
    a[:, 0, :] = 1.0
    b = torch.zeros(m, n, dtype=torch.float64, device=g.device)
    b[:, 0] = 1.0
    return a, b


def _macro_matrices(g, m, n, density):
    """m macro-atom matrices N = I - Q of order n (workloads.macro_matrix) and their row sums R."""
    q = torch.where(_bern(g, density, m, n, n), _lu(g, 1e-8, 1.0, m, n, n), 0.0)
    q.diagonal(0, 1, 2).zero_()
    q *= (~_bern(g, 0.03, m, n, 1)).double()
    rs = q.sum(2, keepdim=True)
    p = 1e-4 + (0.5 - 1e-4) * torch.rand(m, n, 1, generator=g, dtype=torch.float64, device=g.device)
    q *= torch.where(rs > 0, (1.0 - p) / torch.where(rs > 0, rs, 1.0), 0.0)
    a = torch.eye(n, dtype=torch.float64, device=g.device) - q
    return a, a.sum(2)


def _solve_inputs(case, seed, dev):
    """A packed batch of solves on `dev`: (n, offA, offv, A, b)."""
    n = _orders(case)
    g = torch.Generator(device=dev).manual_seed(seed)
    offA, offv = wl.offsets(n, True), wl.offsets(n, False)
    A = torch.empty(int((n.astype(np.int64) ** 2).sum()), dtype=torch.float64, device=dev)
    b = torch.empty(int(n.sum()), dtype=torch.float64, device=dev)
    make = _level_matrices if case["do"] == "levels" else _ion_matrices
    for k, part in _groups(n):
        a, v = make(g, part.size, k)
        A[_at(offA, part, k * k, dev)] = a.reshape(part.size, -1)
        b[_at(offv, part, k, dev)] = v
    return n, offA, offv, A, b


def _inverse_inputs(case, seed, dev):
    """A packed batch of macro-atom matrices on `dev`: (n, offA, offv, N, R)."""
    n = _orders(case)
    g = torch.Generator(device=dev).manual_seed(seed)
    offA, offv = wl.offsets(n, True), wl.offsets(n, False)
    A = torch.empty(int((n.astype(np.int64) ** 2).sum()), dtype=torch.float64, device=dev)
    R = torch.empty(int(n.sum()), dtype=torch.float64, device=dev)
    for k, part in _groups(n):
        a, r = _macro_matrices(g, part.size, k, case.get("density", 0.25))
        A[_at(offA, part, k * k, dev)] = a.reshape(part.size, -1)
        R[_at(offv, part, k, dev)] = r
    return n, offA, offv, A, R


def _one_input(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "solve":
        return wl.ion_matrix(rng, case["n"])
    return wl.macro_matrix(rng, case["n"]), None


def _lock_inputs(case, seed):
    nc = case["cells"]
    tab = wl.ion_table(ZS)
    rates = wl.ion_rates(tab, nc, seed=seed)
    rng = np.random.default_rng([seed, 1])
    nh = np.exp(rng.uniform(np.log(1e6), np.log(1e12), nc))
    den = np.zeros((nc, tab.nions))
    den[:, tab.elem_first] = 1.0
    return tab, rates, nh[:, None] * ABUND[None, :], 0.1 * nh, den


def _totals(g, m, n):
    """Row running totals of m blocks B = N^-1 diag(R): rows of positive weights that sum to 1."""
    w = _lu(g, 1e-6, 1.0, m, n, n)
    return torch.cumsum(w / w.sum(2, keepdim=True), 2)


def prepare(case, seed):
    do, dev = case["do"], torch.device("cuda")
    s = {"case": case}
    if do == "one":
        s["a"], s["b"] = _one_input(case, seed)
        return s
    if do == "lockstep":
        s["tab"], s["rates"], s["dens"], s["ne"], s["den"] = _lock_inputs(case, seed)
        return s
    if do in ("ion", "levels"):
        n, offA, offv, s["A"], s["b"] = _solve_inputs(case, seed, dev)
        s["plan"] = engine.Plan(wl.Batch("solve", n, offA, np.empty(0), offv), engine.FP64)
        s["out"] = torch.zeros_like(s["b"])
        s["status"] = torch.empty(n.size, dtype=torch.int32, device=dev)
    elif do == "host":
        n, offA, offv, A, b = _solve_inputs(case, seed, dev)
        pin = lambda t: torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()
        s["batch"] = wl.Batch("solve", n, offA, pin(A), offv, pin(b))
        s["x"] = torch.empty(b.shape, dtype=b.dtype, pin_memory=True).numpy()
    elif do in ("inverse", "matom"):
        n, offA, offv, s["A"], s["R"] = _inverse_inputs(case, seed, dev)
        s["out"] = torch.empty_like(s["A"])
        s["status"] = torch.empty(n.size, dtype=torch.int32, device=dev)
        s["n"], s["offA"], s["offv"] = n, offA, offv
        if do == "inverse":
            s["plan"] = engine.Plan(wl.Batch("invert", n, offA, np.empty(0)), MODES[case["mode"]])
        else:
            s["C"] = torch.empty_like(s["A"])
    else:
        n = _orders(case)
        g = torch.Generator(device=dev).manual_seed(seed)
        s["n"], s["offA"] = n, wl.offsets(n, True)
        s["C"] = torch.empty(int((n.astype(np.int64) ** 2).sum()), dtype=torch.float64, device=dev)
        for k, part in _groups(n):
            s["C"][_at(s["offA"], part, k * k, dev)] = _totals(g, part.size, k).reshape(part.size, -1)
        nq = case["nq"]
        s["sys"] = torch.randint(0, n.size, (nq,), generator=g, dtype=torch.int32, device=dev)
        u = torch.rand(nq, generator=g, dtype=torch.float64, device=dev)
        s["level"] = (u * torch.from_numpy(n).to(dev)[s["sys"].long()]).to(torch.int32)
        s["z"] = torch.rand(nq, generator=g, dtype=torch.float64, device=dev)
        s["target"] = torch.empty(nq, dtype=torch.int32, device=dev)
    return s


# --------------------------------------------------------------------- runs --
def _call(rc, what):
    if rc:
        raise engine.EngineError(f"{what} failed with {rc}: {engine.last_error()}")


def _p(t):
    return ctypes.c_void_p(t.data_ptr() if isinstance(t, torch.Tensor) else t.ctypes.data)


def run(s):
    case = s["case"]
    do = case["do"]
    if do == "one":
        if case["kind"] == "solve":
            code, x = engine.solve_matrix(s["a"], s["b"])
        else:
            code, x = engine.invert_matrix(s["a"])
        return {"x": x, "status": code}
    if do in ("ion", "levels"):
        s["plan"].execute(s["A"], s["out"], s["status"], b=s["b"])
        return {"x": s["out"], "status": s["status"]}
    if do == "host":
        x, status = engine.solve_batched(s["batch"], engine.FP64, x=s["x"])
        return {"x": x, "status": status}
    if do == "inverse":
        s["plan"].execute(s["A"], s["out"], s["status"])
        return {"x": s["out"], "status": s["status"]}
    if do == "matom":
        engine.set_precision(MODES[case["mode"]])
        _call(engine.load().matom_matrices_batched(s["n"].size, _p(s["n"]), _p(s["offA"]), _p(s["offv"]), _p(s["A"]),
                                                   _p(s["R"]), _p(s["out"]), _p(s["C"]), _p(s["status"])),
              "matom_matrices_batched")
        return {"B": s["out"], "C": s["C"], "status": s["status"]}
    if do == "draws":
        _call(engine.load().matom_sample_batched(case["nq"], s["n"].size, _p(s["n"]), _p(s["offA"]), _p(s["C"]),
                                                 _p(s["sys"]), _p(s["level"]), _p(s["z"]), _p(s["target"])),
              "matom_sample_batched")
        return {"target": s["target"]}
    engine.set_precision(engine.FP64)
    ne, den = s["ne"].copy(), s["den"].copy()
    status, iters = engine.ion_populations_lockstep_rates(s["tab"], s["rates"], 0, s["dens"], ne, den)
    return {"ne": ne, "den": den, "status": status, "iters": iters}


def work(case):
    """Inputs read once, outputs written once; LAPACK's operation counts."""
    do = case["do"]
    if do == "lockstep":
        n = np.tile(np.array(ZS) + 1, case["cells"]).astype(np.float64)   # one round of solves
        ions = float(np.sum(np.array(ZS) + 1))
        return {"bytes": case["cells"] * 8.0 * (12 * ions), "flops": float(np.sum(2 / 3 * n ** 3 + 2 * n ** 2))}
    n = _orders(case).astype(np.float64)
    if do in ("ion", "levels", "host") or (do == "one" and case["kind"] == "solve"):
        return {"bytes": float(np.sum(8 * (n ** 2 + 2 * n) + 4)), "flops": float(np.sum(2 / 3 * n ** 3 + 2 * n ** 2))}
    if do in ("one", "inverse"):
        return {"bytes": float(np.sum(16 * n ** 2 + 4)), "flops": float(np.sum(2 * n ** 3))}
    if do == "matom":
        return {"bytes": float(np.sum(24 * n ** 2 + 8 * n + 4)), "flops": float(np.sum(2 * n ** 3 + 2 * n ** 2))}
    # a draw walks half a row on average
    return {"bytes": case["nq"] * (20.0 + 4.0 * float(n.mean())), "flops": case["nq"] * 0.5 * float(n.mean())}


# -------------------------------------------------------------------- exact --
def _factor(a, b):
    """Batched LU with partial pivoting, in place, b's rows swapped along; returns the pivots."""
    m, n = b.shape
    at = torch.arange(m, device=a.device)
    for j in range(n):
        p = j + torch.argmax(a[:, j:, j].abs(), 1)
        for t in (a, b):
            r, q = t[at, p].clone(), t[:, j].clone()
            t[at, p] = q
            t[:, j] = r
        a[:, j + 1:, j] *= (1.0 / a[:, j, j])[:, None]
        prod = a[:, j + 1:, j, None] * a[:, j, None, j + 1:]
        a[:, j + 1:, j + 1:] -= prod
    return a.diagonal(0, 1, 2)


def _lu_solve(a, b):
    """LU with partial pivoting and row-oriented substitution, every product and difference rounded
    by itself, in the order of a textbook (and GSL's) solve: systems this ill-conditioned have no
    other value that two correct programs would share."""
    a, b = a.clone(), b.clone()
    _factor(a, b)
    n = b.shape[1]
    for j in range(n):
        prod = a[:, j + 1:, j] * b[:, j, None]
        b[:, j + 1:] -= prod
    x = torch.empty_like(b)
    for i in range(n - 1, -1, -1):
        u = b[:, i].clone()
        for k in range(i + 1, n):
            prod = a[:, i, k] * x[:, k]
            u -= prod
        x[:, i] = u / a[:, i, i]
    return x


def _lock_blocks(tab, rates, cells, ne, nh1, nh2):
    """The element systems of the listed cells (populate_ion_rate_matrix, matrix_ion.c:444-659)."""
    out = []
    z_of = np.repeat(tab.elem_z, tab.elem_n)
    cx = [[] for _ in range(tab.nions)]
    for m in range(tab.ncx):
        if z_of[tab.cx_nion2[m]] == 1:
            cx[tab.cx_nion1[m]].append(m)
    inn = [[] for _ in range(tab.nions)]
    for m in range(tab.n_inner):
        if tab.inner_yield[m] >= 0:
            inn[tab.inner_nion[m]].append(m)
    r = {k: getattr(rates, k)[cells] for k in ("pi", "rr", "di", "qr", "dr", "cxr", "cxi", "inner")}
    for e in range(tab.nelem):
        f, n = int(tab.elem_first[e]), int(tab.elem_n[e])
        a = np.zeros((len(cells), n, n))
        for c in range(n):
            i = f + c
            top = tab.ion_istate[i] == tab.elem_istate_max[e]

            def move(rate, d):
                a[:, c, c] -= rate
                if d is not None:
                    a[:, c + d, c] += rate
            if not top:
                move(r["pi"][:, i], 1)
                if tab.ion_di[i] > 0:
                    move(ne * r["di"][:, i], 1)
            if c:
                move(ne * (r["rr"][:, i] + ne * r["qr"][:, i]), -1)
                if tab.ion_dr[i] > 0:
                    a[:, c, c] -= ne * r["dr"][:, i]
                if tab.ion_dr[i - 1] > 0:
                    a[:, c - 1, c] += ne * r["dr"][:, i]
            if tab.ncx and z_of[i] != 1:
                move(r["cxr"][:, i] * nh1, -1 if c else None)
            for m in cx[i]:
                move(r["cxi"][:, m] * nh2, 1)
            nel = min(int(z_of[i] - tab.ion_istate[i] + 1), 11)
            for m in inn[i]:
                move(r["inner"][:, m], None)
                for d in range(1, nel):
                    a[:, c + d, c] += r["inner"][:, m] * tab.yield_prob[tab.inner_yield[m]][d - 1]
        a[:, 0, :] = 1.0
        b = np.zeros((len(cells), n))
        b[:, 0] = 1.0
        out.append((a, b))
    return out


def _lock_exact(tab, rates, dens, ne, den):
    """The n_e iteration of matrix_ion_populations (matrix_ion.c:219-382), all cells at once."""
    nc = ne.size
    ne, den, cur, x = ne.copy(), den.copy(), den.copy(), ne.copy()
    status, iters = np.full(nc, -2, np.int32), np.zeros(nc, np.int32)
    elem = np.repeat(np.arange(tab.nelem), tab.elem_n)
    live = np.arange(nc)
    for it in range(200):
        if not live.size:
            break
        nh1, nh2 = (cur[live, k] * dens[live, 0] for k in (0, 1))
        new = np.concatenate([_lu_solve(torch.from_numpy(a), torch.from_numpy(b)).numpy()
                              for a, b in _lock_blocks(tab, rates, live, x[live], nh1, nh2)], 1)
        iters[live] = it + 1
        new = np.where(new < 1e-20, 1e-20, new)
        xn = np.zeros(live.size)
        for i in range(tab.nions):
            xn = xn + new[:, i] * (int(tab.ion_istate[i]) - 1) * dens[live, elem[i]]
        xn = np.maximum(xn, 1e-20)
        cur[live] = new
        done = (np.abs((x[live] - xn) / xn) < 0.03) | (xn < 1e-6)
        d = live[done]
        status[d], ne[d], den[d] = 0, xn[done], new[done]
        x[live] = (xn + x[live]) / 2.0
        live = live[~done]
    return {"ne": ne, "den": den, "status": None, "iters": None}


def exact(case, seed):
    do, dev = case["do"], torch.device("cuda")
    if do == "one":
        a, b = _one_input(case, seed)
        if b is None:
            return {"x": np.linalg.inv(a), "status": None}
        return {"x": _lu_solve(torch.from_numpy(a[None]), torch.from_numpy(b[None]))[0], "status": None}
    if do in ("ion", "levels", "host"):
        n, offA, offv, A, b = _solve_inputs(case, seed, dev)
        x = torch.empty_like(b)
        for k, part in _groups(n, 1 << 26):
            a = A[_at(offA, part, k * k, dev)].reshape(-1, k, k)
            v = b[_at(offv, part, k, dev)]
            x[_at(offv, part, k, dev)] = torch.linalg.solve(a, v) if do == "levels" else _lu_solve(a, v)
        return {"x": x.cpu().numpy() if do == "host" else x, "status": None}
    if do in ("inverse", "matom"):
        n, offA, offv, A, R = _inverse_inputs(case, seed, dev)
        B, C = torch.empty_like(A), torch.empty_like(A) if do == "matom" else None
        for k, part in _groups(n, 1 << 24):
            at = _at(offA, part, k * k, dev)
            x = torch.linalg.inv(A[at].reshape(-1, k, k))
            if do == "matom":
                x = x * R[_at(offv, part, k, dev)][:, None, :]
                C[at] = torch.cumsum(x, 2).reshape(part.size, -1)
            B[at] = x.reshape(part.size, -1)
        return {"x": B, "status": None} if do == "inverse" else {"B": B, "C": C, "status": None}
    if do == "draws":
        return None
    return _lock_exact(*_lock_inputs(case, seed))
