"""The n_e iteration run wholly on the GPU (ion_populations_lockstep_rates) against
the driver that assembles through a callback and solves round by round: equal
statuses, round counts, n_e and populations, bit for bit, for tables on either
side of the kernel's size classes, one to four warps a cell, singular cells,
cells that never converge, no hydrogen element, and tables it does not take
(an element of more than 32 ions, mixed mode)."""
import numpy as np
import pytest

from python_b200 import workloads as wl

TABLES = {"H": (1,), "to16": (1, 2, 7, 15), "five": (1, 2, 6, 8, 26), "to28": (1, 27), "to32": (1, 2, 30, 31),
          "many": (1, 2, 6, 7, 8, 10, 12, 14, 16, 18, 20, 26, 28), "no hydrogen": (2, 6, 8), "above32": (1, 2, 40)}


def _inputs(zs, nc, seed):
    tab = wl.ion_table(zs, seed=seed)
    rates = wl.ion_rates(tab, nc, seed=seed + 1)
    rng = np.random.default_rng(seed + 2)
    nh = np.exp(rng.uniform(np.log(1e6), np.log(1e12), nc))
    dens = nh[:, None] * np.exp(rng.uniform(np.log(1e-5), 0.0, (nc, tab.nelem)))
    if nc > 4:
        dens[3] *= 1e-25                       # nearly empty: n_e below 1e-6
        for k in ("pi", "rr", "di", "qr", "dr", "cxr", "cxi", "inner"):
            getattr(rates, k)[1] = 0.0         # no rates: singular blocks
        rates.rr[2, :] = np.nan                # never converges
    den = np.zeros((nc, tab.nions))
    den[:, tab.elem_first] = 1.0
    return tab, rates, dens, 0.1 * nh, den


def _callback_driver(engine, tab, rates, h, dens, ne, den):
    def sub(cells):
        return wl.IonRates(*[np.ascontiguousarray(getattr(rates, k)[cells]) for k in
                             ("pi", "rr", "di", "qr", "dr", "cxr", "cxi", "inner")])

    def assemble(cells, nea, nh1, nh2, A, b):
        a2, b2 = engine.ion_rate_matrices(tab, sub(cells), nea, nh1, nh2)
        A[:] = a2
        b[:] = b2.ravel()
    return engine.ion_populations_lockstep(tab.elem_first, tab.elem_n, tab.ion_istate, h, dens, ne, den, assemble)


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(TABLES))
@pytest.mark.parametrize("nc", [1, 700])
def test_device_rounds_match_host_rounds(engine, name, nc):
    zs = TABLES[name]
    tab, rates, dens, ne0, den0 = _inputs(zs, nc, seed=100 + len(zs))
    h = 0 if zs[0] == 1 else -1
    for mode in (engine.FP64, engine.MIXED) if name == "five" else (engine.FP64,):
        engine.set_precision(mode)
        try:
            ne_a, den_a = ne0.copy(), den0.copy()
            st_a, it_a = _callback_driver(engine, tab, rates, h, dens, ne_a, den_a)
            ne_b, den_b = ne0.copy(), den0.copy()
            st_b, it_b = engine.ion_populations_lockstep_rates(tab, rates, h, dens, ne_b, den_b)
        finally:
            engine.set_precision(engine.FP64)
        assert np.array_equal(st_a, st_b) and np.array_equal(it_a, it_b)
        assert np.array_equal(ne_a, ne_b, equal_nan=True) and np.array_equal(den_a, den_b, equal_nan=True)
        if nc > 4:
            assert st_b[1] == -1 and st_b[2] == -2 and it_b[2] == 200 and (st_b == 0).sum() > nc // 2
