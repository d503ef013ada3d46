"""The n_e iteration on the GPU from several host threads at once, with tables
whose kernels are the same but ask different amounts of shared memory: every call
returns what it returns alone."""
import threading

import numpy as np
import pytest

from python_b200 import workloads as wl


def _inputs(zs, nc, seed):
    tab = wl.ion_table(zs, seed=seed)
    rates = wl.ion_rates(tab, nc, seed=seed + 1)
    rng = np.random.default_rng(seed + 2)
    nh = np.exp(rng.uniform(np.log(1e6), np.log(1e12), nc))
    dens = nh[:, None] * np.exp(rng.uniform(np.log(1e-5), 0.0, (nc, tab.nelem)))
    den = np.zeros((nc, tab.nions))
    den[:, tab.elem_first] = 1.0
    return tab, rates, dens, 0.1 * nh, den


def _call(engine, inp):
    tab, rates, dens, ne0, den0 = inp
    ne, den = ne0.copy(), den0.copy()
    h = 0 if tab.elem_z[0] == 1 else -1
    st, it = engine.ion_populations_lockstep_rates(tab, rates, h, dens, ne, den)
    return ne, den, st, it


@pytest.mark.gpu
@pytest.mark.parametrize("large,small", [((1, 2, 30, 31), (31,)),
                                         ((1, 2, 6, 7, 8, 10, 12, 14, 16, 18, 20, 22, 24, 25, 26), (24,))])
def test_tables_of_different_size_in_threads(engine, large, small):
    # one kernel instantiation per pair (largest elements 32 and 32 ions, 27 and 25):
    # four warps a cell and more than 48 KB on one side, one warp on the other
    big, little = _inputs(large, 2, 5), _inputs(small, 1, 6)
    want_big, want_little = _call(engine, big), _call(engine, little)
    stop, errors = threading.Event(), []

    def work(inp, want, calls):
        try:
            for _ in range(calls):
                got = _call(engine, inp)
                for g, w in zip(got, want):
                    assert np.array_equal(g, w, equal_nan=True)
                if stop.is_set():
                    break
        except Exception as e:                       # noqa: BLE001 - reported below
            errors.append(e)
        finally:
            stop.set()

    threads = [threading.Thread(target=work, args=(big, want_big, 1500))]
    threads += [threading.Thread(target=work, args=(little, want_little, 10 ** 9)) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
