"""First calls: a plan, or a table of coefficients, that the same call uploads is used
at once, on streams that do not wait for the default one.  Every layout is new to
its thread, so every call builds what it uses."""
import threading

import numpy as np
import pytest

from oracle import oracle
from python_b200 import workloads as wl
from helpers import same_values


@pytest.mark.gpu
def test_first_drop_in_calls_of_new_threads(engine):
    rng = np.random.default_rng(9)
    sys = {n: (rng.standard_normal((n, n)) + np.eye(n), rng.standard_normal(n)) for n in range(1, 41)}
    ref = {n: oracle.solve(wl.from_matrices("solve", [a], [b]), "port")[0] for n, (a, b) in sys.items()}
    errors = []

    def work():
        try:
            for n, (a, b) in sys.items():
                code, x = engine.solve_matrix(a, b)
                assert code in (0, 2, 3) and same_values(x, ref[n]).all(), n
        except Exception as e:                       # noqa: BLE001 - reported below
            errors.append(e)

    for _ in range(3):
        threads = [threading.Thread(target=work) for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not errors, errors[0]


@pytest.mark.gpu
def test_plans_executed_at_once_on_a_non_blocking_stream(engine):
    import torch
    rng = np.random.default_rng(10)
    dev, s = torch.device("cuda", 0), torch.cuda.Stream()
    for k in range(30):
        ns = rng.integers(2, 50, 40)
        b = wl.from_matrices("solve", [rng.standard_normal((n, n)) for n in ns], [rng.standard_normal(n) for n in ns])
        A, rhs = torch.from_numpy(b.A).to(dev), torch.from_numpy(b.b).to(dev)
        x, st = torch.zeros_like(rhs), torch.full((b.nsys,), -9, dtype=torch.int32, device=dev)
        xr, sr = oracle.solve(b, "port")
        torch.cuda.synchronize()
        plan = engine.Plan(b, engine.FP64)
        plan.execute(A, x, st, b=rhs, stream=s)
        s.synchronize()
        assert np.array_equal(st.cpu().numpy(), sr) and same_values(x.cpu().numpy(), xr).all(), k
        plan.close()
