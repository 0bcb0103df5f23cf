"""Query scratch and portfolio memory from the engine's shared pool: calls on
several host threads, with portfolios created and destroyed between them, give
the same results as the same calls one after the other."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(gpu, synth, i):
    n = (5, 33, 50, 130, 200)[i % 5]
    rng = np.random.default_rng(900 + i)
    mu, sigma, _, _ = synth.factor_sigma(rng, n, 3, 0.005)
    w = rng.dirichlet(np.ones(n))
    q = gpu.make_query(20_000 + 777 * i, 31 + i, x=0.03, k=max(1, n // 10), horizon=1 + i % 3, port_threshold=-0.01,
                       precision=gpu.PREC_BF16X3 if n > 64 and i % 2 else gpu.PREC_AUTO,
                       var_level=0.99 if i % 3 else 0.0)
    return mu, sigma, w, q


def _run(gpu, mu, sigma, w, q, one_shot):
    if one_shot:
        r = gpu.run(mu, sigma, w, q)
    else:
        port = gpu.Portfolio(mu, sigma, w)
        r = port.simulate(q)
        port.close()
    return {k: v for k, v in r.items() if k != "ms_device" and v == v}


def test_concurrent_calls_equal_serial_ones(gpu):
    from riskgpu import synth
    cases = [_case(gpu, synth, i) for i in range(24)]
    want = [_run(gpu, *c, one_shot=False) for c in cases]
    got, errors = {}, []

    def work(t):
        try:
            for i in range(t, 24, 8):
                for one_shot in (True, False):
                    got[i, one_shot] = _run(gpu, *cases[i], one_shot=one_shot)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for i in range(24):
        # CVaR sums the candidates in the order they were appended
        for key in want[i]:
            for one_shot in (True, False):
                if key == "cvar":
                    assert abs(got[i, one_shot][key] - want[i][key]) <= 1e-12
                else:
                    assert got[i, one_shot][key] == want[i][key], (i, key)
