"""Destroying a portfolio waits for launches that still read it, also beside a
stream capture of its own thread or of another, and leaves the capture as it is
(a wait for the whole device is refused there and ends the capture)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _portfolio(gpu, seed, scale=1.0, n=200):
    from riskgpu import synth
    rng = np.random.default_rng(seed)
    mu, sigma, _, _ = synth.factor_sigma(rng, n, 3, 0.005)
    return gpu.Portfolio(mu, scale * sigma, rng.dirichlet(np.ones(n)))


@pytest.mark.parametrize("precision", ["PREC_FP32", "PREC_BF16X3"])
def test_destroyed_beside_a_capture(gpu, precision):
    import torch
    q = gpu.make_query(4_000_000, 5, x=0.05, k=20, horizon=5, port_threshold=-0.01,
                       precision=getattr(gpu, precision))
    port = _portfolio(gpu, 1)
    want = port.simulate(q)
    counts = torch.zeros(2, dtype=torch.int64, device="cuda")
    mine, captured = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    port.launch_counts(q, counts.data_ptr(), mine.cuda_stream)
    with torch.cuda.stream(captured):
        g = torch.cuda.CUDAGraph()
        g.capture_begin(capture_error_mode="relaxed")
        x.add_(1.0)
        port.close()
        try:
            g.capture_end()
        except RuntimeError:  # a refused call may end the capture: not what is tested
            pass
    others = [_portfolio(gpu, 2 + i, 9.0) for i in range(6)]
    torch.cuda.synchronize()
    assert counts.tolist() == [want["crash_count"], want["breach_count"]]
    for p in others:
        p.close()


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("other_thread", [False, True])
def test_a_capture_survives_a_destruction(gpu, mode, other_thread):
    import torch
    port = _portfolio(gpu, 1)
    q = gpu.make_query(2_000_000, 5, x=0.05, k=20, horizon=5)
    counts = torch.zeros(2, dtype=torch.int64, device="cuda")
    mine, captured = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    port.launch_counts(q, counts.data_ptr(), mine.cuda_stream)
    done.record(mine)
    with torch.cuda.stream(captured):
        g = torch.cuda.CUDAGraph()
        g.capture_begin(capture_error_mode=mode)
        x.add_(1.0)
        if other_thread:
            t = threading.Thread(target=port.close)
            t.start()
            t.join()
        else:
            port.close()
        g.capture_end()
    assert done.query()  # the destruction has waited for the launch
    g.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 8


def test_batches_are_created_while_portfolios_come_and_go(gpu):
    """A batch's graph is captured at its creation."""
    stop, errors = threading.Event(), []
    item = _portfolio(gpu, 3, n=40)
    q = gpu.make_query(2000, 5, x=0.05, k=5, precision=gpu.PREC_BF16X3)
    want = item.simulate(q)["crash_count"]

    def churn():
        try:
            while not stop.is_set():
                _portfolio(gpu, 4, n=9).close()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=churn) for _ in range(3)]
    for t in threads:
        t.start()
    try:
        for _ in range(150):
            batch = gpu.Batch([(item, q)])
            assert batch.run()[0]["crash_count"] == want
            batch.close()
    finally:
        stop.set()
        for t in threads:
            t.join()
    assert not errors
