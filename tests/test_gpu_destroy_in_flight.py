"""A portfolio destroyed while a launch on the caller's stream still reads it,
beside a stream capture (which forbids waiting for the device): the launch
counts what it would have counted, whatever is created afterwards."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _portfolio(gpu, seed, scale=1.0):
    from riskgpu import synth
    rng = np.random.default_rng(seed)
    mu, sigma, _, _ = synth.factor_sigma(rng, 200, 3, 0.005)
    return gpu.Portfolio(mu, scale * sigma, rng.dirichlet(np.ones(200)))


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
