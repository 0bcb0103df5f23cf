"""The pipelined FP32 kernel's generator takes two days a turn: odd and even day
counts, the padding quads and a path range that crosses a change of the index's
high word, against the phase-serial kernel, which draws day by day.  The two add
the same terms in different orders: w.R within 2e-5, S equal but for paths with
a return within FP32 rounding of the threshold (at most one in a thousand)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 2 ** 32 - 1000])
@pytest.mark.parametrize("n,horizon", [(65, 1), (65, 2), (67, 3), (96, 4), (129, 5), (130, 20), (257, 7)])
def test_days_agree_with_the_serial_form(gpu, monkeypatch, n, horizon, offset):
    import torch
    from riskgpu import synth
    rng = np.random.default_rng(n + horizon)
    mu, sigma, _, _ = synth.factor_sigma(rng, n, 3, 0.005)
    port = gpu.Portfolio(mu, sigma, rng.dirichlet(np.ones(n)))
    m, x, k = 20_011, 0.028 * horizon ** 0.5, max(1, n // 10)
    out = []
    for form in ("tiled", "tiled-serial"):
        monkeypatch.setenv("RG_PLAIN_KERNEL", form)
        S = torch.full((m + 64,), -7, dtype=torch.int32, device="cuda")
        W = torch.full((m + 64,), -7.0, dtype=torch.float32, device="cuda")
        r = port.simulate(gpu.make_query(m, 11, x=x, k=k, horizon=horizon, port_threshold=-0.01, path_offset=offset,
                                         d_s_values=S.data_ptr(), d_port_values=W.data_ptr()))
        S, W = S.cpu().numpy(), W.cpu().numpy()
        assert (S[m:] == -7).all() and (W[m:] == -7).all()
        assert r["crash_count"] == int((S[:m] >= k).sum())
        out.append((S[:m], W[:m]))
    assert np.abs(out[0][1] - out[1][1]).max() < 2e-5
    assert (out[0][0] != out[1][0]).mean() <= 1e-3
