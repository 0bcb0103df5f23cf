"""The N <= 64 kernel's CTA shapes: S and w.R of every path do not depend on how
many threads a launch has (exact), and no path is left out or written twice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# sizes around full rounds of 152 CTAs of 768, 896 and 1024 threads, and below one warp an SM
SIZES = (1, 31, 33, 4863, 4865, 116735, 116737, 136193, 155649, 233473, 311297)


@pytest.mark.parametrize("n,horizon,var", [(9, 1, False), (12, 2, True), (20, 1, True), (33, 1, False), (50, 1, False),
                                           (50, 3, False), (64, 1, True)])
def test_results_do_not_depend_on_the_launch_shape(gpu, n, horizon, var):
    import torch
    from riskgpu import synth
    rng = np.random.default_rng(n)
    mu, sigma, _, _ = synth.one_factor_sigma(rng, n)
    port = gpu.Portfolio(mu, sigma, rng.dirichlet(np.ones(n)))
    k, x, thr = max(1, n // 4), 0.02, -0.01
    most = max(SIZES)

    def run(offset, m, level):
        S = torch.full((m + 64,), -7, dtype=torch.int32, device="cuda")
        W = torch.full((m + 64,), -7.0, dtype=torch.float32, device="cuda")
        q = gpu.make_query(m, 5, x=x, k=k, horizon=horizon, port_threshold=thr, path_offset=offset, var_level=level,
                           d_s_values=S.data_ptr(), d_port_values=W.data_ptr())
        r = port.simulate(q)
        S, W = S.cpu().numpy(), W.cpu().numpy()
        assert (S[m:] == -7).all() and (W[m:] == -7).all()
        assert r["crash_count"] == int((S[:m] >= k).sum())
        assert r["breach_count"] == int((W[:m] < np.float32(thr)).sum())
        return S[:m], W[:m], r

    parts = [run(o, min(10007, most - o), 0.0) for o in range(0, most, 10007)]
    S, W = (np.concatenate([p[i] for p in parts]) for i in (0, 1))
    for m in SIZES:
        s, w, r = run(0, m, 0.99 if var else 0.0)
        assert np.array_equal(s, S[:m]) and np.array_equal(w, W[:m])
        if var:
            T = gpu.tail_count(m, 0.99)
            assert r["var"] == -float(np.sort(w)[T - 1])


@pytest.mark.parametrize("n", [3, 20, 50])
@pytest.mark.parametrize("offset", [0, 1, 4095, 2 ** 33 + 77])
def test_xorwow_paths_do_not_depend_on_the_launch_shape(gpu, n, offset):
    """The reference's stream: each path's state is reached from the CTA's
    first one by skips of 1, 2, 4, ... and by steps of the CTA's width; S of a
    path is the same whatever range it is part of (both widths, runs that end
    inside a CTA, and a range of one path, which is cuRAND's own
    initialisation)."""
    import torch
    from riskgpu import synth
    rng = np.random.default_rng(n)
    mu, sigma, _, _ = synth.one_factor_sigma(rng, n)
    port = gpu.Portfolio(mu, sigma, rng.dirichlet(np.ones(n)))

    def run(first, m):
        S = torch.full((m + 8,), -7, dtype=torch.int32, device="cuda")
        W = torch.full((m + 8,), -7.0, dtype=torch.float32, device="cuda")
        port.simulate(gpu.make_query(m, 67, x=0.02, k=1, rng=gpu.RNG_XORWOW_REF, path_offset=offset + first,
                                     d_s_values=S.data_ptr(), d_port_values=W.data_ptr()))
        S, W = S.cpu().numpy(), W.cpu().numpy()
        assert (S[m:] == -7).all()
        return S[:m], W[:m]

    S, W = run(0, 311_500)
    for first, m in [(0, 77_825), (1000, 155_000), (37, 64), (63, 65), (5, 9_729), (77_824, 200)]:
        s, w = run(first, m)
        assert np.array_equal(s, S[first:first + m]) and np.array_equal(w, W[first:first + m])
    for p in (0, 1, 2, 3, 62, 63, 64, 255, 256, 257, 1023, 77_823, 77_824, 311_499):
        s, w = run(p, 1)
        assert s[0] == S[p] and w[0] == W[p]
