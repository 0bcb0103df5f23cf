"""The tensor-core kernel's path tiles: S and w.R of a path do not depend on the
tile width (16 to 128 paths, chosen from the path count), on the form (merged or
split) or on the block table, and no path is left out or written twice.  Exact:
an accumulator is the same sum whatever the other columns of its MMA are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 15, 17, 100, 2431, 2433, 4865, 5000, 7297, 9729, 14593, 19457, 20011)


@pytest.mark.parametrize("n,horizon,aggregated", [(65, 2, False), (127, 5, False), (128, 1, False), (333, 5, False),
                                                  (487, 10, True), (511, 1, False), (512, 3, False), (600, 2, False),
                                                  (600, 10, True), (639, 1, False), (640, 2, False)])
def test_paths_do_not_depend_on_the_tile(gpu, monkeypatch, n, horizon, aggregated):
    import torch
    from riskgpu import synth
    rng = np.random.default_rng(n)
    mu, sigma, _, _ = synth.factor_sigma(rng, n, 3, 0.005)
    port = gpu.Portfolio(mu, sigma, rng.dirichlet(np.ones(n)))
    x, k = 0.028 * horizon ** 0.5, max(1, n // 10)

    def run(m, offset=0):
        S = torch.full((m + 160,), -7, dtype=torch.int32, device="cuda")
        W = torch.full((m + 160,), -7.0, dtype=torch.float32, device="cuda")
        q = gpu.make_query(m, 9, x=x, k=k, horizon=horizon, port_threshold=-0.01, precision=gpu.PREC_BF16X3,
                           path_offset=offset, d_s_values=S.data_ptr(), d_port_values=W.data_ptr(),
                           draw_mode=gpu.DRAWS_AGGREGATED if aggregated else gpu.DRAWS_DAILY)
        r = port.simulate(q)
        S, W = S.cpu().numpy(), W.cpu().numpy()
        assert (S[m:] == -7).all() and (W[m:] == -7).all()
        assert r["crash_count"] == int((S[:m] >= k).sum())
        return S[:m], W[:m]

    # enough paths for the widest tiles and the block table
    S, W = run(200_000)
    for m in SIZES:
        s, w = run(m)
        assert np.array_equal(s, S[:m]) and np.array_equal(w, W[:m]), m
    for form in ("merged", "split"):
        monkeypatch.setenv("RG_TC_KERNEL", form)
        for m in (5000, 200_000):
            s, w = run(m)
            assert np.array_equal(s, S[:m]) and np.array_equal(w, W[:m]), (form, m)
    # a range that crosses a change of the path index's high word draws without the table
    monkeypatch.delenv("RG_TC_KERNEL")
    s, w = run(150_000, 2 ** 32 - 75_000)
    lo, wlo = run(75_000, 2 ** 32 - 75_000)
    hi, whi = run(75_000, 2 ** 32)
    assert np.array_equal(s, np.concatenate([lo, hi])) and np.array_equal(w, np.concatenate([wlo, whi]))


def test_batch_forms_agree(gpu):
    """Batches whose totals call for the split and for the merged form, items
    in an order that is not that of their tile cost: counts equal those of the
    same queries alone."""
    from riskgpu import synth
    rng = np.random.default_rng(4)
    for horizons in ((1, 2), (8, 16)):
        items = []
        for i in range(9):
            n = int(rng.integers(10, 601))
            h = int(rng.integers(horizons[0], horizons[1] + 1))
            mu, sigma, _, _ = synth.factor_sigma(rng, n, 3, 0.005)
            q = gpu.make_query(int(rng.integers(1, 30_000)), 100 + i, x=0.02 * h ** 0.5, k=max(1, n // 10), horizon=h,
                               port_threshold=-0.005, precision=gpu.PREC_BF16X3 if i % 2 else gpu.PREC_FP16X3,
                               path_offset=2 ** 32 - 100 if i == 4 else 0)
            items.append((gpu.Portfolio(mu, sigma, rng.dirichlet(np.ones(n))), q))
        batch = gpu.Batch(items)
        for _ in range(2):
            for (port, q), r in zip(items, batch.run()):
                alone = port.simulate(q)
                assert (r["crash_count"], r["breach_count"]) == (alone["crash_count"], alone["breach_count"])
