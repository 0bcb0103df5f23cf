"""The split tensor form where its second MMA issuer owns no row tile (N <= 127:
one row tile), over many path tiles a CTA: the same S and w.R per path as the
merged form, and in batches of each tile width the same counts as each query
alone.  Exact: an accumulator is the same sum in both forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _portfolio(gpu, n):
    from riskgpu import synth
    rng = np.random.default_rng(300 + n)
    mu, sigma, _, _ = synth.factor_sigma(rng, n, 3, 0.005)
    return gpu.Portfolio(mu, sigma, rng.dirichlet(np.ones(n)))


def _query(gpu, n, m, horizon, **more):
    return gpu.make_query(m, 5 + n, x=0.028 * horizon ** 0.5, k=max(1, n // 10), horizon=horizon, port_threshold=-0.01,
                          draw_mode=gpu.DRAWS_AGGREGATED, **more)


@pytest.mark.parametrize("n", [1, 33, 64, 65, 127, 128, 640])
def test_split_equals_merged_over_many_tiles(gpu, monkeypatch, n):
    import torch
    port, m = _portfolio(gpu, n), 1_000_003
    got = []
    for form in ("merged", "split"):
        monkeypatch.setenv("RG_TC_KERNEL", form)
        S = torch.full((m,), -7, dtype=torch.int32, device="cuda")
        W = torch.full((m,), -7.0, dtype=torch.float32, device="cuda")
        r = port.simulate(_query(gpu, n, m, 4, precision=gpu.PREC_FP16X3, d_s_values=S.data_ptr(),
                                 d_port_values=W.data_ptr()))
        got.append((r["crash_count"], r["breach_count"], S, W))
    assert got[0][:2] == got[1][:2]
    assert torch.equal(got[0][2], got[1][2]) and torch.equal(got[0][3], got[1][3])


@pytest.mark.parametrize("largest", [64, 127, 600, 640])  # 128, 128, 96 and 64 paths a tile
def test_split_batches_of_small_items(gpu, monkeypatch, largest):
    sizes = [5, 20, 64, 64, 90, 127]
    items = [(_portfolio(gpu, n), _query(gpu, n, 300_001 + 1000 * i, 1 + i, precision=gpu.PREC_BF16X3))
             for i, n in enumerate([n for n in sizes if n <= largest] + [largest])]
    batch = gpu.Batch(items)
    got = [[(r["crash_count"], r["breach_count"]) for r in batch.run()] for _ in range(3)]
    monkeypatch.setenv("RG_TC_KERNEL", "merged")
    want = [port.simulate(q) for port, q in items]
    assert got == [[(r["crash_count"], r["breach_count"]) for r in want]] * 3
