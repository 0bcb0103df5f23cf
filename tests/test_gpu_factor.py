"""FP64 factorisation and sample moments at the edges of their forms: the one-CTA form's column
counts (16, 32, 48, 64 and their neighbours), the blocked form's 32-column
blocks and 16 x 16 update tiles, and a failing pivot in each place.

Tolerances: |L L^T - Sigma| <= N eps max|Sigma| (the backward error bound of a
Cholesky factorisation is about (N + 1) eps/2 |L||L^T|, and |L||L^T| <=
max|Sigma|), eps = 2^-52; L within 1e-12 of the oracle as in the other
factorisation tests; the moments within 1e-12 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = (1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 80, 81, 95, 96, 97, 112, 113, 128, 129, 161, 600)


@pytest.mark.parametrize("n", EDGES)
def test_factor_edges(gpu, oracle, n):
    from riskgpu import synth
    rng = np.random.default_rng(7000 + n)
    mu, sigma, _, _ = synth.factor_sigma(rng, n, 3, 0.005)
    w = rng.dirichlet(np.ones(n))
    port = gpu.Portfolio(mu, sigma, w)
    L = port.factor()
    assert np.array_equal(L, np.tril(L))
    assert np.max(np.abs(L @ L.T - sigma)) <= n * 2.0 ** -52 * np.max(np.abs(sigma))
    L_ref, info = oracle.cholesky_lower(sigma)
    assert info == 0 and np.max(np.abs(L - L_ref)) <= 1e-12
    inf = port.info()
    assert abs(inf["wsw"] - w @ sigma @ w) <= 1e-12 * (w @ sigma @ w)
    assert abs(inf["wmu"] - w @ mu) <= 1e-12 * abs(w) @ abs(mu)


@pytest.mark.parametrize("n,bad", [(1, 0), (9, 0), (9, 1), (9, 8), (20, 7), (33, 32), (64, 5), (64, 63), (100, 0),
                                   (100, 31), (100, 32), (100, 33), (100, 64), (100, 99)])
def test_first_failing_pivot(gpu, n, bad):
    """The first pivot that is not positive is the one reported; a later one
    is not."""
    a = np.eye(n) * 2.0
    a[bad, bad] = -1.0
    if bad + 3 < n:
        a[bad + 3, bad + 3] = -1.0
    with pytest.raises(gpu.RiskGpuError) as e:
        gpu.Portfolio(np.zeros(n), a)
    assert e.value.status == gpu.RG_ERR_NOT_PD
    assert f"pivot {bad})" in str(e.value)


@pytest.mark.parametrize("n", [5, 50, 100])
@pytest.mark.parametrize("scale", [1e-304, 1e-290, 1e290])
def test_extreme_scales(gpu, n, scale):
    """Variances at the ends of FP64's range (outside the hardware reciprocal
    square root's): L within cond(Sigma) N eps of numpy's, relative to its
    largest entry (the forward error bound)."""
    rng = np.random.default_rng(n)
    B = rng.normal(size=(n, 2))
    unit = B @ B.T + np.diag(rng.uniform(1.0, 2.0, n))
    L = gpu.Portfolio(np.zeros(n), unit * scale).factor()
    ref = np.linalg.cholesky(unit) * np.sqrt(scale)
    assert np.max(np.abs(L - ref)) <= np.linalg.cond(unit) * n * 2.0 ** -52 * np.max(np.abs(ref))


@pytest.mark.parametrize("T,n", [(2, 31), (2, 32), (31, 33), (32, 1), (33, 32), (63, 5), (64, 64), (127, 65), (128, 2),
                                 (129, 97), (2049, 31), (4100, 3)])
def test_moments_edges(gpu, T, n):
    """Row segments and 32 x 32 tiles at their edges, against exactly rounded
    sums (math.fsum).  mu: 2 eps of the mean absolute value; Sigma: two
    roundings of the deviations and at most T of the sum, (T + 4) eps of the
    sum of absolute products."""
    import math
    X = np.random.default_rng(T * 131 + n).normal(3e-4, 0.01, size=(T, n))
    mu, sigma = gpu.moments(X)
    eps = 2.0 ** -52
    for j in range(n):
        assert abs(mu[j] - math.fsum(X[:, j]) / T) <= 2 * eps * np.mean(np.abs(X[:, j]))
    D = X - mu
    S_abs = np.abs(D).T @ np.abs(D) / (T - 1) + eps * np.abs(X).max() ** 2
    for i in range(0, n, max(1, n // 4)):
        for j in range(0, n, max(1, n // 5)):
            ref = math.fsum(D[:, i] * D[:, j]) / (T - 1)
            assert abs(sigma[i, j] - ref) <= (T + 4) * eps * S_abs[i, j]
    assert np.array_equal(sigma, sigma.T)


@pytest.mark.parametrize("T,n,at", [(2, 1, 1), (40, 33, 40 * 33 - 1), (70, 40, 0), (70, 40, 1234), (300, 65, 7777)])
def test_first_entry_not_finite(gpu, T, n, at):
    """The first entry (row by row) that is not finite is named, whichever
    kernel meets it first; the outputs are not written."""
    X = np.zeros((T, n))
    X.flat[at] = np.inf
    if at + 1 < T * n:
        X.flat[-1] = np.nan
    where = rf"returns\[{at // n}\]\[{at % n}\] is not finite"
    with pytest.raises(gpu.RiskGpuError, match=where) as e:
        gpu.moments(X)
    assert e.value.status == gpu.RG_ERR_INVALID
    with pytest.raises(gpu.RiskGpuError, match=where) as e:
        gpu.crash_frequency(X, 0.01, 1)
    assert e.value.status == gpu.RG_ERR_INVALID
