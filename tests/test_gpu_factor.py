"""FP64 factorisation at the edges of its forms: the one-CTA form's column
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
