"""Sample moments of many columns, where the covariance takes one row segment
whatever the number of rows and its tiles are written at once.  Bounds as in
the other moments tests: 2 eps of the mean absolute value; (T + 4) eps of the
sum of absolute products."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,n", [(300, 1537), (129, 1600), (2, 1700)])
def test_moments_of_many_columns(gpu, T, n):
    X = np.random.default_rng(T + n).normal(3e-4, 0.01, size=(T, n))
    mu, sigma = gpu.moments(X)
    eps = 2.0 ** -52
    D = X - mu
    S_abs = np.abs(D).T @ np.abs(D) / (T - 1) + eps * np.abs(X).max() ** 2
    for j in range(0, n, 97):
        assert abs(mu[j] - math.fsum(X[:, j]) / T) <= 2 * eps * np.mean(np.abs(X[:, j]))
    for i in list(range(0, n, 211)) + [n - 1]:
        for j in list(range(0, n, 173)) + [n - 1]:
            ref = math.fsum(D[:, i] * D[:, j]) / (T - 1)
            assert abs(sigma[i, j] - ref) <= (T + 4) * eps * S_abs[i, j]
    assert np.array_equal(sigma, sigma.T)
    assert np.max(np.abs(sigma - D.T @ D / (T - 1))) <= 2 * (T + 4) * eps * S_abs.max()
