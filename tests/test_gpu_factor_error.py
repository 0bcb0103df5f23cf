"""Error of the one-CTA factor (N <= 64) against extended precision: no larger
than that of a plain FP64 factorisation with each column's products summed on
their own, a square root and divisions.

Both errors are sums of many roundings, compared as root mean squares over 24
matrices a size.  The two differ in the order of their sums, which moves such a
mean by a few per cent: 10 % are allowed (the kernel's order, followed in numpy,
is 0.80 to 1.01 of the plain one).  Products subtracted one by one and quotients
through a rounded reciprocal are 1.12 to 1.33 of it up to 24 columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _matrix(n, rep):
    from riskgpu import synth
    rng = np.random.default_rng(1000 * n + rep)
    if rep % 3 == 0:
        return synth.one_factor_sigma(rng, n)[1]
    mu, sigma, B, idio = synth.factor_sigma(rng, n, min(n, 5), 0.005)
    if rep % 3 == 1:
        return sigma
    X = rng.normal(size=(n + 250, B.shape[1])) @ B.T + rng.normal(size=(n + 250, n)) * idio
    sigma = np.cov(X.T).reshape(n, n)
    return (sigma + sigma.T) / 2


def _exact(a):
    a = a.astype(LD)
    L = np.zeros_like(a)
    for j in range(len(a)):
        L[j, j] = np.sqrt(a[j, j] - (L[j, :j] ** 2).sum())
        L[j + 1:, j] = (a[j + 1:, j] - L[j + 1:, :j] @ L[j, :j]) / L[j, j]
    return L


def _fma(a, b, c):
    return (a.astype(LD) * LD(b) + c.astype(LD)).astype(np.float64)


def _tree(v):
    v = np.concatenate([v, np.zeros(64 - len(v))])
    while len(v) > 1:
        v = v[::2] + v[1::2]
    return v[0]


def _plain(a):
    n = len(a)
    L = np.tril(a).copy()
    for j in range(n):
        L[j, j] = np.sqrt(L[j, j] - _tree(L[j, :j] * L[j, :j]))
        even, odd = L[j + 1:, j].copy(), np.zeros(n - j - 1)
        for k in range(j):
            if k % 2 == 0:
                even = _fma(-L[j + 1:, k], L[j, k], even)
            else:
                odd = _fma(-L[j + 1:, k], L[j, k], odd)
        L[j + 1:, j] = (even + odd) / L[j, j]
    return L


def _rms(factor, n):
    total = 0.0
    for rep in range(24):
        a = _matrix(n, rep)
        E = _exact(a)
        total += float(((factor(a) - E) ** 2).sum() / (E ** 2).sum())
    return (total / 24) ** 0.5 * 2.0 ** 52


@pytest.mark.parametrize("n", [2, 5, 9, 16, 17, 20, 24, 32, 33, 48, 49, 64])
def test_error_of_the_factor(gpu, n):
    def factor(a):
        port = gpu.Portfolio(np.zeros(n), a)
        L = port.factor()
        port.close()
        return L

    assert _rms(factor, n) <= 1.1 * _rms(_plain, n)


@pytest.mark.parametrize("exponent", [-1000, -959, -958, -301, -2, -1, 0, 1, 2, 300, 959, 960, 1000])
def test_pivot_root(gpu, exponent):
    """One asset: L = sqrt(Sigma) within half an ulp and the error of the
    reciprocal root's two parts (2^-61 relative, 2^-8 ulp), over mantissas, both
    parities of the exponent and the exponents at which CUDA's own takes over."""
    rng = np.random.default_rng(abs(exponent))
    for m in np.concatenate([[1.0, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52], rng.uniform(1.0, 2.0, 30)]):
        d = float(np.ldexp(m, exponent))
        port = gpu.Portfolio(np.zeros(1), np.array([[d]]))
        got = port.factor()[0, 0]
        port.close()
        root = np.sqrt(LD(d))
        assert abs(LD(got) - root) <= 0.51 * np.spacing(float(root)), (m, exponent)
