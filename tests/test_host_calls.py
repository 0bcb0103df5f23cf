"""Host side of portfolio and query calls on the fake runtime: statuses, memory
and the order of runtime calls where memory is short, a call is refused or many
callers meet."""
import ctypes

import numpy as np
import pytest

import riskgpu
from host_engine import CAPTURE_REFUSED, fake, linked  # noqa: F401


def _create(n=8, bad=None):
    """(status, handle, message) of rg_portfolio_create on an identity Sigma."""
    mu, sigma = np.zeros(n), np.eye(n)
    if bad is not None:
        sigma[bad, 0] = np.nan
    h = ctypes.c_void_p()
    st = riskgpu.lib().rg_portfolio_create(n, mu.ctypes.data, sigma.ctypes.data, n, None, 0, ctypes.byref(h))
    return st, h.value, riskgpu.lib().rg_last_error().decode()


def test_a_refused_admission_stays_refused(fake, monkeypatch):
    """Memory that turns up after the check changes nothing: the call reports
    the refusal, never success without a portfolio."""
    monkeypatch.setenv("RG_MEM_HEADROOM_BYTES", "1000000")
    fake.free_bytes(0, 0, 1 << 40)  # both looks of the check, then plenty
    st, h, message = _create()
    assert (st, h) == (riskgpu.RG_ERR_ADMISSION, None) and "admission refused" in message
    fake.free_bytes(0, 0, 1 << 40)
    assert _create(bad=3)[:2] == (riskgpu.RG_ERR_INVALID, None)
    fake.free_bytes(1 << 40)
    assert _create()[0] == riskgpu.RG_OK


def test_a_missing_device_stays_missing(fake):
    fake.fail("cudaGetDeviceCount", 100)
    st, h, message = _create()
    assert (st, h) == (riskgpu.RG_ERR_NO_DEVICE, None) and "no CUDA device" in message


FREES = ("cudaFree", "cudaFreeAsync")


def test_a_portfolio_outlives_a_refused_wait(fake):
    """Destroyed while a stream capture forbids waiting for the device: work
    launched with it may be in flight, so its memory is not handed on until a
    wait has succeeded, and is then."""
    port = riskgpu.Portfolio(np.zeros(70), np.eye(70))
    before = fake.live()
    fake.reset()
    for name in ("cudaDeviceSynchronize", "cudaFree"):
        fake.fail(name, CAPTURE_REFUSED, count=-1, until="cudaGetErrorString")
    port.close()
    assert fake.live() == before and "cudaFreeAsync" not in fake.names()
    fake.reset()  # the capture has ended
    other = riskgpu.Portfolio(np.zeros(3), np.eye(3))
    names = fake.names()
    free = next(i for i, name in enumerate(names) if name in FREES)
    assert names[free] == "cudaFree" or "cudaDeviceSynchronize" in names[:free]
    other.close()
    assert fake.live() < before
