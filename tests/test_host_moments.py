"""Host side of the preprocessing calls on the fake runtime: device memory, and
what happens where a runtime call fails."""
import numpy as np
import pytest

import riskgpu
from host_engine import OOM, fake, linked  # noqa: F401


@pytest.mark.parametrize("days,n", [(2, 1600), (50, 3000), (70, 1), (2000, 600)])
def test_memory_of_the_moments(fake, days, n):
    """The matrix, mu, Sigma and 64 column sums; partial tiles only where few
    columns leave room for many row segments (20 MB at most)."""
    riskgpu.crash_frequency(np.zeros((2, 2)), 0.02, 1)
    fake.reset()
    riskgpu.moments(np.zeros((days, n)))
    tiles = (n + 31) // 32 * ((n + 31) // 32 + 1) // 2
    partials = 0 if tiles >= 8 * 152 or days < 128 else (8 * 152 + tiles) * 32 * 32
    assert fake.peak() <= 8 * (days * n + n * n + 65 * n + partials + 1)


CALLS = [lambda X: riskgpu.moments(X), lambda X: riskgpu.crash_frequency(X, 0.02, 1)]


@pytest.mark.parametrize("call", CALLS)
@pytest.mark.parametrize("name,skip", [("launch", 0), ("cudaMemcpyAsync", 1), ("cudaMemcpyAsync", 2),
                                       ("cudaMemcpyAsync", 3)])
def test_no_copy_in_flight_when_a_failed_call_returns(fake, call, name, skip):
    """The caller may free or reuse its arrays: the copies issued are waited for."""
    fake.reset()
    fake.fail(name, 700, skip=skip)
    try:
        call(np.zeros((40, 3)))
    except riskgpu.RiskGpuError as e:
        assert e.status == riskgpu.RG_ERR_CUDA
    names = fake.names()
    last_copy = max(i for i, n in enumerate(names) if n == "cudaMemcpyAsync")
    assert "cudaStreamSynchronize" in names[last_copy:]


@pytest.mark.parametrize("call", CALLS)
@pytest.mark.parametrize("name,err,status", [("cudaGetDeviceCount", 100, riskgpu.RG_ERR_NO_DEVICE),
                                             ("cudaMallocFromPoolAsync", OOM, riskgpu.RG_ERR_NOMEM),
                                             ("launch", 700, riskgpu.RG_ERR_CUDA)])
def test_bad_input_is_reported_before_a_failed_call(fake, call, name, err, status):
    X = np.zeros((40, 3))
    for bad in (False, True):
        if bad:
            X[17, 2] = np.inf
        fake.fail(name, err, count=-1)
        with pytest.raises(riskgpu.RiskGpuError) as e:
            call(X)
        assert e.value.status == (riskgpu.RG_ERR_INVALID if bad else status)
        assert ("returns[17][2]" in str(e.value)) == bad
