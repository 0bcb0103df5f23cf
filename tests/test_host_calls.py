"""Host side of portfolio and query calls on the fake runtime: statuses, memory
and the order of runtime calls where memory is short, a call is refused or many
callers meet."""
import ctypes
import threading

import numpy as np
import pytest

import riskgpu
from host_engine import CAPTURE_REFUSED, OOM, fake, linked  # noqa: F401


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
LARGE = 2100  # a portfolio whose memory is not kept for the next one


def _portfolio(n):
    return riskgpu.Portfolio(np.zeros(n), np.eye(n))


@pytest.mark.parametrize("n", [70, LARGE])
def test_a_portfolio_outlives_a_refused_wait(fake, n):
    """Destroyed while a stream capture forbids waiting for the device: work
    launched with it may be in flight, so its memory is not handed on until a
    wait has succeeded, and is then."""
    port = _portfolio(n)
    one = fake.live()
    fake.reset()
    for name in ("cudaDeviceSynchronize", "cudaFree"):
        fake.fail(name, CAPTURE_REFUSED, count=-1, until="cudaGetErrorString")
    port.close()
    assert fake.live() == one and "cudaFreeAsync" not in fake.names()
    second = _portfolio(n)
    assert fake.live() == 2 * one
    fake.reset()  # the capture has ended
    third = _portfolio(n)
    names = fake.names()
    free = [i for i, name in enumerate(names) if name in FREES and name != "cudaFreeAsync"]
    assert "cudaDeviceSynchronize" in names[:free[0] if free else None]
    assert fake.live() == 2 * one
    second.close()
    third.close()


def test_resident_portfolios_own_plain_device_memory(fake):
    """d_L and d_packed are the caller's to map on a peer or to export to
    another process, which memory of a pool does not allow."""
    port = _portfolio(LARGE)
    size = max(int(d) for name, _, d in fake.log() if name == "cudaMalloc")
    assert size >= LARGE * LARGE * 8
    fake.reset()
    port.close()
    assert ("cudaFree", "0", str(size)) in fake.log() and fake.live() == 0
    # a call's own portfolio is the engine's business
    fake.reset()
    riskgpu.run(np.zeros(70), np.eye(70), None, riskgpu.make_query(1000, 3))
    assert not [d for name, _, d in fake.log() if name == "cudaMalloc" and int(d) >= 70 * 70 * 8]


def test_spare_portfolio_memory_is_bounded_and_given_back(fake, monkeypatch):
    ports = [_portfolio(70) for _ in range(20)]
    one = fake.live() // 20
    for p in ports:
        p.close()
    assert fake.live() == 8 * one
    fake.reset()
    again = _portfolio(70)
    assert "cudaMalloc" not in fake.names()
    ports = [_portfolio(900 + 100 * i) for i in range(5)]
    for p in ports + [again]:
        p.close()
    assert fake.live() <= 32 << 20
    # an allocation that fails gets what is kept
    fake.reset()
    fake.fail("cudaMalloc", OOM, count=-1, until="cudaFree")
    port = _portfolio(33)
    size = fake.live()
    port.close()
    assert size < one
    # and so does an admission check that would refuse
    monkeypatch.setenv("RG_MEM_HEADROOM_BYTES", "1000")
    fake.reset()
    fake.free_bytes(0, 1 << 40)
    _portfolio(20).close()
    assert [d for name, _, d in fake.log() if name == "cudaFree"] == [str(size)]


def test_the_latest_portfolio_memory_is_the_spare_one(fake):
    for n in list(range(10, 30)) + [70]:
        _portfolio(n).close()
    fake.reset()
    _portfolio(70).close()
    assert not {"cudaMalloc", "cudaFree"} & set(fake.names())


def _run(**more):
    return riskgpu.run(np.zeros(20), np.eye(20), np.full(20, 0.05), riskgpu.make_query(1000, 3, **more))


@pytest.mark.parametrize("name,call", [
    ("cudaMallocFromPoolAsync", _run),
    ("cudaMallocFromPoolAsync", lambda: riskgpu.moments(np.ones((5, 3)))),
    ("cudaMallocFromPoolAsync", lambda: riskgpu.crash_frequency(np.ones((5, 3)), 0.02, 1)),
    ("cudaMalloc", lambda: _portfolio(LARGE).close()),
    ("cudaMalloc", lambda: riskgpu.Batch([(_portfolio(20), riskgpu.make_query(1000, 3, precision=riskgpu.PREC_FP16X3))])),
])
def test_what_the_engine_keeps_does_not_fail_an_allocation(fake, name, call):
    call()  # (process-wide state exists)
    for skip in range(4):
        fake.reset()
        fake.fail(name, OOM, skip=skip, count=-1, until="cudaMemPoolTrimTo")
        call()
        assert skip or "cudaMemPoolTrimTo" in fake.names()


def test_many_callers_at_once_make_no_device_wide_calls(fake):
    """Sixteen callers inside rg_simulate together, in waves: beyond the eight
    kept resources a call uses stream-ordered memory only, and nothing is given
    back in a way that waits for the device."""
    port, results = _portfolio(20), []

    def call():
        results.append(port.simulate(riskgpu.make_query(1000, 3)))

    for wave in range(3):
        fake.reset()
        fake.gather("cudaEventRecord", 16)
        threads = [threading.Thread(target=call) for _ in range(16)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        names = fake.names()
        made = 8 if wave == 0 else 0
        assert names.count("cudaHostAlloc") == names.count("cudaMalloc") == made
        assert not {"cudaFreeHost", "cudaFree", "cudaDeviceSynchronize"} & set(names)
        assert names.count("cudaMallocFromPoolAsync") == names.count("cudaFreeAsync") == 8
    assert len(results) == 48 and all(r["n_paths"] == 1000 for r in results)


def test_a_query_needs_no_pinned_memory(fake):
    port = _portfolio(20)
    fake.fail("cudaHostAlloc", OOM, count=-1)
    before = fake.live()
    for _ in range(3):
        assert port.simulate(riskgpu.make_query(1000, 3))["n_paths"] == 1000
    assert fake.live() == before
    fake.reset()
    port.simulate(riskgpu.make_query(1000, 3))
    assert "cudaHostAlloc" in fake.names() and "cudaFreeHost" not in fake.names()


def test_block_tables_ask_for_admission(fake, monkeypatch):
    """A table is memory that a query can do without: where the check would
    refuse it the call runs without one, and is not refused."""
    port = _portfolio(640)
    query = riskgpu.make_query(1_000_000, 3, horizon=20, precision=riskgpu.PREC_BF16X3)
    table = 640 // 4 * 20 * 16

    def pooled(call):
        fake.reset()
        call()
        return [int(d) for name, _, d in fake.log() if name in ("cudaMallocFromPoolAsync", "cudaMalloc")]

    counts = np.zeros(2, dtype=np.uint64)
    calls = [lambda: port.simulate(query), lambda: port.launch_counts(query, counts.ctypes.data),
             lambda: riskgpu.Batch([(port, query)]).close()]
    for call in calls:
        assert table in pooled(call)
    monkeypatch.setenv("RG_MEM_HEADROOM_BYTES", str(1 << 30))
    for call in calls:
        assert table in pooled(call)
    for call in calls:  # room for the rest of the call's memory, not for the table
        fake.reset()
        free = (1 << 30) + table - 1
        fake.free_bytes(free)
        call()
        assert table not in [int(d) for name, _, d in fake.log()
                             if name in ("cudaMallocFromPoolAsync", "cudaMalloc")]


@pytest.mark.parametrize("name,err,status", [("cudaMalloc", OOM, riskgpu.RG_ERR_NOMEM),
                                             ("cudaMallocFromPoolAsync", OOM, riskgpu.RG_ERR_NOMEM),
                                             ("launch", 700, riskgpu.RG_ERR_CUDA)])
def test_bad_input_is_reported_before_a_failed_creation(fake, name, err, status):
    for bad in (None, 3):
        fake.fail(name, err, count=-1)
        assert _create(bad=bad)[:2] == (status if bad is None else riskgpu.RG_ERR_INVALID, None)
        assert ("row 3" in riskgpu.lib().rg_last_error().decode()) == (bad is not None)
