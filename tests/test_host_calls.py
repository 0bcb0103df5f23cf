"""Host side of portfolio and query calls on the fake runtime: statuses, memory
and the order of runtime calls where memory is short, a call is refused or many
callers meet."""
import ctypes
import threading

import numpy as np
import pytest

import riskgpu
from host_engine import OOM, fake, linked  # noqa: F401


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


def _portfolio(n):
    return riskgpu.Portfolio(np.zeros(n), np.eye(n))


@pytest.mark.parametrize("n", [3, 70, 700])
def test_resident_portfolios_own_plain_device_memory(fake, n):
    """d_L and d_packed are the caller's to map on a peer or to export to
    another process, which memory of a pool does not allow; work that reads
    them may be in flight, which cudaFree waits for.  A wait for the whole
    device would end a stream capture of any thread."""
    port = _portfolio(n)
    size = max(int(d) for name, _, d in fake.log() if name == "cudaMalloc")
    assert size >= n * n * 8
    port.info()
    fake.reset()
    port.close()
    log = fake.log()
    assert [d for name, _, d in log if name in ("cudaFree", "cudaFreeAsync")] == [str(size)] and fake.live() == 0
    assert "cudaDeviceSynchronize" not in fake.names()
    modes = [d for name, _, d in log[:fake.names().index("cudaFree")] if name == "cudaThreadExchangeStreamCaptureMode"]
    assert modes == ["relaxed"]
    # a call's own portfolio is the engine's business
    fake.reset()
    riskgpu.run(np.zeros(70), np.eye(70), None, riskgpu.make_query(1000, 3))
    assert not [d for name, _, d in fake.log() if name == "cudaMalloc" and int(d) >= 70 * 70 * 8]


def _noalloc(port):
    return riskgpu.lib().rg_simulate_noalloc(port.handle, ctypes.byref(riskgpu.make_query(1000, 3)),
                                             ctypes.byref(riskgpu.Result()), None)


SHARING = {
    "info": lambda port: port.info(),
    "launch_counts": lambda port: port.launch_counts(riskgpu.make_query(1000, 3), np.zeros(2).ctypes.data),
    "noalloc": lambda port: _noalloc(port),
    "batch": lambda port: riskgpu.Batch([(port, riskgpu.make_query(1000, 3, precision=riskgpu.PREC_FP16X3))]).close(),
    "server": lambda port: riskgpu.lib().rg_server_register(SERVER[0]._h, 1, port.handle),
}
SERVER = []


@pytest.mark.parametrize("how", SHARING)
def test_memory_that_others_may_read_is_not_handed_on(fake, how):
    """Work that no call waits for may still read a portfolio after these
    calls: its memory is freed, which waits, and not kept for the next one."""
    if how == "server":
        SERVER.append(riskgpu.Server())
    port = _portfolio(70)
    if how == "noalloc":  # one that fails
        fake.fail("cudaStreamSynchronize", 700)
    SHARING[how](port)
    fake.reset()
    port.close()
    assert "cudaFree" in fake.names()
    fake.reset()
    _portfolio(70)
    assert "cudaMalloc" in fake.names()
    while SERVER:
        SERVER.pop().close()


def test_spare_memory_is_bounded_and_given_back(fake, monkeypatch):
    """Portfolios whose every call has waited leave their memory for the next
    ones: the latest blocks, at most eight and 32 MiB."""
    def use(n):
        port = _portfolio(n)
        port.factor()
        if n <= 768:
            port.simulate(riskgpu.make_query(1000, 3))
            assert _noalloc(port) == riskgpu.RG_OK
        return port

    use(40).close()
    rest = fake.live()  # and the kept query resources
    fake.reset()
    use(40).close()
    assert not {"cudaMalloc", "cudaFree", "cudaDeviceSynchronize"} & set(fake.names())
    ports = [use(70) for _ in range(20)]
    one = (fake.live() - rest) // 20
    for p in ports:
        p.close()
    assert fake.live() <= rest + 8 * one
    for n in list(range(10, 30)) + [70]:
        use(n).close()
    fake.reset()
    use(70).close()
    assert not {"cudaMalloc", "cudaFree"} & set(fake.names())
    for n in range(900, 1400, 100):
        use(n).close()
    assert fake.live() <= rest + (32 << 20)
    # an allocation that fails, or an admission check that would refuse, gets them
    fake.fail("cudaMalloc", OOM, count=-1, until="cudaFree")
    use(33).close()
    assert fake.live() < rest + one
    monkeypatch.setenv("RG_MEM_HEADROOM_BYTES", "1000")
    fake.reset()
    fake.free_bytes(0, 1 << 40)
    _portfolio(20)
    assert "cudaFree" in fake.names()


def _run(**more):
    return riskgpu.run(np.zeros(20), np.eye(20), np.full(20, 0.05), riskgpu.make_query(1000, 3, **more))


@pytest.mark.parametrize("name,call", [
    ("cudaMallocFromPoolAsync", _run),
    ("cudaMallocFromPoolAsync", lambda: riskgpu.moments(np.ones((5, 3)))),
    ("cudaMallocFromPoolAsync", lambda: riskgpu.crash_frequency(np.ones((5, 3)), 0.02, 1)),
    ("cudaMalloc", lambda: _portfolio(20).info()),
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


@pytest.mark.parametrize("name,call", [
    ("cudaMallocFromPoolAsync", _run),
    ("cudaMalloc", lambda: _portfolio(20).info()),
    ("cudaStreamSynchronize", _run),
    ("cudaMallocFromPoolAsync", lambda: riskgpu.moments(np.ones((5, 3)))),
    ("cudaMalloc", lambda: riskgpu.Batch([(_portfolio(20), riskgpu.make_query(1000, 3, precision=riskgpu.PREC_FP16X3))])),
    ("cudaGraphInstantiate", lambda: riskgpu.Batch([(_portfolio(20),
                                                     riskgpu.make_query(1000, 3, precision=riskgpu.PREC_FP16X3))])),
])
def test_a_failed_call_does_not_fail_the_next(fake, name, call):
    """The runtime keeps the last error until it is asked for; the check after
    the next launch must not find this one's."""
    call()
    for _ in range(2):
        if "Malloc" in name:
            fake.fail(name, OOM, count=2)  # and the second try
        else:
            fake.fail(name, 700)
        with pytest.raises(riskgpu.RiskGpuError):
            call()
        call()
