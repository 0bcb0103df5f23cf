"""Host side of batches on the fake runtime: the order of the runtime calls that
set a batch up."""
import json
import os

import numpy as np

import riskgpu
from host_engine import fake, linked  # noqa: F401


def _items(sizes, horizon=8, paths=20_000, **more):
    more = dict(dict(precision=riskgpu.PREC_BF16X3), **more)
    return [(riskgpu.Portfolio(np.zeros(n), np.eye(n), np.full(n, 1.0 / n)),
             riskgpu.make_query(paths, 7 + i, horizon=horizon, **more)) for i, n in enumerate(sizes)]


def test_item_table_is_on_the_device_before_the_table_kernel_reads_it(fake):
    """The upload and the kernel share a stream, or something between them
    waits: a copy from pageable memory on another stream may return before its
    data has arrived."""
    items = _items([10, 80, 300])
    fake.reset()
    batch = riskgpu.Batch(items)
    log = fake.log()
    at = next(i for i, (name, _, d) in enumerate(log) if name == "launch" and "batch_tables" in d)
    up = max(i for i in range(at) if log[i][0].startswith("cudaMemcpy") and log[i][2].startswith("H2D"))
    waited = any(name == "cudaStreamSynchronize" and s == log[up][1] or name == "cudaDeviceSynchronize"
                 for name, s, _ in log[up + 1:at])
    assert log[up][1] == log[at][1] or waited, (log[up], log[at])
    batch.close()


def test_the_two_forms_are_tuned_apart(fake):
    """Same sizes and paths, so the same class but for the form: twenty days a
    path take the merged form, one day the split form."""
    many, one = (riskgpu.Batch(_items([300, 300], horizon=h)) for h in (20, 1))
    assert (many.info()["tuned"], one.info()["tuned"]) == (0, 0)
    path = os.environ["RG_TUNE_CACHE"]
    many.tune()
    with open(path) as f:
        key, = json.load(f)
    with open(path, "w") as f:  # as a file of the form without a suffix holds it
        json.dump({key: [7, 1, 0.5]}, f)
    many, one = (riskgpu.Batch(_items([300, 300], horizon=h)) for h in (20, 1))
    assert many.info()["tuned"] == 1 and many.info()["unit_tiles"] == 7
    assert one.info()["tuned"] == 0 and one.info()["unit_tiles"] == 1
    one.tune()
    with open(path) as f:
        saved = json.load(f)
    assert len(saved) == 2 and saved[key][0] == 7
    assert riskgpu.Batch(_items([300, 300], horizon=1)).info()["tuned"] == 1
