"""The predicted band of the VaR order statistic where few paths lie beyond the
quantile on the other side of the tail: one pass, as with few paths in the tail
itself.  One standard-normal asset; of these 2000 paths the largest (the order
statistic at level 0.0004) is 5.617, 7.3 standard errors from the quantile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_band_is_wide_where_either_side_has_few_paths(gpu):
    port = gpu.Portfolio(np.zeros(1), np.eye(1), np.ones(1))
    r = port.simulate(gpu.make_query(2000, 5929, var_level=0.0004))
    assert r["tail_count"] == 2000 and abs(r["var"] + 5.6170) <= 1e-3
    assert r["var_passes"] == 1
