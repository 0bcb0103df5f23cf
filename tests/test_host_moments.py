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
