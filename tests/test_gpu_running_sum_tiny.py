"""The grow's running sum over subnormal values (GPU) at every edge of its chunks and tiles, from a sum of ordinary size;
from zero, where each value is added by itself, a few."""
import numpy as np
import pytest

from test_gpu_running_sum import device_sum, values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('tiles', [0, 1])
@pytest.mark.parametrize('n', [1, 31, 2047, 2048, 2049, 4095, 4096, 4097, 10000, 300001])
def test_subnormal_values(n, tiles):
    for a, pw in ((0.0, 1.0), (1.0, 1.0), (0.7, 32.0), (1 - 2.0**-53, 1.0), (2.0**-1021, 1.0)):
        m = min(n, 300) if a < 2.0**-900 else n
        v = values('tiny', m)
        want = np.add.accumulate(np.concatenate([[a], np.abs(v)*pw]))[-1]
        assert device_sum(v, a, pw, tiles) == want, (m, a, pw)
