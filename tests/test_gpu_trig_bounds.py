"""sin / cos at the several thousand doubles on either side of each bound of the argument reduction, on the device,
plain and batched: within one representable value of libm's (their errors, 0.51 and 0.55 ulp, add to less than two)."""
import math

import numpy as np
import pytest

import helpers as H
from ralgpu import dtypes as D
from test_gpu_trig import _both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bound", [0.5, 1.0, 2.0 ** -27, 2.0 ** -26, math.pi / 4, math.pi / 2, math.pi, 2.0 ** 51])
def test_neighbourhood(bound):
    k = np.arange(-4000, 4001, dtype=np.int64)
    x = (np.float64(bound).view(np.int64) + k).view(np.float64)
    x = np.concatenate([x, -x])
    assert len(np.unique(x)) == 16002
    s, c = _both([(D.GDF_FLOAT64, x, None)], "LogicalProject(a=[SIN($0)], b=[COS($0)])")
    for got, fn in ((s, math.sin), (c, math.cos)):
        assert H.ulp_distance(got, np.array([fn(v) for v in x])).max() <= 1
