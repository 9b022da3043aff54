"""f64 labels of rows that the FP32 bounds leave open: equal to the oracle's, with
few candidates a row, with more than a block's list holds (every centre ties) and
with more centres than its bounds have room for, at the edges of its tiles."""
import numpy as np
import pytest

from ferrolearn_gb300.kmeans import FittedKMeans
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 63, 65, 200, 1024, 1025])
@pytest.mark.parametrize("kind", ["pairs", "all tie", "nonfinite"])
def test_open_rows(kind, k):
    rng = np.random.default_rng(k)
    for n, d in [(1, 3), (15, 31), (17, 33), (1000, 50)]:
        c = rng.normal(size=(k, d))
        x = c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d)) * 0.1
        if kind == "pairs":  # bisectors of two centres, moved by less than FP32 resolves
            a, b = c[rng.integers(0, k, size=n)], c[rng.integers(0, k, size=n)]
            x = (a + b) / 2 + (a - b) * rng.normal(size=(n, 1)) * 1e-13
        elif kind == "all tie":
            c[:] = c[0]
            c[k // 2:] *= 1 + 1e-15
        else:
            x[0, 0], x[n // 2, d - 1] = np.nan, np.inf
            c[k // 2, 0] = np.nan
            x[n - 1] = 1e300
        got = FittedKMeans(c, None, 0.0, 0, "f64").predict(x)
        assert np.array_equal(got, O.predict(c, x)), (n, d)
