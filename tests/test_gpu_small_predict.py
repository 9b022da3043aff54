"""Small predict calls (one launch): labels equal to the oracle's at the edges of
the lanes a row takes, of a block's rows and of the rule (n d k <= 10^6)."""
import numpy as np
import pytest
import torch

from ferrolearn_gb300.kmeans import FittedKMeans
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k", [(1, 1, 1), (31, 3, 4), (33, 7, 5), (127, 16, 8), (129, 16, 9), (1000, 16, 8),
                                   (65, 128, 32), (100, 64, 33), (100, 64, 65), (3000, 20, 16), (3126, 20, 16),
                                   (15625, 8, 8), (3, 128, 33)])
def test_small_predict(n, d, k, dt):
    rng = np.random.default_rng(n + k)
    c = rng.normal(size=(k, d)).astype(dt)
    x = rng.normal(size=(n, d)).astype(dt)
    if k > 2:
        c[k - 1] = c[1]  # ties: the lower index
        x[::3] = c[1]
        c[0, 0] = np.nan
    if n > 40:
        x[5, 0], x[40, d - 1] = np.nan, np.inf
    model = FittedKMeans(c, None, 0.0, 0, "f32" if dt == np.float32 else "f64")
    want = O.predict(c, x)
    assert np.array_equal(model.predict(x), want)
    assert np.array_equal(np.asarray(model.predict(torch.from_numpy(x).cuda())), want)
