"""The f64 filter's two tile sizes at the row counts where one takes over from the other
(5/8 of a 128-row tile an SM, a whole one up to 64 centres): the oracle's labels, ties
and non-finite values included."""
import numpy as np
import pytest
import torch

from ferrolearn_gb300.kmeans import FittedKMeans
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,k", [(31, 64), (32, 64), (32, 65), (70, 257)])
@pytest.mark.parametrize("tiles_of_8_sms", [5, 8])
def test_labels_on_both_sides_of_the_line(tiles_of_8_sms, d, k):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    edge = (tiles_of_8_sms * sms + 7) // 8 * 128  # the first count that the line excludes starts above (tiles - 1) * 128
    rng = np.random.default_rng(edge + d)
    for n in (edge - 128, edge - 127, edge):
        c = rng.integers(-3, 4, size=(k, d)).astype(np.float64)
        c[k - 1] = c[1]
        x = c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d))
        x[::9] = (c[0] + c[2]) / 2  # exact ties
        x[5, 1], x[6, 0] = np.nan, np.inf
        got = FittedKMeans(c, None, 0.0, 0, "f64").predict(torch.from_numpy(x).cuda())
        assert np.array_equal(got, O.predict(c, x)), n
