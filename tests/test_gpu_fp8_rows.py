"""FP8 rows with infinities, NaN, subnormal and huge values among ordinary ones: the
row scales ignore what is not finite, and every label equals the oracle's."""
import numpy as np
import pytest

from ferrolearn_gb300.kmeans import MIXED_FP8, FittedKMeans
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 128, 252, 256])
def test_fp8_rows_of_every_scale(d):
    rng = np.random.default_rng(d)
    n, k = 5001, 130
    c = rng.normal(size=(k, d)).astype(np.float32)
    x = (c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d)) * 0.3).astype(np.float32)
    x[::50] *= np.float32(1e-39)  # subnormal
    x[1::50] *= np.float32(1e30)
    x[2::50, 0] = np.inf
    x[3::50, d - 1] = -np.inf
    x[4::50, d // 2] = np.nan
    x[5::50] = 0
    x[6] = np.inf
    got = FittedKMeans(c.astype(np.float64), None, 0.0, 0, "f32x64", precision=MIXED_FP8).predict(x)
    assert np.array_equal(got, O.predict(c.astype(np.float64), x.astype(np.float64)))
