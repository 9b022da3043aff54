"""The f64 reduction's sums where several row ranges, small values and
non-finite values meet in one cluster: bit-identical to the oracle's exact
sums (128-bit fixed point, rounded once)."""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["wide range", "tiny", "huge", "inf", "nan"])
def test_f64_reduction_of_awkward_values(kind):
    rng = np.random.default_rng(2)
    n, d, k = 20011, 8, 5  # three row ranges of 8,192 rows
    x = rng.normal(size=(n, d)).astype(np.float32)
    x[:, 0] *= np.float32(50) * rng.integers(0, 2, size=n)  # two groups
    if kind == "wide range":  # below 2^-21 of the largest: the 128-bit remainder
        x[::3] *= np.float32(1e-9)
        x[5] = 1e4
    elif kind == "tiny":  # outside the grids' exponents
        x *= np.float32(1e-33)
    elif kind == "huge":
        x *= np.float32(1e15)
    elif kind == "inf":
        x[7, 2], x[9000, 2], x[12, 3] = np.inf, np.inf, -np.inf
    else:
        x[11, 1] = np.nan
    init = x[[1, 4000, 9001, 15000, 20000]][None].copy()
    fitted, rep = F.fit_batched([dict(x=x, k=k, n_init=1, init=init, max_iter=3, tol=0.0)], reduction="f64")
    o = O.fit_runs(x, k, max_iter=3, tol=0.0, n_init=1, init=init, wide_sums=True)
    assert np.array_equal(fitted[0].cluster_centers(), o["centers"][0], equal_nan=True)
    assert np.array_equal(fitted[0].labels(), o["labels"][0])
    assert fitted[0].n_iter() == o["n_iter"][0]
