"""Batched fits whose rows are first tested against their last label's centre:
labels, centres and iteration counts bit-identical to the oracle, at the edges
of the rows handled together (128, 1,024), of the cluster counts that are bounded
(16 k <= n, k <= 128) and on data where no row, few rows or every row stays."""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _data(kind, n, d, k, rng):
    c = rng.uniform(-10, 10, size=(k, d)).astype(np.float32)
    x = c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d)).astype(np.float32)
    if kind == "offset":  # distances far below the values
        x += np.float32(3000)
    elif kind == "grid":  # ties, and duplicate centres below
        x = np.round(x / 4).astype(np.float32)
    elif kind == "tiny":  # distances underflow
        x *= np.float32(1e-22)
    elif kind == "nan":
        x[n // 2, d - 1] = np.nan
        x[3, 0] = np.inf
    elif kind == "flat":  # one cluster's worth of data: nearly every row is open
        x = rng.normal(size=(n, d)).astype(np.float32)
    init = x[rng.choice(n, size=k, replace=False)].copy()
    if kind == "grid" and k > 2:
        init[1] = init[0]
    return x, init


@pytest.mark.parametrize("kind", ["blobs", "flat", "offset", "grid", "tiny", "nan"])
def test_bounded_rows(kind):
    rng = np.random.default_rng(9)
    shapes = [(8, 1, 16), (8, 4, 8193), (16, 5, 1024), (16, 16, 1025), (32, 33, 1023), (32, 64, 1024), (64, 7, 129),
              (64, 64, 1280), (64, 128, 2048), (8, 129, 2064), (16, 17, 271), (12, 6, 500)]
    problems = []
    for d, k, n in shapes:
        x, init = _data(kind, n, d, k, rng)
        problems.append(dict(x=x, k=k, n_init=1, init=init[None].copy(), max_iter=6, tol=0.0))
    fitted, _ = F.fit_batched(problems, reduction="f64")
    for p, f in zip(problems, fitted):
        o = O.fit_runs(p["x"], p["k"], max_iter=6, tol=0.0, n_init=1, init=p["init"], wide_sums=True)
        shape = p["x"].shape + (p["k"],)
        assert f.n_iter() == o["n_iter"][0], shape
        assert np.array_equal(f.labels(), o["labels"][0]), shape
        assert np.array_equal(f.cluster_centers(), o["centers"][0], equal_nan=True), shape


@pytest.mark.parametrize("max_iter", [40, 1 << 20])
def test_sums_carried_over_and_rebuilt(max_iter):
    """To convergence, with the sums kept between iterations and (too many
    iterations for that) rebuilt in each."""
    rng = np.random.default_rng(4)
    x = rng.normal(size=(3000, 16)).astype(np.float32)
    x[::5] *= np.float32(1e-7)  # remainders below the grids
    init = x[rng.choice(3000, size=6, replace=False)][None].copy()
    fitted, _ = F.fit_batched([dict(x=x, k=6, n_init=1, init=init, max_iter=max_iter, tol=0.02)], reduction="f64")
    o = O.fit_runs(x, 6, max_iter=max_iter, tol=0.02, n_init=1, init=init, wide_sums=True)
    assert fitted[0].n_iter() == o["n_iter"][0]
    assert np.array_equal(fitted[0].labels(), o["labels"][0])
    assert np.array_equal(fitted[0].cluster_centers(), o["centers"][0])
