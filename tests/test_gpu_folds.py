"""The exact parallel folds against sequential sums, through BisectingKMeans:
with k = 1 the centre and the SSE are row-order folds of every row."""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["walk", "drift", "grid", "scales", "specials"])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 8193, 40001])
def test_folds_at_chunk_edges(n, kind, dt):
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 5))
    if kind == "drift":  # the sum leaves zero: one sign, a binade change per doubling
        x += np.array([3.0, -3.0, 0.5, 100.0, -1e-3])
    elif kind == "grid":  # exact halves at every step
        x = rng.integers(-3, 4, size=(n, 5)) * 0.5
    elif kind == "scales":  # binades far apart, beyond f32's range in f64
        x *= 10.0 ** rng.integers(-12, 13, size=(n, 5)) * (1e60 if dt == np.float64 else 1.0)
    elif kind == "specials":
        x[n // 2, 0], x[n // 3, 1], x[n - 1, 2] = np.inf, np.nan, -0.0
    x = np.ascontiguousarray(x, dtype=dt)
    g = F.BisectingKMeans(1, "f32" if dt == np.float32 else "f64").with_n_init(1).fit(x)
    o = O.bisecting_fit(x, 1, n_init=1, seed=0)
    assert np.array_equal(g.cluster_centers(), o["centers"], equal_nan=True)
    assert np.array_equal(g.inertia(), o["inertia"], equal_nan=True)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_masked_folds_of_every_run(dt):
    rng = np.random.default_rng(8)
    x = (rng.normal(size=(9001, 7)) + rng.integers(-1, 2, size=(9001, 1)) * 4).astype(dt)
    g = F.BisectingKMeans(6, "f32" if dt == np.float32 else "f64").with_n_init(5).with_random_state(3).fit(x)
    o = O.bisecting_fit(x, 6, n_init=5, seed=3)
    assert np.array_equal(g.cluster_centers(), o["centers"]) and np.array_equal(g.labels(), o["labels"])
    assert g.inertia() == o["inertia"]
