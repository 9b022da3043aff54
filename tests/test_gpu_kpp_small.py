"""f32 k-means++ of up to 1,024 rows, 256 features and 65,536 values, a seeding a CTA: the oracle's
centres and draws at the edges of the groups of 32 values, of the trials scored at
a time (4) and of the form, on data with ties, equal rows, zero sums and values
that are not finite."""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from ferrolearn_gb300 import _native
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ROWS = [(1, 3, 1), (2, 1, 2), (31, 5, 4), (32, 8, 7), (33, 7, 20), (63, 2, 63), (64, 16, 12), (257, 33, 55), (992, 6, 30),
        (257, 255, 8), (256, 256, 21), (1023, 64, 9), (1024, 63, 5), (1024, 64, 149)]


def _rows(kind, n, d, seed):
    rng = np.random.default_rng(seed)
    if kind == "blobs":
        c = rng.uniform(-20, 20, size=(6, d))
        x = c[rng.integers(0, 6, size=n)] + rng.normal(size=(n, d))
    elif kind == "grid":
        x = rng.integers(-2, 3, size=(n, d)).astype(np.float64)
    elif kind == "few points":  # the sum is zero once every place is a centre
        x = rng.normal(size=(3, d))[rng.integers(0, 3, size=n)]
    elif kind == "huge":  # sums beyond f32
        x = rng.normal(size=(n, d)) * 1e19
    elif kind == "tiny":
        x = rng.normal(size=(n, d)) * 1e-22
    else:
        x = rng.normal(size=(n, d))
        x[n // 2, 0] = np.nan
        x[n // 3, d - 1] = np.inf
    with np.errstate(over="ignore"):
        return np.ascontiguousarray(x, dtype=np.float32)


@pytest.mark.parametrize("kind", ["blobs", "grid", "few points", "huge", "tiny"])
@pytest.mark.parametrize("n,d,k", ROWS)
def test_small_seeding_matches_oracle(n, d, k, kind):
    x = _rows(kind, n, d, n + d)
    dr = F.draws(n * 7 + k, 1 + (k - 1) * (2 + int(np.floor(np.log(k)))))
    before = _native.lib().fk_debug_launch_count()
    gc, gu = F.kmeans_plus_plus(x, k, dr, dtype="f32")
    assert _native.lib().fk_debug_launch_count() - before == 1
    oc, ou = O.kmeanspp(x, k, dr)
    assert gu == ou and np.array_equal(gc, oc, equal_nan=True)
    assert np.array_equal(F.kmeans_plus_plus(x, k, seed=n * 7 + k, dtype="f32")[0], oc, equal_nan=True)


@pytest.mark.parametrize("n,d", [(1025, 8), (1024, 65), (64, 257)])
def test_beyond_the_line(n, d):
    x = _rows("blobs", n, d, 3)
    before = _native.lib().fk_debug_launch_count()
    gc, _ = F.kmeans_plus_plus(x, 9, seed=5, dtype="f32")
    assert _native.lib().fk_debug_launch_count() - before > 1
    assert np.array_equal(gc, O.kmeanspp(x, 9, seed=5)[0])


@pytest.mark.parametrize("kind", ["blobs", "grid", "few points", "nonfinite"])
def test_fits_and_batches_of_small_seedings(kind):
    probs = []
    for i, (n, d, k) in enumerate([(3, 2, 2), (1024, 8, 16), (500, 16, 1), (40, 5, 33), (1000, 32, 9)]):
        probs.append(dict(x=_rows(kind, n, d, i), k=k, n_init=3, max_iter=0, random_state=50 + i))
    fitted, _ = F.fit_batched(probs)
    for f, p in zip(fitted, probs):  # no iteration: run 0 is kept, its centres are its seeds
        want = O.fit_runs(p["x"], p["k"], max_iter=0, tol=0.0, n_init=3, seed=p["random_state"])["centers"][0]
        assert np.array_equal(f.cluster_centers(), want, equal_nan=True)
    if kind == "nonfinite":
        return
    x = _rows(kind, 1000, 6, 4)
    g = F.KMeans(7, dtype="f32").with_n_init(5).with_random_state(3).with_max_iter(4).fit(x)
    o = O.fit(x, 7, max_iter=4, n_init=5, seed=3)
    assert np.array_equal(g.cluster_centers(), o["centers"]) and np.array_equal(g.labels(), o["labels"])


@pytest.mark.parametrize("reduction", ["reference", "f64"])
@pytest.mark.parametrize("d", [8, 16, 20, 64])
def test_batches_of_small_fits_take_no_bounds(d, reduction):
    # (their thresholds' launch would take longer than it saves; larger fits in the call bring them back)
    rng = np.random.default_rng(d)
    probs = []
    for i, (n, k) in enumerate([(1, 1), (127, 3), (1000, 9), (2047, 30), (40, 40)]):
        x = rng.normal(size=(n, d)).astype(np.float32)
        x[: n // 2] += 6
        probs.append(dict(x=x, k=k, n_init=2, max_iter=25, tol=1e-4, random_state=i))
    alone, _ = F.fit_batched(probs, reduction=reduction)
    big = dict(x=rng.normal(size=(3000, d)).astype(np.float32), k=9, n_init=1, max_iter=25, tol=1e-4, random_state=1)
    together, _ = F.fit_batched(probs + [big], reduction=reduction)
    for a, b, p in zip(alone, together, probs):
        assert np.array_equal(a.labels(), b.labels()) and np.array_equal(a.cluster_centers(), b.cluster_centers())
        assert a.n_iter() == b.n_iter() and a.inertia() == b.inertia()
        if reduction == "reference":
            o = O.fit(p["x"], p["k"], max_iter=25, tol=1e-4, n_init=2, seed=p["random_state"])
            assert np.array_equal(a.labels(), o["labels"]) and np.array_equal(a.cluster_centers(), o["centers"])
