"""k-means++ at the edges of its tiles, against the oracle's sequential folds.

Exact equality: every sum is the reference's left fold in F (kmeans.rs:201,
215-237), so the chosen rows and the draws consumed are the oracle's.
"""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rows(n, d, kind, seed, dt):
    rng = np.random.default_rng(seed)
    if kind == "blobs":  # most rows skipped by the candidates' thresholds once the blobs are covered
        c = rng.uniform(-20, 20, size=(6, d))
        x = c[rng.integers(0, 6, size=n)] + rng.normal(size=(n, d))
    elif kind == "grid":  # exact halves and equal distances
        x = rng.integers(-2, 3, size=(n, d)).astype(np.float64)
    else:  # one far row holds almost the whole sum: the folds hardly move
        x = rng.normal(size=(n, d))
        x[n // 2] = 1e6
    return np.ascontiguousarray(x, dtype=dt)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["blobs", "grid", "outlier"])
@pytest.mark.parametrize("n,d,k", [(255, 1, 2), (256, 4, 3), (257, 7, 9), (1023, 64, 5), (1025, 65, 8),
                                   (8193, 60, 21), (20001, 130, 12), (3000, 3, 1100)])
def test_kmeanspp_tile_edges(n, d, k, kind, dt):
    x = _rows(n, d, kind, n + d, dt)
    name = "f32" if dt == np.float32 else "f64"
    dr = F.draws(n * 7 + k, 1 + (k - 1) * (2 + int(np.floor(np.log(k)))))
    oc, ou = O.kmeanspp(x, k, dr)
    gc, gu = F.kmeans_plus_plus(x, k, dr, dtype=name)
    assert gu == ou and np.array_equal(gc, oc)
    gc, _ = F.kmeans_plus_plus(x, k, seed=n * 7 + k, dtype=name)  # the library's own stream: the same draws
    assert np.array_equal(gc, oc)


@pytest.mark.parametrize("name", ["f32", "f64"])
def test_restarts_seeded_together(name):
    x = _rows(9001, 6, "blobs", 4, np.float32 if name == "f32" else np.float64)
    g = F.KMeans(7, dtype=name).with_n_init(5).with_random_state(3).with_max_iter(4).fit(x)
    o = O.fit(x, 7, max_iter=4, n_init=5, seed=3)
    assert np.array_equal(g.cluster_centers(), o["centers"]) and np.array_equal(g.labels(), o["labels"])
    assert g.report["best_run"] == o["best_run"]


def test_batched_seedings_of_uneven_sizes():
    probs = []
    for i, (n, d, k) in enumerate([(3, 2, 2), (1024, 8, 16), (5000, 16, 1), (2049, 5, 64), (30000, 32, 9)]):
        probs.append(dict(x=_rows(n, d, "blobs", i, np.float32), k=k, n_init=3, max_iter=0, random_state=50 + i))
    fitted, _ = F.fit_batched(probs)
    for f, p in zip(fitted, probs):  # no iteration: run 0 is kept, its centres are its seeds
        assert np.array_equal(f.cluster_centers(), O.kmeanspp(p["x"], p["k"], seed=p["random_state"])[0])


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("scale", [1.0, 1e-19, 1e17])
@pytest.mark.parametrize("kind", ["few points", "near ties"])
def test_trials_of_nearly_equal_potential(kind, scale, dt):
    """Equal and nearly equal trials (the first of the smallest wins), and sums at
    the ends of the estimates' range."""
    rng = np.random.default_rng(8)
    if kind == "few points":  # 12 places, many rows each: trials repeat
        x = rng.normal(size=(12, 4))[rng.integers(0, 12, size=5000)]
    else:  # mirror images: potentials equal but for their roundings
        h = rng.normal(size=(2500, 4))
        x = np.concatenate([h, -h])
    x = np.ascontiguousarray(x * scale, dtype=dt)
    name = "f32" if dt == np.float32 else "f64"
    for seed in range(4):
        oc, _ = O.kmeanspp(x, 20, seed=seed)
        gc, _ = F.kmeans_plus_plus(x, 20, seed=seed, dtype=name)
        assert np.array_equal(gc, oc), seed


@pytest.mark.parametrize("kind", ["blobs", "grid", "outlier"])
@pytest.mark.parametrize("n,d,k,runs", [(100001, 5, 9, 1), (102401, 37, 6, 1), (50009, 4, 8, 2), (26000, 16, 12, 5),
                                        (1300001, 3, 5, 1)])
def test_split_steps(n, d, k, runs, kind):
    """f64 steps of 100,000 rows and more: estimates first, then the arrays of the
    trials that can win (n at the edges of both passes' tiles)."""
    x = _rows(n, d, kind, n + d, np.float64)
    if runs == 1:
        x[::9] = x[1]  # equal rows
        oc, _ = O.kmeanspp(x, k, seed=n)
        gc, _ = F.kmeans_plus_plus(x, k, seed=n, dtype="f64")
        assert np.array_equal(gc, oc)
    else:
        g = F.KMeans(k, dtype="f64").with_n_init(runs).with_random_state(n).with_max_iter(2).fit(x)
        o = O.fit(x, k, max_iter=2, n_init=runs, seed=n)
        assert np.array_equal(g.cluster_centers(), o["centers"]) and np.array_equal(g.labels(), o["labels"])
        assert g.report["best_run"] == o["best_run"]
