"""Fits large enough that the plain assignment leaves centres out: labels and
centres bit-identical to the oracle's after every number of iterations that
reaches another route (all centres, kept labels, near centres, open rows)."""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(kind, n, d, k, seed):
    rng = np.random.default_rng(seed)
    if kind == "blobs":  # most labels kept, split blobs compared with a few near centres
        c = rng.uniform(-20, 20, size=(k // 2, d))
        x = c[rng.integers(0, k // 2, size=n)] + rng.normal(size=(n, d))
    elif kind == "uniform":  # no structure: every row against every centre
        x = rng.uniform(-1, 1, size=(n, d))
    elif kind == "grid":  # exact ties and equal centres
        x = rng.integers(-1, 2, size=(n, d)).astype(np.float64)
    elif kind == "far":  # squares beyond f32 for some rows, far below for others
        x = rng.normal(size=(n, d)) * 10.0 ** rng.integers(-25, 25, size=(n, 1))
    else:
        c = rng.uniform(-20, 20, size=(k, d))
        x = c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d))
        x[17, 0], x[n // 2, 1], x[n - 1, 2] = np.nan, np.inf, -np.inf
    init = x[rng.permutation(n)[:k]].copy()
    init[~np.isfinite(init)] = 0.0
    init[3] = init[1]  # two equal centres: the lower index wins, the other stays empty
    return x, init


@pytest.mark.parametrize("name", ["f32", "f64"])
@pytest.mark.parametrize("kind", ["blobs", "uniform", "grid", "far", "nonfinite"])
@pytest.mark.parametrize("n,d,k", [(62501, 64, 256), (120007, 37, 255), (70003, 450, 33), (260001, 3, 1300)])
def test_pruned_fit_matches_oracle(n, d, k, kind, name):
    assert n * k * d >= 1e9  # the size from which the fit prunes
    dt = np.float32 if name == "f32" else np.float64
    x, init = _case(kind, n, d, k, n + d)
    with np.errstate(over="ignore"):
        x, init = np.ascontiguousarray(x, dtype=dt), init.astype(dt)
    init[~np.isfinite(init)] = 0.0
    c = init
    steps = []
    for _ in range(5):  # the oracle's iterations, one at a time
        ol, oc, oi, os_ = O.lloyd_step(x, c)
        steps.append((ol, oc, oi))
        c = oc
    for it in (1, 2, 5):
        g = F.KMeans(k, dtype=name).with_max_iter(it).with_tol(0.0).with_n_init(1).with_init_centers(init).fit(x)
        ol, oc, oi = steps[it - 1]
        assert np.array_equal(g.labels(), ol), it
        assert np.array_equal(g.cluster_centers(), oc, equal_nan=True), it
        assert g.inertia() == oi or not np.isfinite(oi) or abs(g.inertia() - oi) <= (1e-5 if dt == np.float32 else 1e-12) * oi
