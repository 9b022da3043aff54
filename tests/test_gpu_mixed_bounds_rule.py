"""Which fits of the tensor-core forms keep row bounds: on clusters, a fit that
keeps them has listed rows from its fourth iteration on and runs no count pass,
one that does not runs count passes. Labels, centres and n_iter are those of
single steps (which rank every row), bit for bit, and the FP64 oracle's."""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from ferrolearn_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _clusters(n, d, k, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-10, 10, size=(k, d)).astype(np.float32)
    x = c[rng.integers(0, k, size=n)] + 0.5 * rng.standard_normal(size=(n, d), dtype=np.float32)
    return x, k, x[rng.permutation(n)[:k]].astype(np.float64)


def _rows(kind):
    if kind == "nonfinite":
        x, k, init = _clusters(320011, 64, 1024, 3)
        x[5, 3], x[77777, 0], x[300000, 63] = np.nan, np.inf, -np.inf
        return x, k, init
    if kind == "bisector":  # a tenth of the rows stay equidistant: listed, paired, decided in FP64
        w = W.bisector_4096x256(scale=0.0035, k=1024, d=256, predict_scale=0.0001)
        x = np.concatenate([w["x"]] * 6)[:160003]
        x[28000:] += np.random.default_rng(1).normal(0, 0.3, size=x[28000:].shape).astype(np.float32)
        return x, w["k"], w["init"]
    n, d, k = kind
    return _clusters(n, d, k, n)


def _check(kind, precision, steps=8):
    x, k, init = _rows(kind)
    c = init
    for _ in range(steps):
        prev = c
        labels, c, _, _, _ = F.lloyd_step(x, c, dtype="f32x64", precision=precision)
    for _ in range(2):  # the second fit replays the first one's captured iterations
        g = F.KMeans(k, dtype="f32x64").with_precision(precision).with_max_iter(steps).with_tol(0.0) \
            .with_n_init(1).with_init_centers(init).fit(x)
        assert g.n_iter() == steps
        assert np.array_equal(g.labels(), labels)
        assert np.array_equal(g.cluster_centers(), c, equal_nan=True)
    rows = np.random.default_rng(3).permutation(x.shape[0])[:4000]
    assert np.array_equal(labels[rows], O.predict(prev, x[rows].astype(np.float64)))
    return g.report["count_iterations"]


@pytest.mark.parametrize("precision", ["bf16", "fp8"])
@pytest.mark.parametrize("kind", [(320003, 128, 1000), (320011, 47, 1000), (160003, 250, 1025), (640001, 33, 512),
                                  (2300007, 65, 256), (180001, 64, 2801), "bisector"], ids=str)
def test_a_fit_that_pays_for_its_bounds_lists_rows(kind, precision):
    assert _check(kind, precision) == 0


@pytest.mark.parametrize("precision", ["bf16", "fp8"])
@pytest.mark.parametrize("kind", [
    (100003, 200, 4096),  # 24 rows a centre: the centres' distances cost more than the pass
    (170001, 250, 3001),  # 57
    (100003, 256, 1024),  # enough rows a centre, too small a product
    (600011, 128, 300),  # too few centres for its product
], ids=str)
def test_a_fit_that_does_not_pay_counts(kind, precision):
    assert _check(kind, precision) > 0


@pytest.mark.parametrize("precision", ["bf16", "fp8"])
def test_rows_and_a_centre_that_are_not_finite(precision):
    _check("nonfinite", precision)
