"""Fits of the tensor-core forms large enough to keep row bounds: from the
fourth iteration on only the rows that the bounds do not keep are ranked.
Labels, centres and n_iter are the FP64 oracle's, and the centres bit for bit
those of single steps (which rank every row)."""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from ferrolearn_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _workload(kind):
    if kind == "anisotropic":  # the bounds keep most rows
        w = W.anisotropic_1024x128(scale=0.04)
        return w["x"], w["k"], w["init"]
    if kind == "bisector":  # a tenth of the rows stay equidistant: listed, paired, decided in FP64
        w = W.bisector_4096x256(scale=0.0035, k=1024, d=256, predict_scale=0.0001)
        x = np.concatenate([w["x"]] * 3)[:80003]
        x[28000:] += np.random.default_rng(1).normal(0, 0.3, size=x[28000:].shape).astype(np.float32)
        return x, w["k"], w["init"]
    if kind == "uniform":  # no structure: the bounds keep too few, the count pass runs
        x = np.random.default_rng(2).uniform(-1, 1, size=(600011, 33)).astype(np.float32)
        return x, 1100, x[:1100].astype(np.float64)
    w = W.anisotropic_1024x128(scale=0.04)  # rows and a centre that are not finite
    x = w["x"].copy()
    x[5, 3], x[77777, 0], x[100000, 127] = np.nan, np.inf, -np.inf
    return x, w["k"], w["init"]


@pytest.mark.parametrize("precision", ["bf16", "fp8"])
@pytest.mark.parametrize("kind", ["anisotropic", "bisector", "uniform", "nonfinite"])
def test_listed_rows_fit_matches_fp64_oracle_and_single_steps(kind, precision):
    x, k, init = _workload(kind)
    assert x.shape[0] * x.shape[1] * k >= 2e10  # the size from which the fit keeps bounds
    steps = 9
    c, labels = init, []
    for _ in range(steps):
        gl, c, _, _, _ = F.lloyd_step(x, c, dtype="f32x64", precision=precision)
        labels.append((gl, c))
    for it in (4, steps):
        g = F.KMeans(k, dtype="f32x64").with_precision(precision).with_max_iter(it).with_tol(0.0).with_n_init(1) \
            .with_init_centers(init).fit(x)
        assert np.array_equal(g.labels(), labels[it - 1][0])
        assert np.array_equal(g.cluster_centers(), labels[it - 1][1], equal_nan=True)
        assert g.n_iter() == it
    # the last assignment against the oracle, on a sample of the rows
    rows = np.random.default_rng(3).permutation(x.shape[0])[:20000]
    ol = O.predict(labels[steps - 2][1], x[rows].astype(np.float64))
    assert np.array_equal(labels[steps - 1][0][rows], ol)
