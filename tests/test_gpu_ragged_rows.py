"""Mixed forms on rows that 16-byte reads do not fit (a feature count that is no
multiple of four, a start off a 16-byte boundary): every iteration's labels equal
to the FP64 oracle's direct form, centres to its exact sums, and the same fit as
on the same rows with zero features behind them."""
import numpy as np
import pytest
import torch

import ferrolearn_gb300 as F
from ferrolearn_gb300.kmeans import FittedKMeans
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["bf16", "fp8"])
@pytest.mark.parametrize("n,d,k", [(20000, 49, 64), (30011, 127, 300), (12000, 253, 500), (9000, 255, 130),
                                   (7000, 250, 130), (15000, 64, 100)])
def test_ragged_fit_and_predict(n, d, k, prec):
    rng = np.random.default_rng(n + d)
    c = rng.uniform(-10, 10, size=(k, d))
    x = (c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d)) * 3).astype(np.float32)
    x[5::101] = ((c[0] + c[1]) / 2).astype(np.float32)  # near ties
    init = x[rng.choice(n, size=k, replace=False)].astype(np.float64)

    def fit(rows, start):
        m = F.KMeans(k, dtype="f32x64").with_init_centers(start).with_precision(prec).with_max_iter(6).with_tol(0.0)
        return m.with_n_init(1).fit(rows)

    flat = torch.empty(n * d + 1, device="cuda")
    flat[1:] = torch.from_numpy(x).cuda().reshape(-1)
    off = flat[1:].reshape(n, d)  # never on a 16-byte boundary
    g = fit(off, init)
    pad = (-d) % 4
    wide = np.concatenate([x, np.zeros((n, pad), np.float32)], axis=1)
    w = fit(wide, np.concatenate([init, np.zeros((k, pad))], axis=1))
    assert np.array_equal(g.labels(), w.labels())
    assert np.array_equal(g.cluster_centers(), w.cluster_centers()[:, :d])
    assert g.n_iter() == w.n_iter() and abs(g.inertia() - w.inertia()) <= 1e-6 * w.inertia()
    o = O.fit(x.astype(np.float64), k, max_iter=6, tol=0.0, n_init=1, init=init[None])
    assert np.array_equal(g.labels(), o["labels"])
    assert np.allclose(g.cluster_centers(), o["centers"], rtol=1e-13, atol=1e-13)
    model = FittedKMeans(g.cluster_centers(), None, 0.0, 0, "f32x64", precision=g.precision)
    assert np.array_equal(model.predict(off), O.predict(g.cluster_centers(), x.astype(np.float64)))
