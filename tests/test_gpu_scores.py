"""Plain f32 labels through FMA scores: equal to the oracle's direct form at the
edges of the row tiles (128), of the feature slabs (32) and of the centre tiles
(16 per step, 128 per pass), for aligned and unaligned rows, on data with near
ties, ties, a common offset, outlying centres, non-finite, huge and tiny values."""
import numpy as np
import pytest
import torch

from ferrolearn_gb300.kmeans import FittedKMeans
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# n d k >= 2e8, d >= 16, k >= 24 take the scores; the last two lie just outside
SHAPES = [(520960, 16, 24), (170011, 37, 33), (65537, 32, 100), (66000, 31, 112), (24577, 64, 128), (25000, 65, 129),
          (4001, 200, 257), (800, 999, 300), (521000, 15, 26), (600000, 16, 23)]


def _case(kind, n, d, k, rng):
    c = rng.uniform(-10, 10, size=(k, d)).astype(np.float32)
    x = (c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d)) * 4).astype(np.float32)
    if kind == "offset":
        x += np.float32(3e4)
        c += np.float32(3e4)
    elif kind == "ties":
        x, c = np.round(x / 4).astype(np.float32), np.round(c / 4).astype(np.float32)
        c[k // 2] = c[1]
        x[::7] = c[1]
    elif kind == "outlier":
        c[3] = 1e6
        c[k - 1] *= np.float32(1e12)
    elif kind == "nonfinite":
        x[5, 3], x[n - 1, 0], x[77, 1] = np.nan, np.inf, 3e38
        c[2, 1], c[k - 2, 0] = np.nan, np.inf
    elif kind == "huge":
        x *= np.float32(1e17)
        c *= np.float32(1e17)
        x[::11] *= np.float32(50)
    elif kind == "tiny":
        x *= np.float32(1e-20)
        c *= np.float32(1e-20)
    return x, c


@pytest.mark.parametrize("kind", ["blobs", "offset", "ties", "outlier", "nonfinite", "huge", "tiny"])
def test_scored_labels(kind):
    rng = np.random.default_rng(21)
    for n, d, k in SHAPES if kind == "blobs" else SHAPES[1:6:2]:
        x, c = _case(kind, n, d, k, rng)
        model = FittedKMeans(c, None, 0.0, 0, "f32")
        want = O.predict(c, x)
        dev = torch.from_numpy(x).cuda()
        assert np.array_equal(np.asarray(model.predict(x)), want), (kind, n, d, k)
        got = model.predict(dev)
        got = got.cpu().numpy() if isinstance(got, torch.Tensor) else np.asarray(got)
        assert np.array_equal(got, want), (kind, n, d, k)
        # a view that starts off a 16-byte boundary
        flat = torch.empty(n * d + 1, device="cuda")
        flat[1:] = dev.reshape(-1)
        got = model.predict(flat[1:].reshape(n, d))
        got = got.cpu().numpy() if isinstance(got, torch.Tensor) else np.asarray(got)
        assert np.array_equal(got, want), (kind, n, d, k, "unaligned")
