"""Captured iterations replayed on other data in the same buffer: every quantity
that depends on the rows is read on the device, none is kept in the capture.

Rows far from the origin widen the FP64 slack of the tensor-core forms' thresholds
by the norm of the rows' mean. It shows in how many rows are re-checked, long
before it could show in a label."""
import numpy as np
import pytest
import torch

import ferrolearn_gb300 as F

pytestmark = pytest.mark.gpu

COUNTS = ("rows_rechecked", "rows_full_rescan", "rows_fp64", "rows_few", "rows_exhaustive", "rows_moved",
          "count_iterations")


@pytest.mark.parametrize("precision", ["bf16", "fp8"])
@pytest.mark.parametrize("d", [32, 37])  # 37: the padded copy's buffer is the one that is used again
def test_replayed_iterations_take_the_new_rows(precision, d):
    rng = np.random.default_rng(d)
    n, k = 40000, 64
    c = rng.uniform(-1, 1, size=(k, d))
    near = np.round((c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d)) * 0.5) * 3).astype(np.float32)
    far = (near + 6e6).astype(np.float32)
    buf = torch.empty((n, d), device="cuda")

    def fit(x, ctx):
        buf.copy_(torch.from_numpy(x))
        torch.cuda.synchronize()
        m = F.KMeans(k, dtype="f32x64").with_precision(precision).with_max_iter(14).with_tol(0.0).with_n_init(1)
        return m.with_init_centers(x[:k].astype(np.float64)).fit(buf, ctx=ctx)

    ctx, fresh = F.Context(0), F.Context(0)
    fit(near, ctx)  # its buffers
    fit(near, ctx)  # captures its iterations
    got, want = fit(far, ctx), fit(far, fresh)
    assert {q: got.report[q] for q in COUNTS} == {q: want.report[q] for q in COUNTS}
    assert np.array_equal(got.labels(), want.labels())
    assert np.array_equal(got.cluster_centers(), want.cluster_centers()) and got.n_iter() == want.n_iter()
    ctx.close()
    fresh.close()
