"""Rows that the f32 scores leave open: a CTA a row while the list is short, a warp a
row when it is long. The direct form's labels on both sides of the line, with
centres and features at the edges of the lane groups."""
import numpy as np
import pytest
import torch

import ferrolearn_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,k", [(32, 224), (33, 257), (40, 129), (145, 31), (99, 64), (16, 1000)])
def test_open_rows_have_the_direct_forms_labels(d, k):
    n = 400001 if d * k < 12500 else 40003
    line = 2 * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(d * k)
    c = rng.uniform(-8, 8, size=(k, d)).astype(np.float32)
    x = (c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d)) * 0.01).astype(np.float32)
    model = F.FittedKMeans(c, None, 0.0, 0, "f32")
    for m in (0, 1, line, line + 1, 5 * line):  # rows half way between two centres, in no order
        rows = rng.permutation(n)[:m]
        a, b = rng.integers(0, k, size=m), rng.integers(0, k, size=m)
        y = x.copy()
        y[rows] = (c[a] + c[b]) / 2
        if m > 4:
            y[rows[:3], 1] = [np.nan, np.inf, 3e38]
        got = model.predict(torch.from_numpy(y).cuda())
        got = got.cpu().numpy() if isinstance(got, torch.Tensor) else np.asarray(got)
        assert np.array_equal(got, O.predict(c, y)), (m, d, k)
