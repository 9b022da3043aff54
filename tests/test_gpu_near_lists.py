"""Plain fits with bounds at the edges of their lists of near centres (one, two or four
centres a block, one lane or eight a distance, ranks up to 256 centres and merged
parts above) and of the pass over every centre for few rows: labels and centres
bit-identical to the oracle's."""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from oracle import oracle as O
from test_gpu_prune import _case

pytestmark = pytest.mark.gpu

# one centre a block up to 607, two up to 1,215 (or k + d > 4,608), then four; 16-byte reads where
# d is a multiple of four, one lane a distance up to d = 16; 152 tiles of 128 rows and one more
SHAPES = [(16001, 250, 257), (30000, 64, 607), (33001, 52, 608), (60007, 17, 1215), (31000, 31, 1216),
          (60000, 16, 1217), (60001, 15, 1218), (115200, 8, 4601), (19456, 200, 300), (19457, 201, 300)]


@pytest.mark.parametrize("name", ["f32", "f64"])
@pytest.mark.parametrize("kind", ["blobs", "grid", "uniform", "nonfinite"])
@pytest.mark.parametrize("n,d,k", SHAPES)
def test_bounded_fit_matches_oracle(n, d, k, kind, name):
    assert n * k * d >= 1e9 and n >= 24 * k  # fits that keep bounds
    dt = np.float32 if name == "f32" else np.float64
    x, init = _case(kind, n, d, k, n + d)
    x, init = np.ascontiguousarray(x, dtype=dt), init.astype(dt)
    c = init
    for _ in range(3):  # the third is the first whose lists follow moved centres
        ol, c, _, _ = O.lloyd_step(x, c)
    g = F.KMeans(k, dtype=name).with_max_iter(3).with_tol(0.0).with_n_init(1).with_init_centers(init).fit(x)
    assert np.array_equal(g.labels(), ol)
    assert np.array_equal(g.cluster_centers(), c, equal_nan=True)
