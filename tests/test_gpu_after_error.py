"""A call that CUDA refuses leaves nothing behind: the next one runs."""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from ferrolearn_gb300.kmeans import CudaError
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_the_call_after_a_refused_one_runs():
    rng = np.random.default_rng(0)
    x = rng.normal(size=(60000, 2)).astype(np.float32)
    many = F.KMeans(60000, dtype="f32").with_init_centers(x).with_n_init(1).with_max_iter(1)
    with pytest.raises(CudaError):  # the sort's counters of 60,000 clusters exceed a block's shared memory
        many.fit(x)
    few = F.KMeans(5, dtype="f32").with_init_centers(x[:5]).with_n_init(1).with_max_iter(3).with_tol(0.0).fit(x)
    o = O.fit(x, 5, max_iter=3, tol=0.0, n_init=1, init=x[:5][None])
    assert np.array_equal(few.labels(), o["labels"]) and np.array_equal(few.cluster_centers(), o["centers"])
