"""Results of many megabytes into host arrays: the pieces that several threads
carry arrive whole, whatever the size's remainder."""
import threading

import numpy as np
import pytest

import ferrolearn_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [48960, 49003, 65537, 120001])
def test_transform_into_host_memory(n):
    rng = np.random.default_rng(n)
    x, c = rng.normal(size=(n, 5)).astype(np.float32), rng.normal(size=(257, 5)).astype(np.float32)
    model = F.FittedKMeans(c, None, 0.0, 0, "f32")
    want = O.transform(c, x)
    assert np.array_equal(model.transform(x), want)
    assert np.array_equal(model.transform(x), want)  # the pinned pieces again


def test_two_threads_carry_results_at_once():
    rng = np.random.default_rng(1)
    x, c = rng.normal(size=(200003, 4)).astype(np.float32), rng.normal(size=(64, 4)).astype(np.float32)
    want = O.transform(c, x)
    got = {}

    def work(i):
        model = F.FittedKMeans(c, None, 0.0, 0, "f32")
        got[i] = [model.transform(x) for _ in range(3)]  # a context a thread

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert all(np.array_equal(y, want) for v in got.values() for y in v) and len(got) == 2
