"""Plain fits whose bounds keep few rows go on without them and try again: labels,
centres and inertia equal to the oracle's through several rests, and where the
rows settle after one."""
import numpy as np
import pytest

import ferrolearn_gb300 as F
from ferrolearn_gb300 import _native
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rows(kind, n, d, k, dt):
    rng = np.random.default_rng(n)
    if kind == "uniform":
        return rng.uniform(size=(n, d)).astype(dt)
    c = rng.uniform(-10, 10, size=(k, d))
    return (c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d)) * (6 if kind == "wide" else 0.5)).astype(dt)


@pytest.mark.parametrize("name", ["f32", "f64"])
@pytest.mark.parametrize("n,d,k,n_init", [(20000, 64, 1000, 1), (26000, 32, 1300, 2), (20001, 101, 500, 1)])
def test_resting_fit_matches_oracle(n, d, k, n_init, name):
    dt = np.float32 if name == "f32" else np.float64
    launches = {}
    for kind in ("uniform", "wide", "tight"):
        x = _rows(kind, n, d, k, dt)
        init = np.stack([x[np.random.default_rng(r).permutation(n)[:k]] for r in range(n_init)])
        ctx = F.Context(0)
        for it in (5, 8, 18):  # before, in and after a rest; graphs of every pass replayed
            before = _native.lib().fk_debug_launch_count()
            g = F.KMeans(k, dtype=name).with_max_iter(it).with_tol(0.0).with_n_init(n_init).with_init_centers(init) \
                .fit(x, ctx=ctx)
            launches[kind] = _native.lib().fk_debug_launch_count() - before
            o = O.fit(x, k, max_iter=it, tol=0.0, n_init=n_init, init=init)
            assert np.array_equal(g.labels(), o["labels"]), (kind, it)
            assert np.array_equal(g.cluster_centers(), o["centers"]), (kind, it)
            assert abs(g.inertia() - o["inertia"]) <= (1e-5 if dt == np.float32 else 1e-12) * o["inertia"]
        ctx.close()
    # (a bounded iteration launches more kernels than one without bounds)
    assert launches["uniform"] < launches["tight"]
