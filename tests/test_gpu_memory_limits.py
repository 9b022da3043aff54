"""Calls at the limit of device memory. The faster forms take buffers that a call can
do without (padded rows, row bounds, joint seedings, lists): where these leave no
room for what it needs, the call runs without them, with the same results, and
nothing an earlier call left in the context keeps it from running."""
import ctypes as C

import numpy as np
import pytest
import torch

import ferrolearn_gb300 as F
from ferrolearn_gb300 import _native
from ferrolearn_gb300.kmeans import DeviceOutOfMemory, FittedKMeans, InvalidParameter

pytestmark = pytest.mark.gpu


def _held(ctx, limit=0):
    held = C.c_uint64()
    assert _native.lib().fk_debug_memory(ctx.handle, int(limit), C.byref(held)) == 0
    return held.value


def _rows(n, d, k, dt, seed=0):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-10, 10, size=(k, d))
    x = (c[rng.integers(0, k, size=n)] + rng.normal(size=(n, d)) * 2).astype(dt)
    return x, c


def _fit(dtype, n, d, k, precision="plain", **with_):
    x, c = _rows(n, d, k, np.float64 if dtype == "f64" else np.float32)
    dev = torch.from_numpy(x).cuda()

    def call(ctx):
        m = F.KMeans(k, dtype=dtype).with_precision(precision).with_max_iter(8).with_tol(0.0)
        m.with_n_init(with_.get("n_init", 1)).with_random_state(3)
        if "n_init" not in with_:
            m.with_init_centers(x[:k].astype(np.float32 if dtype == "f32" else np.float64))
        f = m.fit(dev, ctx=ctx)
        return f.labels(), f.cluster_centers(), f.n_iter()
    return call


def _predict(dtype, n, d, k, precision="plain"):
    x, c = _rows(n, d, k, np.float64 if dtype == "f64" else np.float32)
    model = FittedKMeans(c.astype(np.float32 if dtype == "f32" else np.float64), None, 0.0, 0, dtype,
                         precision=F.KMeans(1).with_precision(precision).precision)
    dev = torch.from_numpy(x).cuda()
    return lambda ctx: (model.predict(dev, ctx=ctx),)


def _minibatch():
    x, _ = _rows(100000, 8, 50, np.float64)
    dev = torch.from_numpy(x).cuda()
    est = F.MiniBatchKMeans(50, "f64").with_batch_size(512).with_n_init(3).with_max_iter(5).with_random_state(1)

    def call(ctx):
        f = est.fit(dev, ctx=ctx)
        return f.labels(), f.cluster_centers()
    return call


def _bisecting():
    x, _ = _rows(50000, 32, 4, np.float64)
    est = F.BisectingKMeans(3, "f64").with_n_init(10).with_max_iter(5).with_random_state(1)

    def call(ctx):
        f = est.fit(x, ctx=ctx)
        return f.labels(), f.cluster_centers()
    return call


# The share of what the faster form takes that is left: too little for it (its buffers without
# their headroom are 8/9), enough for the others. Padded rows are 42% of a ragged fit's buffers,
# bounds and row lists 40% of a plain f32 fit's, ten seedings two thirds of a small f64 fit's, the
# open rows' list a quarter of a scored predict's, the folds' maps a sixth of a bisection's.
CASES = {
    "ragged bf16 fit": (lambda: _fit("f32x64", 200000, 127, 64, "bf16"), 0.75),
    "ragged fp8 fit": (lambda: _fit("f32x64", 150000, 125, 64, "fp8"), 0.78),
    "ragged bf16 predict": (lambda: _predict("f32x64", 200000, 127, 64, "bf16"), 0.75),
    "bounded bf16 fit": (lambda: _fit("f32x64", 320000, 128, 1024, "bf16"), 0.75),
    "bounded f32 fit": (lambda: _fit("f32", 400000, 16, 256), 0.75),
    "bounded f64 fit": (lambda: _fit("f64", 400000, 16, 256), 0.80),
    "seeded f64 fit": (lambda: _fit("f64", 20000, 8, 20, n_init=10), 0.50),
    "scored f32 predict": (lambda: _predict("f32", 170011, 37, 33), 0.80),
    "minibatch": (_minibatch, 0.60),
    "bisecting": (_bisecting, 0.82),
}


@pytest.mark.parametrize("name", list(CASES))
def test_a_call_runs_without_what_it_can_spare(name):
    make, share = CASES[name]
    call = make()
    roomy, tight = F.Context(0), F.Context(0)
    want = call(roomy)
    full = _held(roomy)
    _held(tight, full * share)
    got = call(tight)
    assert _held(tight, full * share) <= full * share
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
    again = call(tight)
    for g, w in zip(again, want):
        assert np.array_equal(g, w)
    roomy.close()
    tight.close()


def test_buffers_of_an_earlier_call_make_room():
    ctx = F.Context(0)
    _fit("f32x64", 200000, 127, 64, "bf16")(ctx)
    held = _held(ctx)
    x, c = _rows(60000, 64, 512, np.float32)
    model = FittedKMeans(c.astype(np.float32), None, 0.0, 0, "f32")
    want = model.transform(x)
    _held(ctx, held * 1.02)  # the result alone is 120 MB, the fit left 240
    assert np.array_equal(model.transform(x, ctx=ctx), want)
    assert _held(ctx) < held
    ctx.close()


def test_seedings_workspace_makes_room():
    ctx = F.Context(0)
    x, _ = _rows(40000, 8, 20, np.float64)
    F.KMeans(20).with_n_init(10).with_max_iter(2).fit(x, ctx=ctx)
    held = _held(ctx, _held(ctx) * 1.01)
    y, c = _rows(60000, 16, 10, np.float64)
    model = FittedKMeans(c, None, 0.0, 0, "f64")
    assert np.array_equal(model.predict(y, ctx=ctx), model.predict(y))
    assert _held(ctx) < held
    ctx.close()


def test_what_cannot_fit_is_refused_and_the_context_lives_on():
    ctx = F.Context(0)
    _held(ctx, 1 << 20)
    with pytest.raises(DeviceOutOfMemory):
        _fit("f32x64", 200000, 127, 64, "bf16")(ctx)
    _held(ctx, 0)
    small = _fit("f64", 1000, 4, 3)
    other = F.Context(0)
    for g, w in zip(small(ctx), small(other)):
        assert np.array_equal(g, w)
    with pytest.raises(InvalidParameter):
        F.KMeans(0).fit(np.zeros((2, 2)), ctx=ctx)
    ctx.close()
    other.close()


def test_centres_read_and_written_in_place():
    # one buffer as initial centres and result: the second attempt must start from the first values
    n, d, k = 200000, 127, 64
    x, c = _rows(n, d, k, np.float32)
    dev = torch.from_numpy(x).cuda()
    lib = _native.lib()

    def fit(ctx, buf):
        params = F.KMeans(k, dtype="f32x64").with_precision("bf16").with_max_iter(4).with_tol(0.0).with_n_init(1)._params()
        labels = np.empty(n, dtype=np.uint64)
        inertia, n_iter = C.c_double(), C.c_int64()
        st = lib.fk_kmeans_fit_f32x64(ctx.handle, C.c_void_p(dev.data_ptr()), n, d, C.byref(params),
                                      C.c_void_p(buf.data_ptr()), C.c_void_p(buf.data_ptr()),
                                      labels.ctypes.data_as(C.c_void_p), C.byref(inertia), C.byref(n_iter), None)
        assert st == 0
        return labels, buf.cpu().numpy()
    start = x[:k].astype(np.float64)
    roomy = F.Context(0)
    want = fit(roomy, torch.from_numpy(start).cuda())
    full = _held(roomy)
    for share in (0.7, 0.74, 0.78, 0.82, 0.86):  # out of room at different buffers
        tight = F.Context(0)
        _held(tight, full * share)
        got = fit(tight, torch.from_numpy(start).cuda())
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        tight.close()
    roomy.close()
