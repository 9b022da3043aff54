"""Workloads of the K-Means family on one GPU, each one call of the public API.

Every case is one call that a user's program makes: a fit (plain FP32 / FP64,
BF16 and FP8 with exact re-check), a predict, a transform, a batch of
independent fits, a MiniBatchKMeans fit, a BisectingKMeans fit. Sizes and value
distributions are those of ferrolearn_gb300/workloads.py and of the tests, drawn
here on the GPU. Inputs of a large case are device tensors, those of a small one
numpy arrays, as a program that uses the library holds them; a fit on a device
tensor writes its results to device buffers.
"""
import math

import numpy as np
import torch

import ferrolearn_gb300 as F
from ferrolearn_gb300.kmeans import FittedKMeans

_TYPES = {"f64": (torch.float64, torch.float64), "f32": (torch.float32, torch.float32),
          "f32x64": (torch.float32, torch.float64)}


def listed():
    return [
        # one small scoring request: 1,000 rows from host memory against a fitted model
        dict(name="predict_f64_1k", kind="predict", dtype="f64", precision="plain", n=1000, d=16, k=8, host=True),
        # a notebook-sized fit with the estimator's defaults (k-means++, 10 restarts) on a numpy array
        dict(name="fit_f64_5k_defaults", kind="fit", dtype="f64", precision="plain", data="blobs", n=5000, d=20, k=8,
             init="kmeans++", n_init=10, max_iter=300, tol=1e-4, passes=2, host=True),
        # a plain FP32 fit at scale: k-means++, then 100 Lloyd iterations (not converged by then on this data).
        # passes: how many iterations the data takes (in the mean over restarts), for work()
        dict(name="fit_f32_1m", kind="fit", dtype="f32", precision="plain", data="dirichlet", n=1000000, d=64, k=256,
             init="kmeans++", n_init=1, max_iter=100, tol=1e-4, passes=100, host=False),
        # a plain FP64 fit at scale, with row count, feature count and k that fill no tile
        dict(name="fit_f64_333k", kind="fit", dtype="f64", precision="plain", data="dirichlet", n=333337, d=50, k=200,
             init="kmeans++", n_init=1, max_iter=100, tol=1e-4, passes=100, host=False),
        # the BF16 form: 4M rows, 1024 clusters, 20 iterations from given centres
        dict(name="fit_bf16_4m", kind="fit", dtype="f32x64", precision="bf16", data="anisotropic", n=4000000, d=128,
             k=1024, init="rows", n_init=1, max_iter=20, tol=0.0, passes=20, host=False),
        # the FP8 form: a vector-quantisation codebook of 4096 entries over 8M rows, 10% of them equidistant
        dict(name="fit_fp8_8m", kind="fit", dtype="f32x64", precision="fp8", data="bisector", n=8000000, d=256, k=4096,
             init="rows", n_init=1, max_iter=20, tol=0.0, passes=20, host=False),
        # encoding 2M fresh rows with that codebook
        dict(name="predict_fp8_2m", kind="predict", dtype="f32x64", precision="fp8", n=2000000, d=256, k=4096,
             host=False),
        # scoring a medium ragged block in plain FP32
        dict(name="predict_f32_200k", kind="predict", dtype="f32", precision="plain", n=200003, d=37, k=100,
             host=False),
        # distances to every centre as features for a later model
        dict(name="transform_f32_100k", kind="transform", dtype="f32", precision="plain", n=100000, d=64, k=256,
             host=False),
        # many independent uneven problems at once, 10 restarts each
        dict(name="batched_f32_64", kind="batched", problems=64, n_lo=2000, n_hi=200000, n_init=10, max_iter=300,
             tol=1e-4, reduction="f64", passes=9),
        # MiniBatchKMeans with its defaults (k-means++, 3 restarts, 100 batches of 1024)
        dict(name="minibatch_f64_1m", kind="minibatch", dtype="f64", n=1000000, d=64, k=256, batch=1024, n_init=3,
             max_iter=100),
        # BisectingKMeans with its defaults (10 restarts a split)
        dict(name="bisecting_f64_20k", kind="bisecting", dtype="f64", n=20000, d=16, k=16, n_init=10, max_iter=300,
             passes=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges; the upper ends keep it below the largest listed one."""
    kind = rng.choice(["fit", "fit", "mixed", "mixed", "predict", "predict", "transform", "batched", "minibatch",
                       "bisecting"])
    if kind == "fit":
        n, d = _log(rng, 1000, 1000000), rng.randint(2, 100)
        k = min(_log(rng, 4, 300), n // 50)
        it = rng.randint(10, 40)
        return dict(kind="fit", dtype=rng.choice(["f32", "f64"]), precision="plain",
                    data=rng.choice(["blobs", "dirichlet"]), n=n, d=d, k=k, init="kmeans++",
                    n_init=1 if n > 20000 else rng.choice([1, 3, 10]), max_iter=it, tol=0.0, passes=it,
                    host=n < 50000)
    if kind == "mixed":
        n, d, k = _log(rng, 100000, 4000000), rng.randint(48, 256), _log(rng, 256, 4096)
        it = rng.randint(10, 30)
        return dict(kind="fit", dtype="f32x64", precision=rng.choice(["bf16", "fp8"]),
                    data=rng.choice(["anisotropic", "bisector"]), n=n, d=d, k=k, init="rows", n_init=1, max_iter=it,
                    tol=0.0, passes=it, host=False)
    if kind == "predict":
        dtype, precision = rng.choice([("f64", "plain"), ("f32", "plain"), ("f32x64", "bf16"), ("f32x64", "fp8")])
        n = _log(rng, 100, 1000000) if precision == "plain" else _log(rng, 20000, 2000000)
        k = _log(rng, 4, 300) if precision == "plain" else _log(rng, 128, 4096)
        return dict(kind="predict", dtype=dtype, precision=precision, n=n, d=rng.randint(4, 256), k=k,
                    host=n < 20000)
    if kind == "transform":
        return dict(kind="transform", dtype=rng.choice(["f32", "f64"]), precision="plain", n=_log(rng, 100, 200000),
                    d=rng.randint(4, 128), k=_log(rng, 4, 256), host=False)
    if kind == "batched":
        return dict(kind="batched", problems=rng.randint(4, 64), n_lo=1000, n_hi=_log(rng, 10000, 100000),
                    n_init=rng.choice([1, 3, 10]), max_iter=300, tol=1e-4, reduction=rng.choice(["f64", "reference"]),
                    passes=12)
    if kind == "minibatch":
        return dict(kind="minibatch", dtype=rng.choice(["f32", "f64"]), n=_log(rng, 10000, 500000),
                    d=rng.randint(4, 100), k=_log(rng, 4, 200), batch=rng.choice([256, 1000, 1024, 4096]),
                    n_init=rng.choice([1, 3]), max_iter=rng.randint(20, 100))
    return dict(kind="bisecting", dtype=rng.choice(["f32", "f64"]), n=_log(rng, 500, 20000), d=rng.randint(2, 24),
                k=rng.randint(3, 16), n_init=rng.choice([1, 3, 10]), max_iter=300, passes=12)


# ---------------------------------------------------------------- inputs --

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _uniform(shape, lo, hi, g, dt=torch.float32):
    return torch.rand(shape, generator=g, device="cuda", dtype=dt) * (hi - lo) + lo


def _blobs(n, d, k, dt, g, half=10.0):
    """k equally likely isotropic blobs, std 1, centres U[-half, half]^d; (rows, centres)."""
    c = _uniform((k, d), -half, half, g, dt)
    lab = torch.randint(0, k, (n,), generator=g, device="cuda")
    return torch.randn((n, d), generator=g, device="cuda", dtype=dt).add_(c[lab]), c


def _dirichlet(n, d, k, dt, g):
    """k blobs of Dirichlet(1) sizes, std U[0.5, 3], centres U[-20, 20]^d."""
    c = _uniform((k, d), -20.0, 20.0, g, dt)
    std = _uniform((k,), 0.5, 3.0, g, dt)
    w = -torch.log(torch.rand((k,), generator=g, device="cuda", dtype=torch.float64).clamp_min_(1e-300))
    lab = torch.multinomial(w / w.sum(), n, replacement=True, generator=g)
    return torch.randn((n, d), generator=g, device="cuda", dtype=dt).mul_(std[lab][:, None]).add_(c[lab])


def _anisotropic(n, d, k, g):
    """k blobs with covariance A A^T, A ~ N(0, 0.3^2), centres U[-15, 15]^d, in random order."""
    c = _uniform((k, d), -15.0, 15.0, g)
    m = -(-n // k)
    x = torch.empty((k, m, d), device="cuda")
    for lo in range(0, k, 128):
        hi = min(k, lo + 128)
        a = torch.randn((hi - lo, d, d), generator=g, device="cuda") * 0.3
        z = torch.randn((hi - lo, m, d), generator=g, device="cuda")
        torch.baddbmm(c[lo:hi, None, :], z, a.transpose(1, 2), out=x[lo:hi])
    return x.view(k * m, d)[torch.randperm(k * m, generator=g, device="cuda")[:n]]


def _bisector(n, d, k, g):
    """k unit blobs with centres U[-30, 30]^d; a tenth of the rows lie on the perpendicular bisector of two of
    the centres. (rows, centres)"""
    c = _uniform((k, d), -30.0, 30.0, g)
    lab = torch.randint(0, k, (n,), generator=g, device="cuda")
    other = (lab + 1 + torch.randint(0, max(1, k - 1), (n,), generator=g, device="cuda")) % k
    tie = torch.rand((n,), generator=g, device="cuda") < 0.1
    x = torch.empty((n, d), device="cuda")
    for lo in range(0, n, 1 << 20):
        s = slice(lo, min(n, lo + (1 << 20)))
        u = torch.randn((x[s].shape[0], d), generator=g, device="cuda")
        x[s] = u + c[lab[s]]
        at = tie[s].nonzero()[:, 0]
        a, b, v = c[lab[s][at]].double(), c[other[s][at]].double(), u[at].double()
        w = b - a
        v -= ((v * w).sum(1) / (w * w).sum(1).clamp_min(1e-30))[:, None] * w
        x[lo + at] = (0.5 * (a + b) + v).float()
    return x, c


def _rows(case, seed):
    g = _gen(seed)
    n, d, k = case["n"], case["d"], case["k"]
    dt = _TYPES[case["dtype"]][0]
    data = case.get("data", "blobs")
    if data == "blobs":
        return _blobs(n, d, k, dt, g)[0]
    if data == "dirichlet":
        return _dirichlet(n, d, k, dt, g)
    return _anisotropic(n, d, k, g) if data == "anisotropic" else _bisector(n, d, k, g)[0]


def _start_rows(x, k, seed):
    """k rows of a seeded permutation, as the initial centres."""
    return x[torch.randperm(x.shape[0], generator=_gen(seed + 1000003), device="cuda")[:k]].double().cpu().numpy()


def _model(case, seed):
    """Rows and the centres of a fitted model for predict and transform."""
    g = _gen(seed)
    dt, ct = _TYPES[case["dtype"]]
    if case["precision"] == "plain":
        x, c = _blobs(case["n"], case["d"], case["k"], dt, g)
    else:
        x, c = _bisector(case["n"], case["d"], case["k"], g)
    return x, c.to(ct) + 0.01 * torch.randn(c.shape, generator=g, device="cuda", dtype=ct)


def _problem(case, p):
    """Sizes of problem p: n spread over the logarithm of its range, d and k in turn."""
    n = int(round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** ((p + 0.5) / case["problems"])))
    return n, (8, 16, 32, 64)[p % 4], 4 + (p * 37) % 61


def _problems(case, seed):
    g = _gen(seed)
    got = []
    for p in range(case["problems"]):
        n, d, k = _problem(case, p)
        got.append(dict(x=_blobs(n, d, k, torch.float32, g)[0], k=k, n_init=case["n_init"],
                        max_iter=case["max_iter"], tol=case["tol"], random_state=seed * 1000 + p))
    return got


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batched":
        return dict(kind=kind, problems=_problems(case, seed), reduction=case["reduction"])
    if kind in ("predict", "transform"):
        x, c = _model(case, seed)
        model = FittedKMeans(c.cpu().numpy(), None, 0.0, 0, case["dtype"],
                             precision=F.KMeans(1).with_precision(case["precision"]).precision)
        return dict(kind=kind, x=x.cpu().numpy() if case["host"] else x, model=model)
    if kind == "minibatch":
        x = _dirichlet(case["n"], case["d"], case["k"], _TYPES[case["dtype"]][0], _gen(seed))
        est = F.MiniBatchKMeans(case["k"], case["dtype"]).with_batch_size(case["batch"]) \
            .with_n_init(case["n_init"]).with_max_iter(case["max_iter"]).with_random_state(seed)
        return dict(kind=kind, x=x, est=est, out=_buffers(case))
    if kind == "bisecting":
        x = _blobs(case["n"], case["d"], case["k"], _TYPES[case["dtype"]][0], _gen(seed), half=20.0)[0]
        est = F.BisectingKMeans(case["k"], case["dtype"]).with_n_init(case["n_init"]) \
            .with_max_iter(case["max_iter"]).with_random_state(seed)
        return dict(kind=kind, x=x.cpu().numpy(), est=est)
    x = _rows(case, seed)
    est = F.KMeans(case["k"], case["dtype"]).with_n_init(case["n_init"]).with_max_iter(case["max_iter"]) \
        .with_tol(case["tol"]).with_random_state(seed).with_precision(case["precision"])
    if case["init"] == "rows":
        est.with_init_centers(_start_rows(x, case["k"], seed))
    if case["host"]:
        return dict(kind=kind, x=x.cpu().numpy(), est=est, out=None)
    return dict(kind=kind, x=x, est=est, out=_buffers(case))


def _buffers(case):
    return (torch.empty((case["k"], case["d"]), dtype=_TYPES[case["dtype"]][1], device="cuda"),
            torch.empty((case["n"],), dtype=torch.int64, device="cuda"))


# ------------------------------------------------------------------- run --

def run(state):
    kind = state["kind"]
    if kind == "predict":
        return state["model"].predict(state["x"])
    if kind == "transform":
        return state["model"].transform(state["x"])
    if kind == "batched":
        fitted, _ = F.fit_batched(state["problems"], reduction=state["reduction"])
        return dict(centers=np.concatenate([f.cluster_centers().ravel() for f in fitted]),
                    labels=np.concatenate([f.labels() for f in fitted]),
                    inertia=np.array([f.inertia() for f in fitted], dtype=np.float32),
                    n_iter=np.array([f.n_iter() for f in fitted]))
    if kind == "bisecting":
        f = state["est"].fit(state["x"])
        return dict(centers=f.cluster_centers(), labels=f.labels(), inertia=f.inertia())
    f = state["est"].fit(state["x"], out=state["out"])
    return dict(centers=f.cluster_centers(), labels=f.labels(), inertia=f.inertia(), n_iter=f.n_iter())


# ------------------------------------------------------------------ work --

def _seeding(n, d, k, size):
    """k-means++: per centre the rows read once, 2 + ln k trials' direct-form distances."""
    t = 2 + int(math.log(k)) if k > 1 else 1
    return (k - 1) * (n * d * size + 2 * n * size), (k - 1) * 3.0 * t * n * d


def work(case):
    kind = case["kind"]
    if kind == "batched":
        b = f = 0.0
        for p in range(case["problems"]):
            n, d, k = _problem(case, p)
            sb, sf = _seeding(n, d, k, 4)
            runs = case["n_init"]
            # the restarts of a problem can share each read of its rows
            b += n * d * 4 + n * 8 + k * d * 4
            f += runs * (sf + case["passes"] * (2.0 * n * k * d + n * d))
        return {"bytes": b, "flops": f}
    n, d, k = case["n"], case["d"], case["k"]
    size = 4 if case["dtype"].startswith("f32") else 8
    csize = 4 if case["dtype"] == "f32" else 8
    if kind == "predict":
        return {"bytes": n * d * size + k * d * csize + 8 * n, "flops": 2.0 * n * k * d}
    if kind == "transform":
        return {"bytes": n * d * size + k * d * csize + n * k * csize, "flops": 3.0 * n * k * d}
    if kind == "minibatch":
        sb, sf = _seeding(n, d, k, size)
        it = case["max_iter"] * min(case["batch"], n)
        return {"bytes": case["n_init"] * (sb + it * d * size + n * d * size) + 8 * n,
                "flops": case["n_init"] * (sf + 2.0 * (it + n) * k * d)}
    if kind == "bisecting":
        # a balanced tree of splits: every level holds all rows once
        levels = math.ceil(math.log2(max(2, k)))
        one = levels * case["passes"] * case["n_init"]
        return {"bytes": n * d * size + 8 * n, "flops": one * 7.0 * n * d}
    sb, sf = _seeding(n, d, k, size) if case["init"] == "kmeans++" else (0, 0)
    one_b, one_f = n * d * size + 4 * n, 2.0 * n * k * d + n * d
    return {"bytes": case["n_init"] * (sb + case["passes"] * one_b) + 8 * n + k * d * csize,
            "flops": case["n_init"] * (sf + case["passes"] * one_f)}


# ----------------------------------------------------------------- exact --

def _draws(seed, count, pos=0):
    """The estimators' uniform stream: splitmix64, 53 bits a draw."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * (np.arange(1, count + 1, dtype=np.uint64) + np.uint64(pos))
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    return (z >> np.uint64(11)).astype(np.float64) / 9007199254740992.0


def _sq(x, c):
    """Squared distances of x's rows to c's, in 64 bits."""
    return (x.square().sum(1)[:, None] + c.square().sum(1)[None, :] - 2.0 * (x @ c.T)).clamp_min_(0.0)


def _seeds64(x, k, seed):
    """Greedy k-means++ in 64 bits; (centres, draws used)."""
    n = x.shape[0]
    trials = max(1, 2 + int(math.floor(math.log(k))))
    u = _draws(seed, 1 + (k - 1) * trials)
    at = [min(int(u[0] * n), n - 1)]
    near = (x - x[at[0]]).square_().sum(1)
    for c in range(1, k):
        cum = torch.cumsum(near, 0)
        thr = torch.from_numpy(u[1 + (c - 1) * trials:1 + c * trials]).cuda() * cum[-1]
        cand = torch.searchsorted(cum, thr).clamp_max_(n - 1)
        d2 = torch.minimum(_sq(x, x[cand]), near[:, None])
        d2[cand, torch.arange(trials, device="cuda")] = 0.0
        best = int(torch.argmin(d2.sum(0)))
        at.append(int(cand[best]))
        near = d2[:, best].contiguous()
    return x[torch.tensor(at, device="cuda")].clone(), 1 + (k - 1) * trials


def _nearest64(x, c, wide):
    """(labels, squared distances in 64 bits). wide: the two nearest centres are found in 32 bits first."""
    lab = torch.empty((x.shape[0],), dtype=torch.int64, device="cuda")
    d2 = torch.empty((x.shape[0],), dtype=torch.float64, device="cuda")
    step = max(1024, (1 << 28) // max(c.shape[0], x.shape[1]))
    for lo in range(0, x.shape[0], step):
        s = slice(lo, min(x.shape[0], lo + step))
        if wide:
            c32 = c.float()
            score = c32.square().sum(1)[None, :] - 2.0 * (x[s].float() @ c32.T)
            two = [score.argmin(1)]
            score.scatter_(1, two[0][:, None], math.inf)
            two.append(score.argmin(1))
            e = torch.stack([(x[s].double() - c[q]).square_().sum(1) for q in two], 1)
            v, w = e.min(1)
            lab[s], d2[s] = torch.where(w == 0, two[0], two[1]), v
        else:
            lab[s] = _sq(x[s].double(), c).argmin(1)
            d2[s] = (x[s].double() - c[lab[s]]).square_().sum(1)
    return lab, d2


def _lloyd64(x, c, max_iter, tol, wide):
    k = c.shape[0]
    for it in range(max_iter):
        lab, d2 = _nearest64(x, c, wide)
        sums = torch.zeros_like(c)
        for lo in range(0, x.shape[0], 1 << 20):
            sums.index_add_(0, lab[lo:lo + (1 << 20)], x[lo:lo + (1 << 20)].double())
        m = torch.bincount(lab, minlength=k)[:, None]
        new = torch.where(m > 0, sums / m.clamp_min(1), c)
        shift = float((new - c).square().sum(1).max().sqrt())
        c = new
        if shift < tol:
            break
    return c, float(d2.sum()), it + 1


def _exact_minibatch(x, case, seed):
    n, k, m = case["n"], case["k"], min(case["batch"], case["n"])
    best = None
    for r in range(case["n_init"]):
        run_seed = seed + r * 1000003
        c, pos = _seeds64(x, k, run_seed)
        counts = torch.ones((k,), dtype=torch.float64, device="cuda")
        for _ in range(case["max_iter"]):
            u, pool, pick = _draws(run_seed, m, pos), {}, []
            pos += m
            for i in range(m):
                j = i + min(int(u[i] * (n - i)), n - i - 1)
                pick.append(pool.get(j, j))
                pool[j] = pool.get(i, i)
            rows = x[torch.tensor(pick, device="cuda")]
            lab = _sq(rows, c).argmin(1)
            got = torch.bincount(lab, minlength=k).double()
            sums = torch.zeros_like(c).index_add_(0, lab, rows)
            c = (c * counts[:, None] + sums) / (counts + got)[:, None]
            counts += got
        inertia = float(_nearest64(x, c, False)[1].sum())
        if best is None or inertia < best[1]:
            best = (c, inertia)
    return best


def _exact_bisecting(x, case, seed):
    def two_means(v, run_seed):
        u, p = _draws(run_seed, 64), 1
        i0 = min(int(u[0] * len(v)), len(v) - 1)
        i1 = min(int(u[1] * len(v)), len(v) - 1)
        while len(v) > 1 and i1 == i0:
            p += 1
            i1 = min(int(u[p] * len(v)), len(v) - 1)
        c, lab = np.stack([v[i0], v[i1]]), np.zeros(len(v), dtype=bool)
        for _ in range(case["max_iter"]):
            new = ~(((v - c[0]) ** 2).sum(1) <= ((v - c[1]) ** 2).sum(1))
            if np.array_equal(new, lab):
                break
            lab = new
            c = np.stack([v[lab == s].mean(0) if (lab == s).any() else c[s] for s in (0, 1)])
        return ((v - c[lab.astype(int)]) ** 2).sum(), lab, c

    parts = [(np.arange(len(x)), x.mean(0), ((x - x.mean(0)) ** 2).sum())]
    splits = 0
    while len(parts) < case["k"] and splits < 4 * case["k"]:
        t = max((i for i in range(len(parts)) if len(parts[i][0]) > 1), key=lambda i: (len(parts[i][0]), i))
        at = parts.pop(t)[0]
        _, lab, c = min((two_means(x[at], seed + splits * 1000 + r) for r in range(case["n_init"])),
                        key=lambda b: b[0])
        splits += 1
        for s in (0, 1):
            rows = at[lab == s]
            if len(rows):
                parts.append((rows, c[s], ((x[rows] - c[s]) ** 2).sum()))
    return np.stack([p[1] for p in parts]), float(sum(p[2] for p in parts))


def exact(case, seed):
    """In 64 bits, where the result is a function of the inputs alone. A fit in 32 bits that starts from k-means++
    has none: its seeding picks rows by 32-bit running sums. The equidistant rows of the bisector data have none
    either: rounding decides them, and with them the centres."""
    kind = case["kind"]
    if kind in ("predict", "batched"):
        return None
    if kind == "transform":
        x, c = _model(case, seed)
        x, c = x.double(), c.double()
        out = torch.empty((case["n"], case["k"]), dtype=torch.float64, device="cuda")
        for q in range(case["k"]):
            out[:, q] = (x - c[q]).square_().sum(1).sqrt_()
        return out.cpu().numpy()
    if kind == "minibatch":
        if case["dtype"] != "f64":
            return None
        c, inertia = _exact_minibatch(prepare(case, seed)["x"], case, seed)
        return dict(centers=c, labels=None, inertia=inertia, n_iter=None)
    if kind == "bisecting":
        if case["dtype"] != "f64":
            return None
        c, inertia = _exact_bisecting(prepare(case, seed)["x"], case, seed)
        return dict(centers=c, labels=None, inertia=inertia)
    if case["data"] == "bisector" or (case["dtype"] == "f32" and case["init"] == "kmeans++"):
        return None
    x = _rows(case, seed)
    wide = 1.0 * case["n"] * case["k"] * case["d"] * case["passes"] > 2e12
    best = None
    for r in range(case["n_init"]):
        if case["init"] == "rows":
            c = torch.from_numpy(_start_rows(x, case["k"], seed)).cuda()
        else:
            c = _seeds64(x, case["k"], seed + r)[0]
        got = _lloyd64(x, c, case["max_iter"], case["tol"], wide)
        if best is None or got[1] < best[1]:
            best = got
    centers = best[0].cpu().numpy() if case["host"] else best[0]
    return dict(centers=centers, labels=None, inertia=best[1], n_iter=None)
