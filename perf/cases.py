"""Performance cases of the k-means engine: the calls a user's program makes.

Eight kinds of call, all through the public entry points:

  driver     ``kmeans_lloyd_driver`` (float32 / float64 plain form, float32
             tensor-core forms), the whole fit of a feature-major X_t
  step       one Lloyd step put together from the module's functions, as a
             program with a loop of its own does
  predict    ``half_l2_norm_squared`` + ``assignment``
  transform  ``compute_centroid_to_sample_distances``
  estimator  ``KMeans(...).fit`` on row-major samples: transposition,
             k-means++ seeding, tolerance scaling and the fit
  batch      ``kmc_batch_*``: many uneven plain fits advanced together
  server     ``kmc_server_*``: fits submitted together, then predictions
             against their models

Data are Gaussian blobs (equal sizes, shuffled).  Plain fits have separated
blobs and start from random rows of X, as in the benchmark; tensor-core fits
have overlapping blobs and start near their centres, as after a fit of a small
sample (starting from random rows, blobs split in many equivalent ways and the
float32 sums' order alone decides which).  Fits run a fixed number of
iterations (tol = 0) so that every pass does the same work; the estimator
keeps its tolerance.
"""
import ctypes
import math
import random

import numpy as np
import torch

import kmeans_dpcpp_gb300 as kdp
from kmeans_dpcpp_gb300 import KMeans, capi

DTYPES = {"f32": torch.float32, "f64": torch.float64, "i32": torch.int32, "i64": torch.int64}
FORMS = {"plain": 0, "mixed-bf16": 1, "mixed-fp16": 2}


def listed():
    return [
        # the smallest fit of the benchmark: launches and host round trips count
        dict(name="lloyd_f32_small", kind="driver", form="plain", dtype="f32", labels="i32", n=50_000, d=14,
             k=16, iters=20, weights="unit", far=False),
        # the ordinary exact fit, a far centroid that forces one relocation
        dict(name="lloyd_f32", kind="driver", form="plain", dtype="f32", labels="i32", n=5_000_000, d=14,
             k=127, iters=10, weights="unit", far=True),
        # the same in float64, the type NumPy data come in
        dict(name="lloyd_f64", kind="driver", form="plain", dtype="f64", labels="i32", n=2_000_000, d=14,
             k=127, iters=5, weights="unit", far=True),
        # the headline fit: large n, many clusters, tensor-core form
        dict(name="lloyd_fp16_large", kind="driver", form="mixed-fp16", dtype="f32", labels="i32",
             n=10_000_000, d=64, k=1024, iters=8, weights="unit", far=False, apart=0.7),
        # few features, weighted samples, 64-bit labels, odd sizes
        dict(name="lloyd_fp16_narrow", kind="driver", form="mixed-fp16", dtype="f32", labels="i64",
             n=1_000_001, d=16, k=100, iters=20, weights="random", far=False),
        # many features (two 64-feature blocks, ragged), bf16 operands
        dict(name="lloyd_bf16_wide", kind="driver", form="mixed-bf16", dtype="f32", labels="i32",
             n=300_007, d=100, k=500, iters=6, weights="unit", far=False),
        # one Lloyd step from the module's functions, with the private copies
        # that compute_number_of_private_copies asks for
        dict(name="step_f32", kind="step", dtype="f32", labels="i32", n=1_000_000, d=32, k=256,
             weights="random"),
        # labels of new samples against a fitted model
        dict(name="predict_f32", kind="predict", dtype="f32", labels="i32", n=1_000_003, d=64, k=512),
        # distances of new samples to a fitted model's centroids
        dict(name="transform_f32", kind="transform", dtype="f32", n=400_003, d=30, k=250),
        # scikit-learn-style use: row-major samples, k-means++, scaled tolerance
        dict(name="estimator_f32", kind="estimator", form="plain", dtype="f32", n=200_003, d=32, k=64,
             iters=20),
        # uneven independent fits through the batched engine
        dict(name="batch_f32", kind="batch", count=24, lot=4, n_lo=2_000, n_hi=500_000, k_lo=4, k_hi=512,
             iters=10),
        # a small burst of requests: fits, then predictions of their models
        dict(name="server_fp16", kind="server", form="mixed-fp16", count=12, lot=5, n_lo=10_000,
             n_hi=1_000_000, k_lo=8, k_hi=512, iters=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# No drawn case has more work than the largest listed one.
MAX_FLOPS = 2.0 * 10_000_000 * 64 * 1024 * 9


def draw(rng):
    kind = rng.choice(["driver", "driver", "driver", "driver", "step", "predict", "transform", "estimator",
                       "batch", "server"])
    if kind in ("batch", "server"):
        c = dict(kind=kind, count=rng.randint(4, 24 if kind == "batch" else 12), lot=rng.randrange(10_000),
                 n_lo=2_000, n_hi=_log_int(rng, 50_000, 500_000), k_lo=4, k_hi=_log_int(rng, 64, 512),
                 iters=rng.randint(5, 20))
        if kind == "server":
            c["form"] = rng.choice(["mixed-fp16", "mixed-fp16", "mixed-bf16", "plain"])
            c["n_lo"], c["iters"] = 10_000, rng.randint(4, 10)
        return c
    c = dict(kind=kind, dtype="f32")
    if kind == "driver":
        c["form"] = rng.choice(["plain", "plain", "mixed-fp16", "mixed-bf16"])
        c["dtype"] = rng.choice(["f32", "f64"]) if c["form"] == "plain" else "f32"
        c["iters"] = rng.randint(4, 20) if c["form"] == "plain" else rng.randint(4, 8)
        c["weights"] = rng.choice(["unit", "random"])
        c["far"] = c["form"] == "plain" and rng.random() < 0.25
        n, d, k = _log_int(rng, 20_000 if c["form"] == "plain" else 100_000, 5_000_000), _log_int(rng, 2, 128), _log_int(rng, 4, 1024)
        # keep double precision and plain cases within what their rates allow
        cap = MAX_FLOPS * (0.005 if c["dtype"] == "f64" else 0.1 if c["form"] == "plain" else 0.5)
        n = min(n, int(cap / (2.0 * d * k * (c["iters"] + 1))), 2_500_000_000 // (8 * d))
        n = max(n, 20 * k)
    elif kind == "step":
        n, d, k = _log_int(rng, 20_000, 2_000_000), _log_int(rng, 2, 100), _log_int(rng, 8, 512)
        c["weights"] = rng.choice(["unit", "random"])
    elif kind == "predict":
        n, d, k = _log_int(rng, 1_000, 2_000_000), _log_int(rng, 2, 128), _log_int(rng, 4, 1024)
        c["dtype"] = rng.choice(["f32", "f32", "f64"])
        if c["dtype"] == "f64":
            n = min(n, int(2e10 / (2.0 * d * k)))
    elif kind == "transform":
        n, d, k = _log_int(rng, 1_000, 1_000_000), _log_int(rng, 2, 128), _log_int(rng, 4, 512)
    else:
        n, d, k = _log_int(rng, 10_000, 400_000), _log_int(rng, 2, 32), _log_int(rng, 4, 100)
        c["form"] = rng.choice(["plain", "mixed-fp16"])
        c["iters"] = rng.randint(5, 25)
    c.update(n=n, d=d, k=min(k, n))
    if kind in ("driver", "step", "predict"):
        c["labels"] = rng.choice(["i32", "i64"])
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _lots(case):
    """(n, d, k) of every instance of a batch or server case."""
    rng = random.Random(case["lot"])
    dims = [8, 16, 32, 64, 128] if case["kind"] == "batch" else [16, 32, 64]
    out = []
    for _ in range(case["count"]):
        n, k = _log_int(rng, case["n_lo"], case["n_hi"]), _log_int(rng, case["k_lo"], case["k_hi"])
        out.append((n, rng.choice(dims), min(k, n // 20)))
    return out


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _blobs(n, d, k, dtype, g):
    """Feature-major blobs (d, n) and k of their rows as initial centroids (d, k)."""
    centers = torch.rand((d, k), generator=g, device="cuda", dtype=dtype) * 20 - 10
    std = torch.rand(k, generator=g, device="cuda", dtype=dtype) * 1.5 + 0.5
    blob = torch.randperm(n, generator=g, device="cuda") % k
    X = torch.empty((d, n), device="cuda", dtype=dtype)
    for f in range(d):
        X[f] = torch.randn(n, generator=g, device="cuda", dtype=dtype) * std[blob] + centers[f][blob]
    rows = torch.randperm(n, generator=g, device="cuda")[:k]
    return X, X[:, rows].contiguous()


def _overlapping(n, d, k, dtype, g, apart):
    """Blobs whose half distances are about apart * sqrt(2 ln(20 k)) standard
    deviations (0.85: a few percent of the samples lie nearer to another
    centre), and centroids as 32 samples of each blob would give them."""
    half = apart * math.sqrt(2 * math.log(20 * k)) * math.sqrt(6 / d)
    centers = (torch.rand((d, k), generator=g, device="cuda", dtype=dtype) * 2 - 1) * half
    std = torch.rand(k, generator=g, device="cuda", dtype=dtype) * 0.6 + 0.7
    blob = torch.randperm(n, generator=g, device="cuda") % k
    X = torch.empty((d, n), device="cuda", dtype=dtype)
    for f in range(d):
        X[f] = torch.randn(n, generator=g, device="cuda", dtype=dtype) * std[blob] + centers[f][blob]
    return X, centers + torch.randn((d, k), generator=g, device="cuda", dtype=dtype) * std / math.sqrt(32)


def _weights(case, n, dtype, g):
    if case.get("weights", "unit") == "unit":
        return torch.ones(n, device="cuda", dtype=dtype)
    return torch.rand(n, generator=g, device="cuda", dtype=dtype) + 0.5


class _Server:
    """A request server that a program keeps open between bursts."""

    def __init__(self, form, slots):
        self.h = ctypes.c_void_p()
        capi.check(capi.lib().kmc_server_open(FORMS[form], 20 * 10 ** 9, slots,
                                              torch.cuda.current_stream().cuda_stream, ctypes.byref(self.h)))

    def __del__(self):
        capi.lib().kmc_server_close(self.h)


def _tensors(case, seed):
    """The inputs alone, as a dict (or a list of them), from the seed."""
    g = _generator(seed)
    kind = case["kind"]

    def make(n, d, k, dtype, g):
        if case.get("form", "plain") == "plain" or kind == "estimator":
            return _blobs(n, d, k, dtype, g)
        # beyond 32 features the sums are float32 in arrival order, so labels on
        # a border change from run to run: many of them in the largest fit,
        # hardly any elsewhere
        return _overlapping(n, d, k, dtype, g, 0.85 if d <= 32 else case.get("apart", 1.2))

    if kind in ("batch", "server"):
        items = []
        for n, d, k in _lots(case):
            X, C0 = make(n, d, k, torch.float32, g)
            items.append(dict(n=n, d=d, k=k, X=X, C0=C0, w=torch.ones(n, device="cuda")))
        if kind == "server":
            for it in items[::3]:  # every third model also labels new samples
                n_new = max(1000, it["n"] // 4)
                it["new"] = it["X"][:, torch.randint(0, it["n"], (n_new,), generator=g, device="cuda")]
                it["new"] += torch.randn(it["new"].shape, generator=g, device="cuda") * 0.25
        return items
    n, d, k, dtype = case["n"], case["d"], case["k"], DTYPES[case["dtype"]]
    X, C0 = make(n, d, k, dtype, g)
    if case.get("far"):
        C0[:, 0] = 1e3
    return dict(X=X, C0=C0, w=_weights(case, n, dtype, g))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, seed=seed, kind=kind)
    t = _tensors(case, seed)
    if kind in ("batch", "server"):
        s["items"] = t
        for it in t:
            it["C"] = torch.empty_like(it["C0"])
            it["labels"] = torch.empty(it["n"], dtype=torch.int32, device="cuda")
            if "new" in it:
                it["new_labels"] = torch.empty(it["new"].shape[1], dtype=torch.int32, device="cuda")
        if kind == "server":
            s["server"] = _Server(case["form"], case["count"])
        return s
    s.update(t)
    X, C0 = t["X"], t["C0"]
    n, d, k = case["n"], case["d"], case["k"]
    if "labels" in case:
        s["labels"] = torch.empty(n, dtype=DTYPES[case["labels"]], device="cuda")
    if kind == "driver":
        s["C"], s["res"] = torch.empty_like(C0), torch.empty_like(C0)
    elif kind == "step":
        copies = kdp.compute_number_of_private_copies(X, n, d, k, 0.7, 128)
        s["hn"], s["sizes"], s["shifts"] = (torch.empty(k, dtype=X.dtype, device="cuda") for _ in range(3))
        s["size_copies"] = torch.empty((copies, k), dtype=X.dtype, device="cuda")
        s["copies"] = torch.empty((copies, d, k), dtype=X.dtype, device="cuda")
        s["res"] = torch.empty_like(C0)
        s["inertia"] = torch.empty(n, dtype=X.dtype, device="cuda")
        s["empty"] = torch.empty(k, dtype=s["labels"].dtype, device="cuda")
        s["n_empty"] = torch.empty(1, dtype=s["labels"].dtype, device="cuda")
    elif kind == "predict":
        s["hn"] = torch.empty(k, dtype=X.dtype, device="cuda")
    elif kind == "transform":
        s["dist"] = torch.empty((k, n), dtype=X.dtype, device="cuda")
    else:
        s["rows"] = X.t().contiguous()
        del s["X"]
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _run_driver(s):
    c = s["case"]
    s["C"].copy_(s["C0"])  # the driver overwrites its initial centroids
    n_iter, inertia = kdp.kmeans_lloyd_driver(s["X"], s["w"], s["C"], s["labels"], s["res"], 0.0, False,
                                              c["iters"], 8, 128, 0.7, None, form=c["form"])
    return {"centroids": s["res"], "labels": s["labels"], "inertia": inertia, "n_iter": n_iter}


def _run_step(s):
    X, C = s["X"], s["C0"]
    kdp.half_l2_norm_squared(C, s["hn"], 128, None)
    s["copies"].zero_()
    s["size_copies"].zero_()
    s["n_empty"].zero_()
    kdp.fused_lloyd_single_step(X, s["w"], C, s["hn"], s["labels"], s["copies"], s["size_copies"], 8, 128, None)
    kdp.reduce_centroids_data(s["size_copies"], s["copies"], s["sizes"], s["res"], s["empty"], s["n_empty"],
                              128, None)
    kdp.broadcast_divide(s["res"], s["sizes"], 128, None)
    kdp.compute_centroid_shifts_squared(C, s["res"], s["shifts"], None)
    kdp.compute_inertia(X, s["w"], s["res"], s["labels"], s["inertia"], 128, None)
    return {"centroids": s["res"], "sizes": s["sizes"], "labels": s["labels"], "n_empty": s["n_empty"],
            "shifts": s["shifts"], "inertia": s["inertia"]}


def _run_predict(s):
    kdp.half_l2_norm_squared(s["C0"], s["hn"], 128, None)
    kdp.assignment(s["X"], s["C0"], s["hn"], s["labels"], 8, 128, None)
    return {"half_norms": s["hn"], "labels": s["labels"]}


def _run_transform(s):
    kdp.compute_centroid_to_sample_distances(s["X"], s["C0"], s["dist"], 128, 8, None)
    return s["dist"]


def _run_estimator(s):
    c = s["case"]
    km = KMeans(n_clusters=c["k"], init="k-means++", max_iter=c["iters"], tol=1e-4, random_state=s["seed"],
                form=c["form"]).fit(s["rows"])
    return {"centroids": km.cluster_centers_, "labels": km.labels_, "inertia": km.inertia_, "n_iter": km.n_iter_}


def _run_batch(s):
    L = capi.lib()
    h, out = ctypes.c_void_p(), []
    capi.check(L.kmc_batch_create(len(s["items"]), torch.cuda.current_stream().cuda_stream, ctypes.byref(h)))
    try:
        slots = []
        for it in s["items"]:
            it["C"].copy_(it["C0"])
            q = ctypes.c_int64()
            capi.check(L.kmc_batch_add_fit_f32(h, it["X"].data_ptr(), it["w"].data_ptr(), it["C"].data_ptr(),
                                               it["labels"].data_ptr(), it["n"], it["d"], it["k"], 0.0,
                                               s["case"]["iters"], ctypes.byref(q)))
            slots.append(q.value)
        capi.check(L.kmc_batch_run(h))
        iters, inertia = [], []
        for q in slots:
            done, ni, inr = ctypes.c_int(), ctypes.c_int64(), ctypes.c_double()
            capi.check(L.kmc_batch_result(h, q, ctypes.byref(done), ctypes.byref(ni), ctypes.byref(inr)))
            iters.append(ni.value)
            inertia.append(inr.value)
    finally:
        capi.check(L.kmc_batch_destroy(h))
    # the labels of all instances as one array, so that a pass has few outputs
    return {"centroids": [it["C"] for it in s["items"]], "labels": torch.cat([it["labels"] for it in s["items"]]),
            "inertia": np.array(inertia, np.float32), "n_iter": np.array(iters)}


def _wait(srv, ticket):
    status, ni, inr = ctypes.c_int(), ctypes.c_int64(), ctypes.c_double()
    capi.check(capi.lib().kmc_server_wait(srv, ticket, ctypes.byref(status), ctypes.byref(ni), ctypes.byref(inr)))
    capi.check(status.value)
    return ni.value, inr.value


def _run_server(s):
    L, srv, fits, news = capi.lib(), s["server"].h, [], []
    for it in s["items"]:
        q = ctypes.c_int64()
        capi.check(L.kmc_server_submit_fit_f32(srv, it["X"].data_ptr(), it["w"].data_ptr(), it["C0"].data_ptr(),
                                               it["labels"].data_ptr(), it["C"].data_ptr(), it["n"], it["d"],
                                               it["k"], 0.0, s["case"]["iters"], ctypes.byref(q)))
        fits.append(q.value)
    for it, model in zip(s["items"], fits):
        if "new" in it:
            q = ctypes.c_int64()
            capi.check(L.kmc_server_submit_predict_f32(srv, it["new"].data_ptr(), model,
                                                       it["new_labels"].data_ptr(), it["new"].shape[1],
                                                       ctypes.byref(q)))
            news.append(q.value)
    done = [_wait(srv, q) for q in fits]
    for q in news:
        _wait(srv, q)
    for q in news + fits:
        capi.check(L.kmc_server_release(srv, q))
    return {"centroids": [it["C"] for it in s["items"]], "labels": torch.cat([it["labels"] for it in s["items"]]),
            "new_labels": torch.cat([it["new_labels"] for it in s["items"] if "new" in it]),
            "inertia": np.array([v for _, v in done], np.float32), "n_iter": np.array([i for i, _ in done])}


_RUN = dict(driver=_run_driver, step=_run_step, predict=_run_predict, transform=_run_transform,
            estimator=_run_estimator, batch=_run_batch, server=_run_server)


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------------------
# work of one pass
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("batch", "server"):
        lots, it = _lots(case), case["iters"]
        flops = sum(2.0 * n * d * k * (it + 1) for n, d, k in lots)
        nbytes = sum(4.0 * (n * d + 2 * n + 2 * d * k) for n, d, k in lots)
        if kind == "server":
            for n, d, k in lots[::3]:
                m = max(1000, n // 4)
                flops += 2.0 * m * d * k
                nbytes += 4.0 * (m * d + m)
        return {"bytes": nbytes, "flops": flops}
    n, d, k = case["n"], case["d"], case["k"]
    b = 8 if case["dtype"] == "f64" else 4
    lab = 8 if case.get("labels") == "i64" else 4
    once = 2.0 * n * d * k
    if kind == "driver":
        return {"bytes": b * (n * d + n + 2.0 * d * k) + lab * n, "flops": once * (case["iters"] + 1)}
    if kind == "step":
        return {"bytes": b * (n * d + 2 * n + 2.0 * d * k + 3 * k) + lab * n, "flops": once + 3.0 * n * d}
    if kind == "predict":
        return {"bytes": b * (n * d + 1.0 * d * k) + lab * n, "flops": once}
    if kind == "transform":
        return {"bytes": b * (n * d + d * k + 1.0 * n * k), "flops": 1.5 * once}
    # seeding (one distance per sample and centre) and the fit
    return {"bytes": b * (n * d + 1.0 * d * k) + 8 * n, "flops": once * (case["iters"] + 2)}


# ---------------------------------------------------------------------------
# the same results in 64 bits, from torch alone
# ---------------------------------------------------------------------------
def _assign64(X, C):
    """Labels of the columns of X (d, n) against C (d, k), float64, in chunks."""
    hn, step = (C * C).sum(0) / 2, max(1, (1 << 27) // C.shape[1])
    return torch.cat([(hn - X[:, i:i + step].double().t() @ C).argmin(1) for i in range(0, X.shape[1], step)])


def _sqdist64(X, C, labels):
    out, step = torch.empty(X.shape[1], device=X.device, dtype=torch.float64), 1 << 21
    for i in range(0, X.shape[1], step):
        out[i:i + step] = ((X[:, i:i + step].double() - C[:, labels[i:i + step]]) ** 2).sum(0)
    return out


def _lloyd64(X, w, C0, iters, tol=0.0):
    """Lloyd iterations with relocation of empty clusters: (centroids (d, k), inertia)."""
    C, w, (d, k), step = C0.double(), w.double(), C0.shape, 1 << 21
    for _ in range(iters):
        labels = _assign64(X, C)
        sums, sizes = torch.zeros((k, d), device=X.device, dtype=torch.float64), torch.zeros(
            k, device=X.device, dtype=torch.float64)
        for i in range(0, X.shape[1], step):
            sums.index_add_(0, labels[i:i + step], (X[:, i:i + step].double() * w[i:i + step]).t())
        sizes.index_add_(0, labels, w)
        empty = (sizes == 0).nonzero().flatten()
        if len(empty):
            far = torch.topk(_sqdist64(X, C, labels), len(empty)).indices
            for j, i in zip(empty.tolist(), far.tolist()):
                xw = X[:, i].double() * w[i]
                sums[labels[i]] -= xw
                sums[j] = xw
                sizes[labels[i]] -= w[i]
                sizes[j] = w[i]
        new = (sums / sizes[:, None]).t()
        shift = float(((new - C) ** 2).sum())
        C = new
        if shift <= tol:
            break
    return C, float((_sqdist64(X, C, _assign64(X, C)) * w).sum())


def _splitmix(z):
    m = (1 << 64) - 1
    z = (z + 0x9E3779B97F4A7C15) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def _seeds64(X, k, seed):
    """The k-means++ rows of unit-weight samples: draw t takes the first row
    whose running sum of min ||x - c||^2 exceeds u_t times the total."""
    n, rows, best = X.shape[1], [], None
    for t in range(k):
        v = torch.ones(n, device=X.device, dtype=torch.float64) if best is None else best.double()
        run_sum = v.cumsum(0)
        u = (_splitmix(seed ^ _splitmix(t)) >> 11) * 2.0 ** -53
        r = int(torch.searchsorted(run_sum, u * run_sum[-1], right=True))
        rows.append(min(r, n - 1))
        acc = torch.zeros(n, device=X.device, dtype=X.dtype)
        for f in range(X.shape[0]):
            diff = (X[f] - X[f, rows[-1]]).double()
            acc = (diff * diff + acc.double()).to(X.dtype)
        best = acc if best is None else torch.minimum(best, acc)
    return X[:, torch.tensor(rows, device=X.device)].contiguous()


def exact(case, seed):
    kind, t = case["kind"], _tensors(case, seed)
    if kind in ("batch", "server"):
        got = [_lloyd64(it["X"], it["w"], it["C0"], case["iters"]) for it in t]
        out = {"centroids": [c for c, _ in got], "labels": None, "n_iter": None,
               "inertia": np.array([v for _, v in got])}
        if kind == "server":
            out["new_labels"] = None
        return out
    X, C0, w = t["X"], t["C0"], t["w"]
    if kind == "driver":
        C, inertia = _lloyd64(X, w, C0, case["iters"])
        return {"centroids": C, "labels": None, "inertia": np.array([inertia]), "n_iter": None}
    if kind == "estimator":
        drawn = int(np.random.default_rng(seed).integers(0, 2 ** 63 - 1))
        tol = 1e-4 * float(X.double().var(1, unbiased=False).mean())
        C, inertia = _lloyd64(X, w, _seeds64(X, case["k"], drawn), case["iters"], tol)
        return {"centroids": C.t().contiguous(), "labels": None, "inertia": inertia, "n_iter": None}
    C = C0.double()
    if kind == "predict":
        return {"half_norms": (C * C).sum(0) / 2, "labels": None}
    if kind == "transform":
        out = torch.empty((case["k"], case["n"]), device="cuda", dtype=torch.float64)
        Xd = X.double()
        for j in range(case["k"]):
            out[j] = ((Xd - C[:, j:j + 1]) ** 2).sum(0).sqrt()
        return out
    labels = _assign64(X, C)
    wd, Xd = w.double(), X.double()
    sums = torch.zeros((case["k"], case["d"]), device="cuda", dtype=torch.float64).index_add_(0, labels, (Xd * wd).t())
    sizes = torch.zeros(case["k"], device="cuda", dtype=torch.float64).index_add_(0, labels, wd)
    new = (sums / sizes[:, None]).t()
    return {"centroids": new, "sizes": sizes, "labels": None, "n_empty": None, "shifts": ((C - new) ** 2).sum(0),
            "inertia": _sqdist64(X, new, labels) * wd}
