"""Calls of different shapes that share one kernel, from several host threads at
once and in one captured graph.

A kernel's limit of dynamic shared memory belongs to the function, not to a
launch: a call must not narrow it for a larger call that another thread is
about to launch, nor for one captured earlier.  Every call succeeds and gives
what it gives alone."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, D = 2000, 32
SHAPES = [100, 700]  # clusters: the same kernel instances, 20 and 100 KB


class _Call:
    """Half norms, labels and (float32) distances of one shape."""

    def __init__(self, k, dt):
        import torch

        from kmeans_dpcpp_gb300 import capi

        self.L, self.k, self.suf = capi.lib(), k, "f32" if dt == np.float32 else "f64"
        rng = np.random.default_rng(k)
        X = rng.standard_normal((D, N)).astype(dt)
        self.X = torch.from_numpy(X).cuda()
        self.C = torch.from_numpy(np.ascontiguousarray(X[:, :k])).cuda()
        self.hn = torch.empty(k, dtype=self.X.dtype, device="cuda")
        self.lab = torch.empty(N, dtype=torch.int32, device="cuda")
        self.dist = torch.empty((k, N), dtype=self.X.dtype, device="cuda")
        torch.cuda.synchronize()

    def enqueue(self, s):
        p = [t.data_ptr() for t in (self.X, self.C, self.hn, self.lab, self.dist)]
        rc = [getattr(self.L, "kmc_half_l2_norm_squared_" + self.suf)(p[1], p[2], D, self.k, 128, s),
              getattr(self.L, f"kmc_assignment_{self.suf}_i32")(p[0], p[1], p[2], p[3], N, D, self.k, 8, 128, s)]
        if self.suf == "f32":
            rc.append(self.L.kmc_compute_centroid_to_sample_distances_f32(p[0], p[1], p[4], N, D, self.k, 128, 8, s))
        return [(r, self.L.kmc_last_error()) for r in rc if r != 0]

    def outputs(self):
        return [t.clone() for t in ((self.lab, self.dist) if self.suf == "f32" else (self.lab,))]


def _alone(call):
    import torch

    s = torch.cuda.Stream()
    assert not call.enqueue(s.cuda_stream)
    torch.cuda.synchronize()
    return call.outputs()


def _run(jobs):
    out = [None] * len(jobs)

    def work(q):
        try:
            out[q] = jobs[q]()
        except Exception as e:  # reported by the caller
            out[q] = e

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for o in out:
        if isinstance(o, Exception):
            raise o
    return out


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_threads_with_two_shapes_of_one_kernel(dt):
    import torch

    calls = [_Call(SHAPES[q % 2], dt) for q in range(4)]
    want = [_alone(c) for c in calls]
    streams = [torch.cuda.Stream() for _ in calls]

    def job(q):
        def go():
            bad = []
            for _ in range(3000):
                bad += calls[q].enqueue(streams[q].cuda_stream)
            return bad
        return go

    bad = _run([job(q) for q in range(4)])
    torch.cuda.synchronize()
    assert [len(b) for b in bad] == [0] * 4, [b[0] for b in bad if b]
    for c, w in zip(calls, want):
        for a, b in zip(c.outputs(), w):
            assert torch.equal(a, b)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("order", [(700, 100), (100, 700)])
def test_one_graph_with_two_shapes_of_one_kernel(dt, order):
    import torch

    calls = [_Call(k, dt) for k in order]
    want = [_alone(c) for c in calls]
    for c in calls:
        c.lab.fill_(-1)
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=s):
        for c in calls:
            assert not c.enqueue(s.cuda_stream)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    for c, w in zip(calls, want):
        for a, b in zip(c.outputs(), w):
            assert torch.equal(a, b)


def _fit(L, capi, X, C0, form, max_iter, stream):
    import torch

    d, n = X.shape
    k = C0.shape[1]
    suf = "f64" if X.dtype == torch.float64 else "f32"
    with torch.cuda.stream(stream):
        w = torch.ones(n, dtype=X.dtype, device="cuda")
        cur = C0.clone()
        res, lab = torch.empty_like(cur), torch.empty(n, dtype=torch.int32, device="cuda")
        fit = ctypes.c_void_p()
        capi.check(getattr(L, f"kmc_fit_create_{suf}_i32")(
            X.data_ptr(), w.data_ptr(), cur.data_ptr(), lab.data_ptr(), res.data_ptr(), n, d, k, 0.0, max_iter,
            form, stream.cuda_stream, ctypes.byref(fit)))
        try:
            capi.check(L.kmc_fit_run(fit))
            it, inr = ctypes.c_int64(), ctypes.c_double()
            capi.check(L.kmc_fit_finalize(fit, ctypes.byref(it), ctypes.byref(inr)))
        finally:
            capi.check(L.kmc_fit_destroy(fit))
        stream.synchronize()
        return it.value, inr.value, lab, res


# float64 labels and ordered sums (all of a CTA's copies in shared memory);
# tensor-core sums sorted by label with the largest tiles
@pytest.mark.parametrize("n,d,ks,dt,form,reps", [(3000, 32, (100, 300), np.float64, 0, 12),
                                                 (2_480_000, 4, (10, 1500), np.float32, 2, 4)])
def test_threads_with_fits_of_two_shapes(n, d, ks, dt, form, reps):
    import torch

    from kmeans_dpcpp_gb300 import capi

    L = capi.lib()
    rng = np.random.default_rng(n)
    # small integers: every sum is exact
    X = torch.from_numpy(rng.integers(-64, 65, (d, n)).astype(dt)).cuda()
    C0 = [X[:, :k].contiguous() for k in ks]
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    want = [_fit(L, capi, X, c, form, 12, streams[0]) for c in C0]

    def job(q):
        return lambda: [_fit(L, capi, X, C0[q % 2], form, 12, streams[q]) for _ in range(reps)]

    for q, runs in enumerate(_run([job(q) for q in range(4)])):
        for it, inr, lab, res in runs:
            assert (it, inr) == want[q % 2][:2]
            assert torch.equal(lab, want[q % 2][2]) and torch.equal(res, want[q % 2][3])
