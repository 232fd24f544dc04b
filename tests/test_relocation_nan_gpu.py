"""Relocation when samples have no distance (NaN features).

Such samples rank below all others and are never moved; where fewer samples than
empty clusters have a distance, the last empty clusters get none.  Whatever the
scratch memory held before must not matter.

Samples are small integers, so the expected sums are exact."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, D, K, EMPTY = 6000, 3, 9, 5
REST = K - 1 - EMPTY
ALL_BUT_ONE = -1


def _problem(n_nan, dt):
    """Samples of cluster 0; clusters 1..EMPTY are its duplicates and get none;
    the rest lie far away, each with one sample of its own."""
    X, C = np.zeros((D, N), dt), np.zeros((D, K), dt)
    X[0], X[1] = np.arange(N) % 1000, np.arange(N) // 1000
    C[2, 1 + EMPTY:] = 10_000 * np.arange(1, REST + 1)
    X[:, N - REST:] = C[:, 1 + EMPTY:]
    nan = np.delete(np.arange(N - REST), 1234) if n_nan == ALL_BUT_ONE else np.arange(7, 7 + 11 * n_nan, 11)
    X[2, nan] = np.nan
    lab = np.zeros(N, np.int64)
    lab[N - REST:] = np.arange(1 + EMPTY, K)
    dist = np.square(X.astype(np.float64)).sum(axis=0)
    dist[N - REST:] = 0
    return X, C, lab, dist


def _relocated(X, lab, dist):
    """Sums and sizes after the moves."""
    sums = np.stack([X[:, lab == j].astype(np.float64).sum(axis=1) for j in range(K)], axis=1)
    size = np.bincount(lab, minlength=K).astype(np.float64)
    ok = np.flatnonzero(~np.isnan(dist))
    order = ok[np.lexsort((ok, -dist[ok]))][:EMPTY]
    for cl, i in zip(range(1, 1 + EMPTY), order):
        sums[:, lab[i]] -= X[:, i]
        sums[:, cl] = X[:, i]
        size[lab[i]] -= 1
        size[cl] = 1
    return sums, size


def _run(form, dt, labels, X, C0):
    import torch

    from kmeans_dpcpp_gb300 import capi

    L = capi.lib()
    Xg, cur = torch.from_numpy(X).cuda(), torch.from_numpy(C0.copy()).cuda()
    w, res = torch.ones(N, dtype=Xg.dtype, device="cuda"), torch.empty_like(cur)
    lab = torch.empty(N, dtype=torch.int64 if labels == "i64" else torch.int32, device="cuda")
    s, h = torch.cuda.current_stream().cuda_stream, ctypes.c_void_p()
    if form == "batch":
        inst = ctypes.c_int64()
        capi.check(L.kmc_batch_create(2, s, ctypes.byref(h)))
        try:
            capi.check(L.kmc_batch_add_fit_f32(h, Xg.data_ptr(), w.data_ptr(), cur.data_ptr(), lab.data_ptr(), N,
                                               D, K, 0.0, 1, ctypes.byref(inst)))
            capi.check(L.kmc_batch_run(h))
        finally:
            capi.check(L.kmc_batch_destroy(h))
    else:
        capi.check(getattr(L, f"kmc_fit_create_{'f64' if dt == np.float64 else 'f32'}_{labels}")(
            Xg.data_ptr(), w.data_ptr(), cur.data_ptr(), lab.data_ptr(), res.data_ptr(), N, D, K, 0.0, 1,
            {"plain": 0, "bf16": 1, "fp16": 2}[form], s, ctypes.byref(h)))
        try:
            capi.check(L.kmc_fit_run(h))
        finally:
            capi.check(L.kmc_fit_destroy(h))
    torch.cuda.synchronize()
    return cur.cpu().numpy()


@pytest.mark.parametrize("n_nan", [0, 1, 3, EMPTY, EMPTY + 4, ALL_BUT_ONE])
@pytest.mark.parametrize("form,dt,labels", [("plain", np.float32, "i32"), ("plain", np.float64, "i64"),
                                            ("fp16", np.float32, "i64"), ("bf16", np.float32, "i32"),
                                            ("batch", np.float32, "i32")])
def test_only_samples_with_a_distance_move(n_nan, form, dt, labels):
    X, C0, lab, dist = _problem(n_nan, dt)
    # leaves other sample numbers in the scratch memory that the next fit gets
    _run(form, dt, labels, np.ascontiguousarray(np.nan_to_num(X)[:, ::-1]), C0)
    got = _run(form, dt, labels, X, C0)
    sums, size = _relocated(X, lab, dist)
    with np.errstate(invalid="ignore", divide="ignore"):
        want = (sums / size).astype(dt)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("n_nan", [0, 2, EMPTY, ALL_BUT_ONE])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_the_separate_call_moves_the_same_samples(n_nan, dt):
    import torch

    from kmeans_dpcpp_gb300 import capi

    X, _, lab, dist = _problem(n_nan, dt)
    relocate = getattr(capi.lib(), f"kmc_relocate_empty_clusters_{'f64' if dt == np.float64 else 'f32'}_i32")

    def call(X, lab, dist):
        def g(a):
            return torch.from_numpy(np.ascontiguousarray(a)).cuda()

        before = np.stack([X[:, lab == j].sum(axis=1) for j in range(K)], axis=1).astype(dt)
        sums, sizes = g(before), g(np.bincount(lab, minlength=K).astype(dt))
        inertia, d = g(dist.astype(dt)), g(dist.astype(dt))
        a = [g(X), g(np.ones(N, dt)), g(lab.astype(np.int32)), g(np.arange(1, 1 + EMPTY, dtype=np.int32)), d]
        capi.check(relocate(EMPTY, *[t.data_ptr() for t in a], sums.data_ptr(), sizes.data_ptr(),
                            inertia.data_ptr(), N, D, K, 128, torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        return sums.cpu().numpy(), sizes.cpu().numpy()

    call(np.nan_to_num(X)[:, ::-1], lab[::-1], np.nan_to_num(dist)[::-1])
    sums, sizes = call(X, lab, dist)
    want, size = _relocated(X, lab, dist)
    np.testing.assert_array_equal(sums, want.astype(dt))
    np.testing.assert_array_equal(sizes, size.astype(dt))
