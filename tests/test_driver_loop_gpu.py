"""The host loop of a fit, which keeps two batches of iterations in flight: every
iteration limit around the batches' sizes, convergence inside a batch, empty
clusters in the first and in later iterations, and fits of several threads at
once, against the same fit advanced one iteration at a time.

Samples are small integers, so every sum is exact and the results must be
equal."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, d, k, empty, seed):
    rng = np.random.default_rng(seed)
    X = rng.integers(-8, 9, (d, n)).astype(np.float32)
    C = np.ascontiguousarray(X[:, rng.choice(n, k, replace=False)])
    if empty:
        C[:, 1:1 + empty] = C[:, :1]
    return X, C


def _fit(X, C0, tol, max_iter, by_steps, stream):
    import torch

    from kmeans_dpcpp_gb300 import capi

    L = capi.lib()
    d, n = X.shape
    k = C0.shape[1]
    with torch.cuda.stream(stream):
        Xg, cur, w = torch.from_numpy(X).cuda(), torch.from_numpy(C0.copy()).cuda(), torch.ones(n, device="cuda")
        res, lab = torch.empty_like(cur), torch.empty(n, dtype=torch.int32, device="cuda")
        fit = ctypes.c_void_p()
        capi.check(L.kmc_fit_create_f32_i32(Xg.data_ptr(), w.data_ptr(), cur.data_ptr(), lab.data_ptr(),
                                            res.data_ptr(), n, d, k, tol, max_iter, 0, stream.cuda_stream,
                                            ctypes.byref(fit)))
        try:
            for _ in range(by_steps):
                capi.check(L.kmc_fit_step(fit, 1))
            capi.check(L.kmc_fit_run(fit))
            it, inr = ctypes.c_int64(), ctypes.c_double()
            capi.check(L.kmc_fit_finalize(fit, ctypes.byref(it), ctypes.byref(inr)))
        finally:
            capi.check(L.kmc_fit_destroy(fit))
        stream.synchronize()
        return it.value, inr.value, lab.cpu().numpy(), res.cpu().numpy()


def _same(a, b):
    assert a[:2] == b[:2]
    np.testing.assert_array_equal(a[2], b[2])
    np.testing.assert_array_equal(a[3], b[3])


@pytest.mark.parametrize("max_iter", [0, 1, 2, 3, 4, 7, 8, 11, 12, 300])
@pytest.mark.parametrize("empty", [0, 5])
def test_run_equals_single_steps(max_iter, empty):
    import torch

    # few samples per cluster: relocated centroids keep leaving clusters empty
    X, C0 = _problem(400, 3, 40, empty, 5)
    s = torch.cuda.Stream()
    want = _fit(X, C0, 0.0, max_iter, max_iter, s)
    assert want[0] <= max_iter
    _same(_fit(X, C0, 0.0, max_iter, 0, s), want)
    _same(_fit(X, C0, 0.0, max_iter, min(2, max_iter), s), want)


def test_concurrent_fits_equal_fits_alone():
    import torch

    problems = [_problem(3000 + 100 * q, 4, 10 + q, q % 3, q) for q in range(24)]
    alone = [_fit(X, C0, 0.0, 30, 0, torch.cuda.Stream()) for X, C0 in problems]
    out = [None] * len(problems)

    def work(q0):
        s = torch.cuda.Stream()
        for q in range(q0, len(problems), 8):
            out[q] = _fit(*problems[q], 0.0, 30, 0, s)

    threads = [threading.Thread(target=work, args=(q,)) for q in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(out, alone):
        _same(a, b)
