"""The 128-sample tiles where they still run: more features than a panel takes
(148), float64 distances and steps, and float64 fits whose ordered sums do not
fit shared memory.  Every centroid width gives the same labels, and the batched
engine's tiles those of the oracle.

Samples are small integers, so every sum is exact and results must be equal."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, d, k, dt, seed):
    rng = np.random.default_rng(seed)
    X = rng.integers(-8, 9, (d, n)).astype(dt)
    return X, np.ascontiguousarray(X[:, rng.choice(n, k, replace=False)])


def _fit(X, C0, variant, max_iter):
    import torch

    from kmeans_dpcpp_gb300 import capi

    L = capi.lib()
    d, n = X.shape
    Xg, cur = torch.from_numpy(X).cuda(), torch.from_numpy(C0.copy()).cuda()
    w, res = torch.ones(n, dtype=Xg.dtype, device="cuda"), torch.empty_like(cur)
    lab = torch.empty(n, dtype=torch.int32, device="cuda")
    create = L.kmc_fit_create_f64_i32 if X.dtype == np.float64 else L.kmc_fit_create_f32_i32
    fit = ctypes.c_void_p()
    capi.check(create(Xg.data_ptr(), w.data_ptr(), cur.data_ptr(), lab.data_ptr(), res.data_ptr(), n, d,
                      C0.shape[1], 0.0, max_iter, 0, torch.cuda.current_stream().cuda_stream, ctypes.byref(fit)))
    try:
        capi.check(L.kmc_fit_set_tile_variant(fit, variant))
        capi.check(L.kmc_fit_run(fit))
        it, inr = ctypes.c_int64(), ctypes.c_double()
        capi.check(L.kmc_fit_finalize(fit, ctypes.byref(it), ctypes.byref(inr)))
    finally:
        capi.check(L.kmc_fit_destroy(fit))
    return it.value, lab.cpu().numpy(), res.cpu().numpy()


@pytest.mark.parametrize("n,d,k,dt", [
    (5003, 149, 3, np.float32), (4001, 160, 70, np.float32), (3000, 300, 130, np.float32),
    (5003, 149, 3, np.float64), (2001, 300, 33, np.float64), (4001, 64, 400, np.float64),
    (3000, 14, 1000, np.float64)])
def test_every_width_gives_the_oracles_fit(oracle, n, d, k, dt):
    X, C0 = _problem(n, d, k, dt, d + k)
    it, lab, C, _, _ = oracle.kmeans_lloyd_driver(X, np.ones(n, dt), C0, 0.0, 3)
    for v in (0, 1, 2):
        got = _fit(X, C0, v, 3)
        assert got[0] == it
        np.testing.assert_array_equal(got[2], C)
        np.testing.assert_array_equal(got[1], lab)


@pytest.mark.parametrize("n,d,k", [(3001, 149, 9), (5000, 200, 70), (1200, 1024, 140), (130, 149, 1)])
def test_batched_instances_beyond_the_panels(oracle, n, d, k):
    import torch

    from kmeans_dpcpp_gb300 import capi

    L = capi.lib()
    X, C0 = _problem(n, d, k, np.float32, n + d)
    it_o, lab_o, C_o, inr_o, _ = oracle.kmeans_lloyd_driver(X, np.ones(n, np.float32), C0, 0.0, 3)
    Xg, w = torch.from_numpy(X).cuda(), torch.ones(n, device="cuda")
    C, P = torch.from_numpy(C0.copy()).cuda(), torch.from_numpy(C0).cuda()
    lab, pred = (torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    batch, fit, inst = ctypes.c_void_p(), ctypes.c_int64(), ctypes.c_int64()
    capi.check(L.kmc_batch_create(4, torch.cuda.current_stream().cuda_stream, ctypes.byref(batch)))
    try:
        capi.check(L.kmc_batch_add_fit_f32(batch, Xg.data_ptr(), w.data_ptr(), C.data_ptr(), lab.data_ptr(), n, d,
                                           k, 0.0, 3, ctypes.byref(fit)))
        capi.check(L.kmc_batch_add_predict_f32(batch, Xg.data_ptr(), P.data_ptr(), pred.data_ptr(), n, d, k,
                                               ctypes.byref(inst)))
        capi.check(L.kmc_batch_run(batch))
        fin, it, inr = ctypes.c_int(), ctypes.c_int64(), ctypes.c_double()
        capi.check(L.kmc_batch_result(batch, fit, ctypes.byref(fin), ctypes.byref(it), ctypes.byref(inr)))
    finally:
        capi.check(L.kmc_batch_destroy(batch))
    torch.cuda.synchronize()
    assert fin.value == 1 and it.value == it_o
    np.testing.assert_array_equal(C.cpu().numpy(), C_o)
    np.testing.assert_array_equal(lab.cpu().numpy(), lab_o)
    np.testing.assert_array_equal(pred.cpu().numpy(), oracle.assignment(X, C0))
    assert inr.value == pytest.approx(inr_o, rel=1e-6)
