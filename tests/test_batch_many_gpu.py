"""More instances in one engine step than a grid's y or z extent can count
(65,535): every one advances, stops and finishes."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_more_fits_than_a_grid_dimension_counts():
    import torch

    from kmeans_dpcpp_gb300 import capi

    L = capi.lib()
    count, n = 65_540, 3
    rng = np.random.default_rng(1)
    X = rng.integers(-50, 51, (count, n)).astype(np.float32)
    Xg, w = torch.from_numpy(X).cuda(), torch.ones(n, device="cuda")
    C = Xg[:, 0].clone().contiguous()
    lab = torch.full((count, n), -1, dtype=torch.int32, device="cuda")
    batch = ctypes.c_void_p()
    capi.check(L.kmc_batch_create(count, torch.cuda.current_stream().cuda_stream, ctypes.byref(batch)))
    try:
        inst = ctypes.c_int64()
        add, x, c, t = L.kmc_batch_add_fit_f32, Xg.data_ptr(), C.data_ptr(), lab.data_ptr()
        for q in range(count):
            capi.check(add(batch, x + 12 * q, w.data_ptr(), c + 4 * q, t + 12 * q, n, 1, 1, 0.0, 2,
                           ctypes.byref(inst)))
            assert inst.value == q
        capi.check(L.kmc_batch_run(batch))
        fin, it, inr = ctypes.c_int(), ctypes.c_int64(), ctypes.c_double()
        mean = X.sum(axis=1) / np.float32(n)  # exact sums, one rounding
        for q in list(range(0, count, 997)) + list(range(65_530, count)):
            capi.check(L.kmc_batch_result(batch, q, ctypes.byref(fin), ctypes.byref(it), ctypes.byref(inr)))
            want = np.square(X[q].astype(np.float64) - mean[q]).sum()
            assert fin.value == 1 and 1 <= it.value <= 2
            assert inr.value == pytest.approx(want, rel=1e-6)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(C.cpu().numpy(), mean)
        assert int(lab.abs().max()) == 0
    finally:
        capi.check(L.kmc_batch_destroy(batch))
