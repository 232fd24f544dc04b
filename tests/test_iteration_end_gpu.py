"""The end of an iteration where its kernels change path: features beyond one
round, clusters beyond one per CTA, direct and copied sums, and relocations of
one, many and more clusters than are ranked by counting pairs, with many equal
distances, through the driver (host-launched relocation) and kmc_fit_step
(enqueued with the iteration).

Samples, weights and initial centroids are small integers, so every sum is
exact in float32, float64 and fixed point: centroids and labels must equal the
oracle's exactly."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = {"plain": 0, "mixed-bf16": 1, "mixed-fp16": 2}


def _problem(n, d, k, empty, seed):
    rng = np.random.default_rng(seed)
    X = rng.integers(-8, 9, (d, n)).astype(np.float32)
    C = np.ascontiguousarray(X[:, rng.choice(n, k, replace=n < k)])
    # duplicates of centroid 0: only the first of them gets samples
    C[:, rng.choice(np.arange(1, k), empty, replace=False)] = C[:, :1]
    return X, C


CASES = [  # n, d, k, duplicated (empty) centroids
    (1000, 2, 3, 1), (5000, 14, 16, 3), (700, 1500, 4, 1), (3000, 7, 129, 20), (20_000, 3, 4200, 100),
    (30_000, 5, 9000, 6000), (50, 4, 40, 30), (60_001, 33, 70, 8), (40_000, 64, 300, 25), (9000, 100, 40, 2)]


@pytest.mark.parametrize("n,d,k,empty", CASES)
@pytest.mark.parametrize("form,dt", [("plain", np.float32), ("plain", np.float64), ("mixed-fp16", np.float32),
                                     ("mixed-bf16", np.float32)])
@pytest.mark.parametrize("how", ["driver", "step"])
def test_iterations_equal_the_oracles(oracle, n, d, k, empty, form, dt, how):
    import torch

    import kmeans_dpcpp_gb300 as kdp
    from kmeans_dpcpp_gb300 import capi

    if form != "plain" and (d > 256 or k > 4096):
        pytest.skip("outside the tensor-core forms' interesting range")
    X, C0 = _problem(n, d, k, empty, n + d + k)
    X, C0 = X.astype(dt), C0.astype(dt)
    iters = 2
    it_o, lab_o, C_o, inr_o, reloc_o = oracle.kmeans_lloyd_driver(X, np.ones(n, dt), C0, 0.0, iters)
    assert reloc_o > 0
    Xg, w = torch.from_numpy(X).cuda(), torch.ones(n, dtype=torch.from_numpy(X).dtype, device="cuda")
    cur = torch.from_numpy(C0.copy()).cuda()
    res = torch.empty_like(cur)
    lab = torch.empty(n, dtype=torch.int64, device="cuda")
    if how == "driver":
        it, inr = kdp.kmeans_lloyd_driver(Xg, w, cur, lab, res, 0.0, False, iters, 8, 128, 0.7, None, form=form)
        inr = float(np.asarray(inr).reshape(-1)[0])
    else:
        L, fit = capi.lib(), ctypes.c_void_p()
        create = getattr(L, "kmc_fit_create_%s_i64" % ("f64" if dt == np.float64 else "f32"))
        capi.check(create(Xg.data_ptr(), w.data_ptr(), cur.data_ptr(), lab.data_ptr(), res.data_ptr(), n, d, k,
                          0.0, iters, FORMS[form], torch.cuda.current_stream().cuda_stream, ctypes.byref(fit)))
        try:
            capi.check(L.kmc_fit_step(fit, iters))
            ni, v = ctypes.c_int64(), ctypes.c_double()
            capi.check(L.kmc_fit_finalize(fit, ctypes.byref(ni), ctypes.byref(v)))
            it, inr = ni.value, v.value
        finally:
            capi.check(L.kmc_fit_destroy(fit))
    assert it == it_o
    np.testing.assert_array_equal(cur.cpu().numpy(), C_o)
    np.testing.assert_array_equal(res.cpu().numpy(), C_o)
    np.testing.assert_array_equal(lab.cpu().numpy(), lab_o)
    # per-sample distances in dataT, summed in float64 / long double
    assert inr == pytest.approx(inr_o, rel=1e-6 if dt == np.float32 else 1e-12)
