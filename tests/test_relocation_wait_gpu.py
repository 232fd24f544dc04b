"""The plain form's device-side waits: the grid barriers of a relocation.

With a limit of one clock the first CTA to arrive gives up while the others
still work, so the wait runs out by itself: the kernel winds down, the loop
stops, the next blocking call reports it, and the context stays usable."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KMC_ERR_DEVICE_TIMEOUT = 5


def _problem(dt):
    rng = np.random.default_rng(2)
    X = rng.integers(-8, 9, (5, 60_000)).astype(dt)
    C = np.ascontiguousarray(X[:, rng.choice(X.shape[1], 12, replace=False)])
    C[:, 5:8] = C[:, :1]  # three clusters start empty
    return X, C


def _session(X, C0, labels, max_iter=4):
    import torch

    from kmeans_dpcpp_gb300 import capi

    d, n = X.shape
    t = dict(X=torch.from_numpy(X).cuda(), C=torch.from_numpy(C0.copy()).cuda(),
             lab=torch.empty(n, dtype=torch.int64 if labels == 64 else torch.int32, device="cuda"))
    t["w"], t["res"] = torch.ones(n, dtype=t["X"].dtype, device="cuda"), torch.empty_like(t["C"])
    create = getattr(capi.lib(), f"kmc_fit_create_{'f64' if X.dtype == np.float64 else 'f32'}_i{labels}")
    fit = ctypes.c_void_p()
    capi.check(create(t["X"].data_ptr(), t["w"].data_ptr(), t["C"].data_ptr(), t["lab"].data_ptr(),
                      t["res"].data_ptr(), n, d, C0.shape[1], 0.0, max_iter, 0,
                      torch.cuda.current_stream().cuda_stream, ctypes.byref(fit)))
    return fit, t


@pytest.mark.parametrize("dt,labels", [(np.float32, 32), (np.float64, 64)])
@pytest.mark.parametrize("how", ["run", "step"])
def test_a_plain_fits_limit_is_kept(oracle, dt, labels, how):
    import torch

    from kmeans_dpcpp_gb300 import capi

    L = capi.lib()
    X, C0 = _problem(dt)
    fit, t = _session(X, C0, labels)
    try:
        capi.check(L.kmc_fit_set_wait_limit(fit, 1, 0))
        if how == "run":
            rc = L.kmc_fit_run(fit)
        else:
            capi.check(L.kmc_fit_step(fit, 1))
            rc = L.kmc_fit_status(fit, None, None, None)
        assert rc == KMC_ERR_DEVICE_TIMEOUT
        assert "device-side wait" in L.kmc_last_error().decode()
        err = ctypes.c_int()
        capi.check(L.kmc_fit_rechecked(fit, None, None, ctypes.byref(err)))
        assert err.value == 1
        # the loop was stopped: later calls do nothing and keep reporting it
        capi.check(L.kmc_fit_step(fit, 2))
        assert L.kmc_fit_run(fit) == KMC_ERR_DEVICE_TIMEOUT
    finally:
        capi.check(L.kmc_fit_destroy(fit))
    torch.cuda.synchronize()

    # the default limit again (clocks <= 0), in a new session
    fit, t = _session(X, C0, labels)
    try:
        capi.check(L.kmc_fit_set_wait_limit(fit, 1, 0))
        capi.check(L.kmc_fit_set_wait_limit(fit, 0, 0))
        capi.check(L.kmc_fit_run(fit))
        it, inr, err = ctypes.c_int64(), ctypes.c_double(), ctypes.c_int()
        capi.check(L.kmc_fit_finalize(fit, ctypes.byref(it), ctypes.byref(inr)))
        capi.check(L.kmc_fit_rechecked(fit, None, None, ctypes.byref(err)))
        assert err.value == 0
    finally:
        capi.check(L.kmc_fit_destroy(fit))
    it_o, lab_o, C_o, _, reloc = oracle.kmeans_lloyd_driver(X, np.ones(X.shape[1], dt), C0, 0.0, 4)
    assert reloc > 0 and it.value == it_o
    np.testing.assert_array_equal(t["lab"].cpu().numpy(), lab_o)
    np.testing.assert_array_equal(t["res"].cpu().numpy(), C_o)
