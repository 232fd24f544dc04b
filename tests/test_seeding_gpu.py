"""k-means++ rows where the draw's sums change path: block edges of the 4096-
sample sums, more block sums than threads, sums that are exact in any order and
sums whose order matters, and degenerate weights.  The rows must equal the
oracle's sequential restatement, so there is no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _samples(kind, n, d, rng):
    if kind == "grid":  # exact sums, many zero distances
        return rng.integers(-3, 4, (d, n)).astype(np.float32)
    if kind == "range":  # distances spread over many binades: order matters
        return (rng.standard_normal((d, n)) * 10.0 ** rng.integers(-12, 4, n)).astype(np.float32)
    return rng.standard_normal((d, n)).astype(np.float32)


def _weights(kind, n, rng):
    if kind == "none":
        return None
    if kind == "powers":
        return (2.0 ** rng.integers(-6, 7, n)).astype(np.float32)
    if kind == "mostly_zero":
        return np.where(rng.random(n) < 0.01, 1.0, 0.0).astype(np.float32)
    if kind == "zero":
        return np.zeros(n, np.float32)
    return rng.uniform(0.1, 2.0, n).astype(np.float32)


@pytest.mark.parametrize("n,d,k,data,weights", [
    (1, 1, 1, "normal", "none"), (4095, 2, 9, "normal", "none"), (4096, 2, 9, "range", "none"),
    (4097, 2, 9, "normal", "random"), (8192 + 1, 600, 5, "normal", "none"), (30_011, 3, 40, "grid", "none"),
    (30_011, 3, 12, "grid", "powers"), (50_000, 5, 30, "range", "random"), (20_000, 4, 20, "normal", "mostly_zero"),
    (9_000, 3, 6, "normal", "zero"), (4096 * 513 + 7, 1, 4, "normal", "none"),
    (4096 * 513 + 7, 1, 3, "range", "random")])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_rows_equal_the_sequential_draw(oracle, n, d, k, data, weights, dt):
    import torch

    from kmeans_dpcpp_gb300 import capi

    rng = np.random.default_rng(n + 7 * d + k)
    X, w = _samples(data, n, d, rng).astype(dt), _weights(weights, n, rng)
    w = None if w is None else w.astype(dt)
    rows_o, C_o = oracle.kmeans_plusplus(X, k, 5, w)
    Xg, wg = torch.from_numpy(X).cuda(), None if w is None else torch.from_numpy(w).cuda()
    C = torch.zeros((d, k), dtype=Xg.dtype, device="cuda")
    rows = torch.full((k,), -1, dtype=torch.int32, device="cuda")
    fn = getattr(capi.lib(), "kmc_kmeans_plusplus_" + ("f32" if dt == np.float32 else "f64"))
    capi.check(fn(Xg.data_ptr(), None if wg is None else wg.data_ptr(), n, d, k, 5, C.data_ptr(),
                  rows.data_ptr(), torch.cuda.current_stream().cuda_stream))
    np.testing.assert_array_equal(rows.cpu().numpy(), rows_o)
    np.testing.assert_array_equal(C.cpu().numpy(), C_o)


@pytest.mark.parametrize("n,d", [(1, 1), (2047, 3), (2049, 700), (100_003, 5)])
def test_variance_of_split_features(n, d):
    import ctypes

    import torch

    from kmeans_dpcpp_gb300 import capi

    X = np.random.default_rng(n).normal(5.0, 2.0, (d, n))
    Xg, out = torch.from_numpy(X).cuda(), ctypes.c_double()
    capi.check(capi.lib().kmc_mean_feature_variance_f64(Xg.data_ptr(), n, d, ctypes.byref(out),
                                                        torch.cuda.current_stream().cuda_stream))
    # two passes in float64: the mean's error enters squared
    np.testing.assert_allclose(out.value, np.mean(np.var(X, axis=1)), rtol=1e-12, atol=1e-28)


@pytest.mark.parametrize("n,k,weights", [(511, 30, "none"), (512, 30, "random"), (513, 30, "powers"),
                                         (4096 + 513, 40, "mostly_zero"), (4096 * 1024 + 5, 3, "none"),
                                         (4096 * 1024 - 5, 3, "powers")])
@pytest.mark.parametrize("data", ["normal", "grid", "range"])
def test_rows_at_the_edges_of_a_blocks_parts(oracle, n, k, weights, data):
    import torch

    from kmeans_dpcpp_gb300 import capi

    rng = np.random.default_rng(n + k)
    X, w = _samples(data, n, 2, rng), _weights(weights, n, rng)
    rows_o, _ = oracle.kmeans_plusplus(X, k, 11, w)
    Xg, wg = torch.from_numpy(X).cuda(), None if w is None else torch.from_numpy(w).cuda()
    C, rows = torch.zeros((2, k), device="cuda"), torch.full((k,), -1, dtype=torch.int32, device="cuda")
    capi.check(capi.lib().kmc_kmeans_plusplus_f32(Xg.data_ptr(), None if wg is None else wg.data_ptr(), n, 2, k, 11,
                                                  C.data_ptr(), rows.data_ptr(),
                                                  torch.cuda.current_stream().cuda_stream))
    np.testing.assert_array_equal(rows.cpu().numpy(), rows_o)
