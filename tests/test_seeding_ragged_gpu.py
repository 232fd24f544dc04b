"""k-means++ rows of blocks whose last part is ragged: within a warp, at its edges,
and in the first or the second half of the part.  The rows must equal the oracle's
sequential restatement, so there is no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 255, 256, 257, 288, 289, 513, 800, 4096 + 300])
@pytest.mark.parametrize("d", [3, 260])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_rows_equal_the_sequential_draw(oracle, n, d, dt):
    import torch

    from kmeans_dpcpp_gb300 import capi

    k = min(n, 12)
    rng = np.random.default_rng(n + d)
    X, w = rng.standard_normal((d, n)).astype(dt), rng.uniform(0.1, 2.0, n).astype(dt)
    rows_o, C_o = oracle.kmeans_plusplus(X, k, 5, w)
    Xg, wg = torch.from_numpy(X).cuda(), torch.from_numpy(w).cuda()
    C = torch.zeros((d, k), dtype=Xg.dtype, device="cuda")
    rows = torch.full((k,), -1, dtype=torch.int32, device="cuda")
    fn = getattr(capi.lib(), "kmc_kmeans_plusplus_" + ("f32" if dt == np.float32 else "f64"))
    capi.check(fn(Xg.data_ptr(), wg.data_ptr(), n, d, k, 5, C.data_ptr(), rows.data_ptr(),
                  torch.cuda.current_stream().cuda_stream))
    np.testing.assert_array_equal(rows.cpu().numpy(), rows_o)
    np.testing.assert_array_equal(C.cpu().numpy(), C_o)
