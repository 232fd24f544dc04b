"""Reduction of private copies where its kernel changes: up to 8 copies, 16
threads per element, and one thread per element.  Beyond 8 copies the sums are the
same bits in either: 16 partial sums of every sixteenth copy, added in order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("P", [1, 3, 4, 7, 8, 9, 15, 16, 17, 31, 33, 152])
@pytest.mark.parametrize("d,k", [(1, 1), (3, 11), (32, 256), (31, 512), (127, 128), (63, 512), (123, 250)])
def test_sums_in_the_stated_order(dt, P, d, k):
    import torch

    import kmeans_dpcpp_gb300 as kdp

    rng = np.random.default_rng(P + d)
    cp, sz = rng.uniform(-1, 1, (P, d, k)).astype(dt), rng.uniform(0, 1, (P, k)).astype(dt)
    sz[:, ::7] = 0  # empty clusters
    C, S = (torch.full(s, np.nan, dtype=torch.from_numpy(cp).dtype, device="cuda") for s in ((d, k), (k,)))
    lst, cnt = torch.full((k,), -1, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    kdp.reduce_centroids_data(torch.from_numpy(sz).cuda(), torch.from_numpy(cp).cuda(), S, C, lst, cnt, 128, None)
    torch.cuda.synchronize()

    def total(a):
        G = 1 if P <= 8 else 16
        parts = np.zeros((G,) + a.shape[1:], dt)
        for p in range(P):
            parts[p % G] += a[p]
        for g in range(1, G):
            parts[0] += parts[g]
        return parts[0]

    np.testing.assert_array_equal(C.cpu().numpy(), total(cp))
    np.testing.assert_array_equal(S.cpu().numpy(), total(sz))
    empty = np.arange(0, k, 7)
    assert cnt.item() == len(empty)
    np.testing.assert_array_equal(lst.cpu().numpy()[:len(empty)], empty)
