"""Labels, distances and sums where the dispatch between the register and the
panel kernels, and the warps of a panel CTA that hold samples, change with the
number of samples: one warp, two warps per SM, one round of all warps, two and
three rounds, and one sample more or less.

Samples are small integers, so labels, squared distances and sums are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sizes():
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    edges = [32, sms * 32, 2 * sms * 64, 2 * sms * 128, sms * 8 * 32, sms * 16 * 32, 2 * sms * 16 * 32,
             3 * sms * 16 * 32]
    return sorted({e + o for e in edges for o in (-1, 0, 1)} | {1})


# (d, k): registers and panels; 16, 32 and 64 columns per step; 12 and 8 warps
@pytest.mark.parametrize("d,k", [(5, 11), (20, 12), (33, 12), (20, 64), (3, 100), (90, 17), (148, 5)])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_every_number_of_samples(oracle, d, k, dt):
    import torch

    import kmeans_dpcpp_gb300 as kdp

    rng = np.random.default_rng(d)
    sizes = _sizes()
    X = rng.integers(-8, 9, (d, sizes[-1])).astype(dt)
    C = rng.integers(-8, 9, (d, k)).astype(dt)
    want = oracle.assignment(X, C)
    Cg = torch.from_numpy(C).cuda()
    hn = torch.empty(k, dtype=Cg.dtype, device="cuda")
    kdp.half_l2_norm_squared(Cg, hn, 128, None)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in sizes:
        Xg = torch.from_numpy(np.ascontiguousarray(X[:, :n])).cuda()
        lab = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        kdp.assignment(Xg, Cg, hn, lab, 8, 128, None)
        np.testing.assert_array_equal(lab.cpu().numpy(), want[:n], err_msg=str(n))
        if dt == np.float64:
            continue
        dist = torch.full((k, n), -1.0, device="cuda")
        kdp.compute_centroid_to_sample_distances(Xg, Cg, dist, 128, 8, None)
        exact = ((Cg.double() ** 2).sum(0)[:, None] - 2 * Cg.double().t() @ Xg.double()
                 + (Xg.double() ** 2).sum(0)[None, :]).sqrt().float()
        assert torch.equal(dist, exact), n
        # one step into as many copies as CTAs; integers far below 2^24
        lab.fill_(-1)
        cp = torch.zeros((sms, d, k), device="cuda")
        sz = torch.zeros((sms, k), device="cuda")
        kdp.fused_lloyd_single_step(Xg, torch.ones(n, device="cuda"), Cg, hn, lab, cp, sz, 8, 128, None)
        assert np.array_equal(lab.cpu().numpy(), want[:n]), n
        total = torch.zeros((k, d), device="cuda").index_add_(0, lab.long(), Xg.t().contiguous())
        assert torch.equal(cp.sum(0), total.t()), n
        assert torch.equal(sz.sum(0), torch.bincount(lab.long(), minlength=k).float()), n
