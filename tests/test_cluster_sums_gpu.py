"""Cluster sums of the tensor-core forms (sorted by label, or sample by sample
beyond 2048 clusters) and of the plain form (float64 copies whose number follows
the sizes).

One iteration from given centroids: the next centroids are the weighted means of
the samples by their exact float32 labels.  Up to 32 features the sums are exact
integers rounded once, so a mean is within a few units in the last place.
Beyond, m products are added in float32 in any order: each sum is within
(m + 1) 2^-24 sum |w x| of the exact one and each size within m 2^-24 of its own
(relative), the division adds one rounding.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    (1, 3, 1),            # one sample
    (255, 32, 3),         # one short tile, 9 vectors per packed row
    (257, 31, 16),        # padded column, two tiles
    (5_000, 17, 2048),    # the most clusters that are sorted
    (5_000, 32, 2049),    # one more
    (5_000, 40, 2049),
    (3_000, 33, 5),       # the fewest features of the float32 sums
    (9_999, 64, 100),     # two rows per warp
    (3_000, 130, 7),      # 33 vectors per row: two column blocks
    (2_000, 256, 3),      # the most features
    (700_001, 4, 9),      # many samples per tile, ragged end
    (700_001, 36, 9),
]


# plain: copies per warp (few clusters), 16 copies, 4 copies, one
PLAIN = [(700_001, 4, 3), (400_003, 40, 5), (100_001, 64, 300), (70_000, 128, 700), (9_000, 140, 4000)]


@pytest.mark.parametrize("n,d,k", PLAIN)
def test_plain_sums_with_any_number_of_copies(oracle, n, d, k):
    _one_iteration(oracle, n, d, k, "plain", np.int32)


@pytest.mark.parametrize("n,d,k", SHAPES)
@pytest.mark.parametrize("form,labels", [("mixed-fp16", np.int32), ("mixed-bf16", np.int64)])
def test_one_iteration_gives_the_weighted_means(oracle, n, d, k, form, labels):
    _one_iteration(oracle, n, d, k, form, labels)


def _one_iteration(oracle, n, d, k, form, labels):
    import torch

    import kmeans_dpcpp_gb300 as kdp

    rng = np.random.default_rng(n + 7 * d + k)
    X = (rng.standard_normal((d, n)) * 3).astype(np.float32)
    # terms far below the rest, which the packed sums hand to float64
    X[0, ::97] *= np.float32(1e-12)
    w = rng.uniform(0.5, 1.5, n).astype(np.float32)
    C0 = np.ascontiguousarray(X[:, rng.permutation(n)[:k]])
    lab = oracle.assignment(X, C0)
    X64, w64 = X.astype(np.float64), w.astype(np.float64)
    size = np.bincount(lab, weights=w64, minlength=k)
    m = np.bincount(lab, minlength=k)
    assert m.min() > 0
    mean = np.stack([np.bincount(lab, weights=X64[f] * w64, minlength=k) for f in range(d)]) / size
    mag = np.stack([np.bincount(lab, weights=np.abs(X64[f]) * w64, minlength=k) for f in range(d)]) / size

    C = torch.from_numpy(C0).cuda()
    res = torch.empty_like(C)
    out = torch.empty(n, dtype=torch.int32 if labels == np.int32 else torch.int64, device="cuda")
    kdp.kmeans_lloyd_driver(torch.from_numpy(X).cuda(), torch.from_numpy(w).cuda(), C, out, res, 0.0, False,
                            1, 8, 128, 0.7, None, form=form)
    got = res.cpu().numpy().astype(np.float64)
    u = 2.0 ** -24
    # packed or float64: products, sum, size and quotient are rounded once each
    terms = 4 if d <= 32 or form == "plain" else 2 * m[None, :] + 4
    assert np.all(np.abs(got - mean) <= terms * u * mag * 1.01 + 1e-37)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.assignment(X, res.cpu().numpy()))
