"""The kernels that hold the samples in registers (few centroids) or in panels
of shared memory, at the edges of their feature classes, of a warp's samples
and of the centroids that shared memory holds at once, in every data type;
beyond 148 features the tile kernels answer.  Labels, distances and (with integer data) sums must equal the
oracle's exactly: the arithmetic per score is the same.

Float64 labels come from float32 scores wherever those decide them, so they are
also checked where they cannot: ties, differences far below float32's
resolution, operands beyond float32's range in either direction, infinities and
NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gpu(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _labels(X, C, hn=None, it="int64"):
    import torch

    import kmeans_dpcpp_gb300 as kdp

    Xg, Cg = _gpu(X), _gpu(C)
    lab = torch.full((X.shape[1],), -1, dtype=getattr(torch, it), device="cuda")
    if hn is None:
        h = torch.empty(C.shape[1], dtype=Xg.dtype, device="cuda")
        kdp.half_l2_norm_squared(Cg, h, 128, None)
    else:
        h = _gpu(hn)
    kdp.assignment(Xg, Cg, h, lab, 8, 128, None)[0].wait()
    return lab.cpu().numpy()


SHAPES = [(1, 1, 1), (31, 2, 2), (127, 4, 7), (129, 5, 33), (1000, 8, 16), (257, 9, 300), (513, 12, 5),
          (300, 13, 1700), (5000, 16, 127), (1025, 17, 64), (700, 20, 1), (333, 24, 40), (640, 28, 90),
          (2000, 32, 900), (400, 33, 20), (800, 40, 65), (150, 48, 3), (260, 56, 128), (4000, 64, 1000),
          (500, 65, 30), (30_000, 14, 50), (70_001, 14, 100), (2500, 1, 65), (1111, 2, 66), (900, 3, 129),
          (1300, 30, 191), (4000, 64, 1025), (700, 65, 64), (650, 99, 800), (330, 128, 33), (300, 148, 70),
          (200, 149, 90), (150, 300, 17)]


@pytest.mark.parametrize("n,d,k", SHAPES)
@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("it", ["int32", "int64"])
def test_labels_equal_the_oracles(oracle, n, d, k, dt, it):
    rng = np.random.default_rng(n + 3 * d + k)
    X, C = rng.standard_normal((d, n)).astype(dt), rng.standard_normal((d, k)).astype(dt)
    np.testing.assert_array_equal(_labels(X, C, it=it), oracle.assignment(X, C))


@pytest.mark.parametrize("n,d,k", SHAPES)
def test_distances_equal_the_oracles(oracle, n, d, k):
    import torch

    import kmeans_dpcpp_gb300 as kdp

    rng = np.random.default_rng(n + 5 * d + k)
    X, C = rng.standard_normal((d, n)).astype(np.float32), rng.standard_normal((d, k)).astype(np.float32)
    out = torch.full((k, n), np.nan, dtype=torch.float32, device="cuda")
    kdp.compute_centroid_to_sample_distances(_gpu(X), _gpu(C), out, 128, 8, None)[0].wait()
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.distances(X, C))


def _hard(kind, d, n, k, rng, dt):
    C = rng.standard_normal((d, k)) * 3
    X = C[:, rng.integers(0, k, n)] + rng.standard_normal((d, n)) * 0.1
    if kind == "ties":  # equal centroids, and samples halfway between two
        C[:, 1::2] = C[:, 0:-1:2] if k % 2 == 0 else C[:, 0::2][:, :C[:, 1::2].shape[1]]
        X[:, ::2] = (C[:, rng.integers(0, k, n)] + C[:, rng.integers(0, k, n)])[:, ::2] / 2
    elif kind == "close":  # centroids 1e-12 apart
        C = C[:, :1] + rng.standard_normal((d, k)) * 1e-12
    elif kind == "tiny":
        X, C = X * 1e-200, C * 1e-200
    elif kind == "small":
        X, C = X * 1e-30, C * 1e-30
    elif kind == "huge":
        X, C = X * 1e120, C * 1e120
    elif kind == "large":
        X, C = X * 1e25, C * 1e25
    elif kind == "spread":  # centroids over 60 decades
        C *= 10.0 ** rng.integers(-30, 31, k)
        X *= 10.0 ** rng.integers(-30, 31, n)
    elif kind == "special":
        X.reshape(-1)[rng.integers(0, X.size, n // 8)] = rng.choice([np.inf, -np.inf, np.nan, 0.0], n // 8)
        C[rng.integers(0, d), rng.integers(0, k)] = np.nan
        C[rng.integers(0, d), rng.integers(0, k)] = np.inf
    elif kind == "zero":
        C[:], X[:, ::3] = 0.0, 0.0
    return X.astype(dt), C.astype(dt)


@pytest.mark.parametrize("kind", ["ties", "close", "tiny", "small", "huge", "large", "spread", "special", "zero"])
@pytest.mark.parametrize("d,k", [(3, 20), (14, 127), (30, 9), (64, 40)])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_labels_of_hard_values(oracle, kind, d, k, dt):
    with np.errstate(all="ignore"):
        X, C = _hard(kind, d, 700, k, np.random.default_rng(d + k), dt)
        np.testing.assert_array_equal(_labels(X, C), oracle.assignment(X, C))


@pytest.mark.parametrize("seed", range(4))
def test_float64_labels_with_given_half_norms(oracle, seed):
    # half norms that do not belong to the centroids: the bound takes them as given
    rng = np.random.default_rng(seed)
    X, C = rng.standard_normal((6, 3000)), rng.standard_normal((6, 17))
    hn = rng.standard_normal(17) * 10.0 ** rng.integers(-8, 9, 17)
    if seed == 3:
        hn[4], hn[9] = np.inf, np.nan
    np.testing.assert_array_equal(_labels(X, C, hn), oracle.assignment(X, C, hn))


@pytest.mark.parametrize("d,k", [(1, 3), (14, 127), (15, 40), (16, 200), (31, 20), (33, 300), (64, 64), (64, 400),
                                 (14, 2000), (100, 70), (128, 150), (148, 40), (160, 33)])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("it", ["int32", "int64"])
def test_weighted_iterations_equal_the_oracles(oracle, d, k, dt, it):
    # small integers: every sum is exact, whatever path adds it
    import torch

    import kmeans_dpcpp_gb300 as kdp

    rng = np.random.default_rng(d + k)
    n = 20_011
    X = rng.integers(-9, 10, (d, n)).astype(dt)
    w = rng.choice([1.0, 1.0, 2.0, 0.5, 3.0], n).astype(dt)
    C0 = np.ascontiguousarray(X[:, rng.choice(n, k, replace=False)])
    it_o, lab_o, C_o, _, _ = oracle.kmeans_lloyd_driver(X, w, C0, 0.0, 2)
    cur, res = _gpu(C0.copy()), _gpu(np.zeros_like(C0))
    lab = torch.empty(n, dtype=getattr(torch, it), device="cuda")
    n_iter, _ = kdp.kmeans_lloyd_driver(_gpu(X), _gpu(w), cur, lab, res, 0.0, False, 2, 8, 128, 0.7, None)
    assert n_iter == it_o
    np.testing.assert_array_equal(res.cpu().numpy(), C_o)
    np.testing.assert_array_equal(lab.cpu().numpy(), lab_o)


@pytest.mark.parametrize("d,k,copies", [(14, 16, 200), (14, 16, 3), (32, 256, 300), (64, 90, 152), (70, 30, 400),
                                        (100, 300, 160), (150, 20, 200)])
def test_fused_step_with_many_and_few_copies(oracle, d, k, copies):
    import torch

    import kmeans_dpcpp_gb300 as kdp

    rng = np.random.default_rng(d + k + copies)
    n = 30_005
    X = rng.integers(-9, 10, (d, n)).astype(np.float32)
    w = rng.choice([1.0, 2.0, 0.5], n).astype(np.float32)
    C = np.ascontiguousarray(X[:, rng.choice(n, k, replace=False)])
    lab_o, sums_o, sizes_o = oracle.fused_lloyd_single_step(X, w, C)
    Cg = _gpu(C)
    hn = torch.empty(k, device="cuda")
    kdp.half_l2_norm_squared(Cg, hn, 128, None)
    lab = torch.empty(n, dtype=torch.int32, device="cuda")
    cc, sc = torch.zeros((copies, d, k), device="cuda"), torch.zeros((copies, k), device="cuda")
    kdp.fused_lloyd_single_step(_gpu(X), _gpu(w), Cg, hn, lab, cc, sc, 8, 128, None)[0].wait()
    np.testing.assert_array_equal(lab.cpu().numpy(), lab_o)
    # sums of multiples of 1/2 below 2^23: exact in float32
    np.testing.assert_array_equal(cc.sum(0).cpu().numpy(), sums_o)
    np.testing.assert_array_equal(sc.sum(0).cpu().numpy(), sizes_o)


@pytest.mark.parametrize("copies", [1, 7, 8, 9, 16, 17, 130, 1000])
@pytest.mark.parametrize("d,k", [(1, 1), (3, 11), (14, 33)])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_copies_of_any_number_are_reduced(copies, d, k, dt):
    # small integers: exact sums in any order; cluster 0 stays empty
    import torch

    import kmeans_dpcpp_gb300 as kdp

    rng = np.random.default_rng(copies + d + k)
    cc, sc = rng.integers(-4, 5, (copies, d, k)).astype(dt), rng.integers(1, 4, (copies, k)).astype(dt)
    sc[:, 0] = 0
    out, sizes = _gpu(np.full((d, k), np.nan, dt)), _gpu(np.full(k, np.nan, dt))
    empty, n_empty = torch.full((k,), -1, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda")
    kdp.reduce_centroids_data(_gpu(sc), _gpu(cc), sizes, out, empty, n_empty, 128, None)[0].wait()
    np.testing.assert_array_equal(out.cpu().numpy(), cc.sum(0))
    np.testing.assert_array_equal(sizes.cpu().numpy(), sc.sum(0))
    assert n_empty.item() == 1 and empty[0].item() == 0
