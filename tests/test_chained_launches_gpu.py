"""Launches that may be set up while the kernel before them still runs: results
must not depend on it, whether another library's kernel wrote the inputs just
before, the calls are captured into a graph and replayed on new inputs, or many
fits run on streams of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(20_000, 5, 7), (30_001, 40, 200), (50_000, 16, 64)]


def _pass(kdp, X, C, b):
    import torch

    s = torch.cuda.current_stream()
    kdp.half_l2_norm_squared(C, b["hn"], 128, s)
    kdp.assignment(X, C, b["hn"], b["lab"], 8, 128, s)
    kdp.compute_centroid_to_sample_distances(X, C, b["dist"], 128, 8, s)


def _buffers(n, k):
    import torch

    return dict(hn=torch.empty(k, device="cuda"), lab=torch.empty(n, dtype=torch.int32, device="cuda"),
                dist=torch.empty((k, n), device="cuda"))


@pytest.mark.parametrize("n,d,k", SIZES)
def test_captured_passes_equal_eager_ones(oracle, n, d, k):
    import torch

    import kmeans_dpcpp_gb300 as kdp

    g = torch.Generator(device="cuda").manual_seed(n)
    X, C = torch.zeros((d, n), device="cuda"), torch.zeros((d, k), device="cuda")
    b = _buffers(n, k)
    _pass(kdp, X, C, b)  # kernel attributes are set outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=s):
        X.add_(0.0)  # another library's kernel in front
        _pass(kdp, X, C, b)
    for _ in range(3):
        X.copy_(torch.randn((d, n), generator=g, device="cuda"))
        C.copy_(X[:, :k])
        graph.replay()
        torch.cuda.synchronize()
        got = {q: v.clone() for q, v in b.items()}
        X.mul_(1.0)
        _pass(kdp, X, C, b)
        torch.cuda.synchronize()
        for q in b:
            assert torch.equal(got[q], b[q]), q
        np.testing.assert_array_equal(got["lab"].cpu().numpy(), oracle.assignment(X.cpu().numpy(), C.cpu().numpy()))


@pytest.mark.parametrize("form", ["plain", "mixed-fp16"])
def test_inputs_written_just_before(oracle, form):
    """Each fit's inputs are made by kernels enqueued right in front of it, on
    one of four streams; integer data, so every sum is exact."""
    import torch

    import kmeans_dpcpp_gb300 as kdp

    rng = np.random.default_rng(4)
    streams, jobs = [torch.cuda.Stream() for _ in range(4)], []
    for q in range(12):
        n, d, k = SIZES[q % 3]
        X = rng.integers(-8, 9, (d, n)).astype(np.float32)
        C0 = np.ascontiguousarray(X[:, rng.choice(n, k, replace=False)])
        jobs.append((X, C0, oracle.kmeans_lloyd_driver(X, np.ones(n, np.float32), C0, 0.0, 4)))
    for q, (X, C0, want) in enumerate(jobs):
        with torch.cuda.stream(streams[q % 4]):
            half = torch.from_numpy(X).cuda() * 0.5
            Xg = torch.empty_like(half)
            C, w = torch.from_numpy(C0).cuda(), torch.empty(X.shape[1], device="cuda")
            res, lab = torch.empty_like(C), torch.empty(X.shape[1], dtype=torch.int64, device="cuda")
            w.fill_(1.0)
            torch.add(half, half, out=Xg)
            it, _ = kdp.kmeans_lloyd_driver(Xg, w, C, lab, res, 0.0, False, 4, 8, 128, 0.7, streams[q % 4],
                                            form=form)
            streams[q % 4].synchronize()
        assert it == want[0]
        np.testing.assert_array_equal(res.cpu().numpy(), want[2])
        np.testing.assert_array_equal(lab.cpu().numpy(), want[1])
