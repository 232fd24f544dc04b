"""Relocation of several empty clusters: groups of eight moves, ranks by a warp per
sample, and divisions spread over more thread blocks than the samples need.

Samples are small integers, so distances, sums and moves are exact in any order and
the centroids have one right value."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, d, sources, empty, dt):
    """Samples spread around `sources` centroids; `empty` duplicates of the first
    one, listed between and behind the others, get none."""
    rng = np.random.default_rng(n + 7 * d + 31 * sources + 101 * empty)
    k = sources + empty
    which = np.zeros(k, np.int64)  # the source that a centroid stands for
    place = np.concatenate([[0], np.sort(rng.choice(np.arange(1, k), sources - 1, replace=False))])
    which[place] = np.arange(sources)
    C = np.zeros((d, k), dt)
    C[0] = 64 * which
    lab = place[rng.integers(0, sources, n)]
    lab[:3 * sources] = np.repeat(place, 3)  # no source loses all of its samples at once
    X = rng.integers(-6, 7, (d, n)).astype(dt)
    X[:, :3 * sources] = 0
    X[0] = C[0, lab]
    return X, C, lab, np.square((X - C[:, lab]).astype(np.float64)).sum(axis=0), np.setdiff1d(np.arange(k), place)


def _run(form, dt, X, C0):
    import torch

    from kmeans_dpcpp_gb300 import capi

    L, (d, n), k = capi.lib(), X.shape, C0.shape[1]
    Xg, cur = torch.from_numpy(X).cuda(), torch.from_numpy(C0.copy()).cuda()
    w, res = torch.ones(n, dtype=Xg.dtype, device="cuda"), torch.empty_like(cur)
    lab = torch.empty(n, dtype=torch.int32, device="cuda")
    h = ctypes.c_void_p()
    create = L.kmc_fit_create_f64_i32 if dt == np.float64 else L.kmc_fit_create_f32_i32
    capi.check(create(Xg.data_ptr(), w.data_ptr(), cur.data_ptr(), lab.data_ptr(), res.data_ptr(), n, d, k, 0.0, 1,
                      {"plain": 0, "fp16": 2}[form], torch.cuda.current_stream().cuda_stream, ctypes.byref(h)))
    try:
        capi.check(L.kmc_fit_run(h))
    finally:
        capi.check(L.kmc_fit_destroy(h))
    torch.cuda.synchronize()
    return cur.cpu().numpy()


@pytest.mark.parametrize("n,d,sources,empty", [
    (500, 3, 1, 1), (500, 3, 1, 7), (500, 3, 1, 8), (500, 3, 1, 9), (500, 5, 1, 17),  # one source
    (700, 4, 3, 16), (700, 33, 5, 31), (9000, 4, 6, 300),
    (600, 140, 12, 188), (1300, 100, 17, 513),  # more blocks for the divisions
])
@pytest.mark.parametrize("form,dt", [("plain", np.float32), ("plain", np.float64), ("fp16", np.float32)])
def test_the_farthest_samples_move_in_order(n, d, sources, empty, form, dt):
    X, C0, lab, dist, empties = _problem(n, d, sources, empty, dt)
    k = sources + empty
    sums = np.stack([X[:, lab == j].astype(np.float64).sum(axis=1) for j in range(k)], axis=1)
    size = np.bincount(lab, minlength=k).astype(np.float64)
    assert np.array_equal(np.flatnonzero(size == 0), empties)
    for cl, i in zip(empties, np.lexsort((np.arange(n), -dist))[:empty]):
        sums[:, lab[i]] -= X[:, i]
        size[lab[i]] -= 1
        sums[:, cl], size[cl] = X[:, i], 1
    want = sums.astype(dt) / size.astype(dt)
    np.testing.assert_array_equal(_run(form, dt, X, C0), want)
