"""The work queue of the batched engine's instances that are taken in panels (no
GPU): the engine's own planner, its items pulled by CPU threads."""
import ctypes
import itertools
import threading

import numpy as np
import pytest

from kmeans_dpcpp_gb300 import capi


def _items(n, d, k, transform, sms):
    L = capi.lib()

    def P(a, t):
        return np.ascontiguousarray(a).ctypes.data_as(ctypes.POINTER(t))

    total = ctypes.c_int64()
    a = [np.ascontiguousarray(v, dtype=np.int64) for v in (n, d, k)]
    args = (len(n), *[P(v, ctypes.c_int64) for v in a], transform, sms)
    capi.check(L.kmc_debug_batch_panel_items(*args, 0, None, None, None, ctypes.byref(total)))
    m = total.value
    inst, tiles, first = np.empty(m, np.int32), np.empty(m, np.int32), np.empty(m, np.int64)
    capi.check(L.kmc_debug_batch_panel_items(*args, m, P(inst, ctypes.c_int32), P(tiles, ctypes.c_int32),
                                             P(first, ctypes.c_int64), ctypes.byref(total)))
    return inst, tiles, first


def _problem(seed, transform):
    rng = np.random.default_rng(seed)
    count = 40
    n = rng.integers(0, 300_000, count)
    n[:4] = [0, 1, 512, 513]  # empty, one sample, one round, one more
    return n, rng.integers(1, _most(transform) + 1, count), rng.integers(1, 513, count)


def _round(d, transform):
    """128-sample tiles that a CTA's warps take at once: 16, 12 or 8 warps of 32
    samples, as many as fit 224 KB beside two blocks of 64 centroids."""
    dp = d + d % 2
    for warps in (16, 12, 8):
        if 4 * (2 * 64 * (dp + 1) + warps * 32 * (dp + 1 + 33 * transform)) <= 224 * 1024:
            return warps // 4
    return 0


def _most(transform):
    return max(d for d in range(1, 300) if _round(d, transform))


@pytest.mark.parametrize("transform", [0, 1])
@pytest.mark.parametrize("sms", [1, 148, 152])
def test_every_tile_is_pulled_once(transform, sms):
    n, d, k = _problem(5 + transform, transform)
    inst, tiles, first = _items(n, d, k, transform, sms)
    assert np.all(tiles >= 1)
    seen = [np.zeros(-(-int(v) // 128), np.int32) for v in n]
    lock, counter = threading.Lock(), itertools.count()

    def worker():
        while True:
            with lock:
                j = next(counter)
            if j >= len(inst):
                return
            for t in range(first[j], first[j] + tiles[j]):
                with lock:
                    seen[inst[j]][t] += 1

    threads = [threading.Thread(target=worker) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for q in range(len(n)):
        assert np.all(seen[q] == 1), q


@pytest.mark.parametrize("transform", [0, 1])
def test_items_are_whole_rounds_and_the_heaviest_come_first(transform):
    n, d, k = _problem(11, transform)
    inst, tiles, first = _items(n, d, k, transform, 152)
    ends = -(-n // 128)
    last = first + tiles == ends[inst]
    per = {}
    for j in range(len(inst)):
        if not last[j]:
            per.setdefault(int(inst[j]), set()).add(int(tiles[j]))
    for q, sizes in per.items():
        assert len(sizes) == 1  # an instance's items are equal, but for its last
        size = sizes.pop()
        assert size % _round(d[q], transform) == 0 and size <= 64 * _round(d[q], transform)
        assert all(tiles[j] <= size for j in range(len(inst)) if inst[j] == q)
    # an instance's items in order, its smaller last one behind them
    for q in per:
        mine = np.flatnonzero(inst == q)
        assert np.all(np.diff(tiles[mine]) <= 0)
        assert np.all(np.diff(first[mine]) > 0)
    work = tiles.astype(np.float64) * 128 * d[inst] * (k[inst] + 100)
    head, tail = work[: len(work) // 4].mean(), work[-(len(work) // 4):].mean()
    assert head > tail


def test_instances_beyond_the_panels_are_refused():
    total = ctypes.c_int64()
    one = (ctypes.c_int64 * 1)(100)
    for d, transform in ((_most(0) + 1, 0), (_most(1) + 1, 1), (0, 0)):
        rc = capi.lib().kmc_debug_batch_panel_items(1, one, (ctypes.c_int64 * 1)(d), one, transform, 152, 0, None,
                                                    None, None, ctypes.byref(total))
        assert rc == 1 and "not taken in panels" in capi.lib().kmc_last_error().decode()
