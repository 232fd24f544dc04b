"""The autotuner's cache file: which fits are tuned.  Each case runs in a process
of its own, because the file is read once per process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FIT = """
import sys, numpy as np, torch
import kmeans_dpcpp_gb300 as kdp
n, d, k, dt, form = int(sys.argv[1]), int(sys.argv[2]), int(sys.argv[3]), sys.argv[4], sys.argv[5]
g = torch.Generator(device="cuda").manual_seed(1)
X = torch.randn((d, n), generator=g, device="cuda", dtype=getattr(torch, dt))
C = X[:, :k].contiguous()
lab = torch.empty(n, dtype=torch.int32, device="cuda")
kdp.kmeans_lloyd_driver(X, torch.ones(n, device="cuda", dtype=X.dtype), C, lab, torch.empty_like(C), 0.0, False,
                        1, 8, 128, 0.7, None, form=form)
"""


def _lines(cache, *args):
    env = dict(os.environ, KMC_TILE_CACHE=str(cache), PYTHONPATH=REPO)
    env.pop("KMC_TUNE", None)
    subprocess.run([sys.executable, "-c", FIT, *map(str, args)], env=env, cwd=REPO, check=True, timeout=300)
    return cache.read_text().split("\n") if cache.exists() else []


# (n, d, k, dtype): fits whose labels or sums run in the tiles, whose width is
# chosen by timing, and fits that never reach them
TILES = [(4000, 64, 400, "float64"), (4000, 14, 1000, "float64"), (3000, 160, 20, "float32"),
         (3000, 160, 20, "float64")]
OTHERS = [(4000, 64, 100, "float64"), (4000, 64, 400, "float32"), (4000, 148, 3, "float32")]


@pytest.mark.parametrize("n,d,k,dt", TILES + OTHERS)
def test_the_width_is_timed_where_the_tiles_run(tmp_path, n, d, k, dt):
    lines = _lines(tmp_path / "tiles.txt", n, d, k, dt, "plain")
    bucket = 1
    while bucket < k:
        bucket *= 2
    tag = f"{d} {bucket} fit-{'f64' if dt == 'float64' else 'f32'} "
    assert any(q.startswith(tag) for q in lines) == ((n, d, k, dt) in TILES)
