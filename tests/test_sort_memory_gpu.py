"""Sums sorted by label whose tile and histogram take just under the 48 KB of
shared memory that a kernel gets without asking, its own static arrays included.
A process of its own: another shape's launch may have raised the limit before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FITS = """
import sys
import numpy as np, torch
import kmeans_dpcpp_gb300 as kdp
d, form = int(sys.argv[1]), sys.argv[2]
sms = torch.cuda.get_device_properties(0).multi_processor_count
n = sms * 4 * 4064  # tiles of 4064 samples in one round of all resident CTAs
g = torch.Generator(device="cuda").manual_seed(1)
X = torch.randint(-64, 65, (d, n), generator=g, device="cuda").float()
w = torch.ones(n, device="cuda")
for k in (79, 87, 88, 95, 96):  # 12 B x 4064 + 4 B x (k + 1): 49,088 ... 49,156 bytes
    C = X[:, :k].contiguous()
    lab = torch.empty(n, dtype=torch.int32, device="cuda")
    kdp.kmeans_lloyd_driver(X, w, C, lab, torch.empty_like(C), 0.0, False, 1, 8, 128, 0.7, None, form=form)
    # labels of the first centroids; their means are the next centroids
    first = X[:, :k].contiguous()
    hn = torch.empty(k, device="cuda")
    s = torch.cuda.current_stream()
    kdp.half_l2_norm_squared(first, hn, 128, s)
    kdp.assignment(X, first, hn, lab, 8, 128, s)
    sums = torch.zeros((k, d), dtype=torch.float64, device="cuda").index_add_(0, lab.long(), X.t().double())
    size = torch.bincount(lab.long(), minlength=k).double()
    mean = (sums / size[:, None]).t().float()
    # exact sums up to 32 features; beyond, integers far below 2^24
    assert torch.equal(C, mean), (k, (C - mean).abs().max())
"""


@pytest.mark.parametrize("d,form", [(4, "mixed-fp16"), (33, "mixed-bf16")])
def test_shapes_at_the_default_limit(d, form):
    env = dict(os.environ, KMC_TUNE="0", PYTHONPATH=REPO)
    subprocess.run([sys.executable, "-c", FITS, str(d), form], env=env, cwd=REPO, check=True, timeout=600)
