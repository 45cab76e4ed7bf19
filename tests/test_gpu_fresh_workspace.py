"""A call's first wave on a fresh workspace sorts its rays while the caller has work pending on the
legacy default stream and the memory held other values before. The same call again, on the pooled
workspace, gives the same radiance.
"""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# A process of its own, so that no earlier call's workspace is pooled. 300,000 paths over more than
# 4,096 triangle slots are sorted.
PROGRAM = """
import numpy as np
import torch
from minirender_b200 import api, scene as sc
scene = api.Scene(sc.job_scene(12_000, 5).snapshot())
tracer = api.PathTracer(scene, api.IntegratorSettings("mis", 4, True, 3))
n = 300_000
rng = np.random.default_rng(1)
o = rng.uniform((-0.45, 0.05, -0.45), (0.45, 0.95, 0.45), (n, 3)).astype(np.float32)
d = rng.normal(size=(n, 3))
d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
keys = np.stack([np.full(n, 7), np.arange(n), np.zeros(n)], 1).astype(np.uint64)
a = torch.randn(8192, 8192, device="cuda")
used = torch.full((1 << 28,), -1, dtype=torch.int32, device="cuda")
torch.cuda.synchronize()
del used
torch.cuda.empty_cache()
for _ in range(20):
    a = a @ a * 1e-4
first, counts = tracer.trace(o, d, 1e-4, np.inf, keys)
torch.cuda.synchronize()
again, counts_again = tracer.trace(o, d, 1e-4, np.inf, keys)
np.testing.assert_array_equal(first, again)
for key in ("paths", "shadow_rays", "scattering_events", "roulette_terminations"):
    assert counts[key] == counts_again[key], key
assert first.mean() > 0
print("equal")
"""


def test_first_sorted_wave_behind_pending_legacy_work():
    result = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert result.returncode == 0 and result.stdout.strip() == "equal", result.stderr
