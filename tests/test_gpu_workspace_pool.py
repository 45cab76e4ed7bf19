"""Idle pooled workspaces give way to any other allocation of the library, and the workspaces of a
batch's lanes stay pooled when a batch of another shape follows, however large their waves.
"""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run(program):
    """In a process of its own: the pools are the process's."""
    result = subprocess.run([sys.executable, "-c", program], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert result.returncode == 0 and result.stdout.strip() == "done", result.stderr


# A frame of 8,388,608 paths leaves a workspace of 2 GiB in the pool; the caller then holds all but 256 MiB
# of the device's memory, and the call needs some 460 MiB.
FULL = """
import numpy as np
import torch
from minirender_b200 import api, scene as sc
tracer = api.PathTracer(api.Scene(sc.job_scene(500, 5).snapshot()), api.IntegratorSettings("mis", 2, True, 3))
tracer.render(api.RenderSettings(2048, 2048, 2, 1))
rng = np.random.default_rng(1)
d = rng.normal(size=(8_000_000, 3)).astype(np.float32)
d /= np.linalg.norm(d, axis=1, keepdims=True)
o = np.full_like(d, 0.3)
few = api.Scene(sc.job_scene(500, 5).snapshot()).intersect(o[:1000], d[:1000])[0]
torch.cuda.synchronize()
free, _ = torch.cuda.mem_get_info()
held = torch.empty(free - (256 << 20), dtype=torch.uint8, device="cuda")
%s
print("done")
"""
CALLS = {
    "query": """
hits, _ = tracer.scene.intersect(o, d)
np.testing.assert_array_equal(hits[:1000], few)
""",
    "scene": """
rng = np.random.default_rng(2)
v = rng.uniform(-1, 1, (1_500_000, 3, 3)).astype(np.float32)
n = np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
n /= np.linalg.norm(n, axis=1, keepdims=True)
doc = sc.SceneDocument()
doc.materials = [sc.Material()]
doc.meshes = [sc.MeshData(v.reshape(-1, 3), np.arange(4_500_000, dtype=np.uint32).reshape(-1, 3),
                          np.repeat(n[:, None], 3, axis=1).astype(np.float32), None)]
doc.objects = [sc.SceneObject(0, 0)]
assert api.Scene(doc.snapshot()).statistics()["triangles"] == 1_500_000
""",
    "server": """
with api.RenderServer(1 << 30, batch=api.BatchSettings(wave_paths=1 << 16, concurrent_waves=1)) as server:
    job = server.submit(tracer.scene, api.RenderSettings(3200, 3200, 1, 1), tracer.settings)
    assert server.wait(job) and server.info(job)["status"] == 0, server.info(job)
""",
}


@pytest.mark.parametrize("call", list(CALLS))
def test_allocations_take_the_place_of_idle_workspaces(call):
    run(FULL % CALLS[call])


LARGE_LANES = """
import torch
from minirender_b200 import api, scene as sc
scene = api.Scene(sc.job_scene(500, 5).snapshot())
jobs = [api.BatchJob(scene, api.RenderSettings(64, 64, 2, 1), api.IntegratorSettings("mis", 2, True, 3))]
small, large = (api.BatchSettings(wave_paths=1 << k, concurrent_waves=4) for k in (16, 24))
assert api.render_batch(jobs, small)[1] == [0]  # loads the kernels
free = torch.cuda.mem_get_info()[0]
for lanes in (large, small, large, small):  # a batch of another shape gives the lanes' workspaces back
    assert api.render_batch(jobs, lanes)[1] == [0]
    # Four workspaces of 2^24 paths, of more than 192 bytes each (a path's records).
    assert free - torch.cuda.mem_get_info()[0] > 4 * 192 * (1 << 24)
print("done")
"""


def test_lanes_of_large_waves_stay_pooled():
    run(LARGE_LANES)
