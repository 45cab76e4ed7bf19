"""Device memory of a flattened scene: its wide nodes take no more than 128 bytes for each interior node of
the binary tree, the rest is what the layout says.
"""

import pytest

from minirender_b200 import scene as sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("triangles", [20_000, 60_000])
def test_device_bytes(triangles):
    from minirender_b200 import api
    scene = api.Scene(sc.job_scene(triangles, 3).snapshot())
    nodes, order, count = scene.export_bvh()
    slots, prims = len(order), scene.statistics()["triangles"]
    interior = (count - 1) // 2
    tables = 1 << 16  # materials, lights and their distribution
    layout = 48 * slots + 48 * prims + 36 * count + 4 * slots + 4 * prims
    assert layout < scene.device_bytes() <= layout + 128 * (interior + 2) + tables
