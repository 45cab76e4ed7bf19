"""The streamed traversal (waves of many paths) against the plain one: full frames equal the same
frame rendered in row bands bit for bit, where each frame is large enough to stream, even over a few
triangles, and each band small enough not to. Scenes where streaming can go wrong: a lone leaf, few
triangles, exact distance ties, one-sided surfaces, traversal stacks far deeper than their shared
part, rays that miss everything, media.
"""

import numpy as np
import pytest

from minirender_b200 import scene as sc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from minirender_b200 import api as a
    return a


def soup(count, size, seed=1, copies=1, double_sided=True):
    """`count` random triangles of about `size` in a unit cube, every one `copies` times."""
    rng = np.random.default_rng(seed)
    centers = rng.uniform(-0.5, 0.5, (count, 1, 3))
    positions = (centers + rng.normal(scale=size, size=(count, 3, 3))).astype(np.float32)
    positions = np.repeat(positions, copies, axis=0)
    normal = np.cross(positions[:, 1] - positions[:, 0], positions[:, 2] - positions[:, 0])
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    n = len(positions)
    mesh = sc.MeshData(positions.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(n, 3),
                       np.repeat(normal[:, None], 3, axis=1).astype(np.float32), None)
    doc = sc.SceneDocument()
    doc.camera = sc.Camera((0.1, 0.2, 2.5), (0, 0, 0), vertical_fov_degrees=35.0)
    doc.environment = (0.4, 0.5, 0.6)
    doc.directional_lights = [sc.DirectionalLight((0.0, -1.0, 0.0), (1, 1, 1), 2.0)]
    doc.materials = [sc.Material("diffuse", (0.6, 0.5, 0.4), double_sided=double_sided)]
    doc.meshes = [mesh]
    doc.objects = [sc.SceneObject(0, 0)]
    return doc


def fog(doc):
    doc.media = [sc.MediumRegion((-0.4, -0.4, -0.4), (0.4, 0.4, 0.4), (0.1, 0.2, 0.3), (1.0, 1.0, 1.0),
                                 0.3)]
    return doc


SCENES = {
    "one triangle": lambda: soup(1, 0.3),
    "lone leaf": lambda: soup(4, 0.3),
    "two leaves": lambda: soup(5, 0.3),
    "seventeen": lambda: soup(17, 0.3),
    "ties": lambda: soup(300, 0.1, copies=3),
    "one-sided": lambda: soup(2000, 0.05, double_sided=False),
    # Every node's four boxes overlap, so a descent stacks up to three entries a level.
    "deep stacks": lambda: soup(20_000, 0.4),
    "deep stacks in fog": lambda: fog(soup(8_000, 0.4)),
    "field": lambda: sc.sphere_field(9, 8.0, 4, subdivisions=2),
}


@pytest.mark.parametrize("name", list(SCENES))
def test_streamed_frame_equals_row_bands(api, name):
    scene = api.Scene(SCENES[name]().snapshot())
    render = api.RenderSettings(331, 240, 27, 11)  # 2,144,880 paths: streamed
    tracer = api.PathTracer(scene, api.IntegratorSettings("mis", 6, True, 3))
    image, counts = tracer.render(render)
    bands, total = [], {k: 0 for k in counts if not k.endswith("tests")}
    for begin in range(0, 240, 48):  # 428,976 paths a band: not streamed
        band, part = tracer.render_rows(render, begin, begin + 48, statistics=True)
        bands.append(band)
        total = {k: v + part[k] for k, v in total.items()}
    np.testing.assert_array_equal(image, np.concatenate(bands))
    assert total == {k: counts[k] for k in total}
    batch, codes, _ = api.render_batch(
        [api.BatchJob(scene, render, tracer.settings),
         api.BatchJob(scene, api.RenderSettings(331, 240, 1, 12), tracer.settings)])
    assert codes == [0, 0]
    np.testing.assert_array_equal(batch[0], image)
