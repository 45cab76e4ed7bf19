"""Waves whose paths fit on the device at once run whole paths in one launch; the batched engine
runs the same jobs as a wavefront. Images and path counts are equal bit for bit, from one path to
both sides of the largest such wave, for every integrator mode, depth limits, media and two levels.
"""

import numpy as np
import pytest

from minirender_b200 import scene as sc

pytestmark = pytest.mark.gpu

COUNTS = ("paths", "shadow_rays", "scattering_events", "roulette_terminations",
          "medium_scattering_events")


@pytest.fixture(scope="module")
def api():
    from minirender_b200 import api as a
    return a


def foggy_room():
    doc = sc.job_scene(20_000, 17)
    doc.media = [sc.MediumRegion((-0.4, 0.0, -0.4), (0.4, 0.6, 0.4), (0.2, 0.3, 0.4),
                                 (0.8, 0.8, 0.8), 0.2)]
    return doc


SCENES = {"box": sc.cornell_box, "room": lambda: sc.job_scene(20_000, 3), "foggy": foggy_room,
          "field": lambda: sc.sphere_field(6, 8.0, 4, subdivisions=2)}
# 148 SMs x 4 blocks x 128 lanes hold 75,776 paths: 296 x 256 fits exactly, 257 x 295 does not.
SIZES = [(1, 1, 1), (5, 7, 1), (128, 1, 1), (43, 3, 1), (33, 31, 5), (296, 256, 1), (257, 295, 1)]


@pytest.mark.parametrize("two_level", [False, True])
@pytest.mark.parametrize("name", list(SCENES))
def test_whole_paths_equal_the_wavefront(api, name, two_level):
    scene = api.Scene(SCENES[name]().snapshot(), two_level=two_level)
    cases = [(size, api.IntegratorSettings("mis", 8, True, 3)) for size in SIZES]
    cases += [((61, 37, 3), api.IntegratorSettings(mode, depth, roulette, 2))
              for mode, depth, roulette in (("light", 5, True), ("bsdf", 12, True), ("mis", 0, True),
                                            ("mis", 1, False), ("mis", 128, True))]
    for k, ((width, height, spp), settings) in enumerate(cases):
        render = api.RenderSettings(width, height, spp, 5 + k)
        image, counts = api.PathTracer(scene, settings).render(render)
        batch, codes, info = api.render_batch([api.BatchJob(scene, render, settings)])
        assert codes == [0]
        np.testing.assert_array_equal(image, batch[0])
        assert {c: counts[c] for c in COUNTS} == {c: info["paths"][c] for c in COUNTS}
