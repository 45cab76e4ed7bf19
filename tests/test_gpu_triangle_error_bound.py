"""The triangle test refuses a hit no farther than its error bound, also where the quotient that is the
bound is subnormal and rounds up to the distance. The vertices were found by evaluating the test's FP32
steps in numpy: of each triangle (distance, bound before rounding) is about (1.26e-42, 1.2594e-42),
(1.885e-42, 1.8849e-42) and (3.704e-42, 3.7034e-42).
"""

import numpy as np
import pytest

from minirender_b200 import scene as sc

pytestmark = pytest.mark.gpu

Z = [("0x1.7a52160000000p-121", "-0x1.77a0fe0000000p-122", "-0x1.7d01de0000000p-122"),
     ("0x1.1b2d380000000p-120", "-0x1.23dd4e0000000p-121", "-0x1.127c240000000p-121"),
     ("0x1.161ed40000000p-119", "-0x1.fea16c0000000p-121", "-0x1.2cebfa0000000p-120")]


@pytest.mark.parametrize("z", Z)
@pytest.mark.parametrize("two_level", [False, True])
def test_distance_at_a_subnormal_bound_is_refused(z, two_level):
    from minirender_b200 import api
    doc = sc.SceneDocument()
    doc.materials = [sc.Material()]
    doc.meshes = [sc.MeshData(np.float32([(-1e6, -1e6, float.fromhex(z[0])), (2e6, -1e6, float.fromhex(z[1])),
                                          (-1e6, 2e6, float.fromhex(z[2]))]),
                              np.uint32([(0, 1, 2)]), np.tile(np.float32((0, 0, 1)), (1, 3, 1)), None)]
    doc.objects = [sc.SceneObject(0, 0)]
    scene = api.Scene(doc.snapshot(), two_level=two_level)
    o, d = np.zeros((1, 3), np.float32), np.float32([(0, 0, 1)])
    assert scene.intersect(o, d, 0.0, np.inf)[0]["primitive"][0] == 0xffffffff
    assert not scene.occluded(o, d, 0.0, np.inf)[0][0]
    above = o + np.float32((0, 0, -1))  # an ordinary distance
    assert scene.intersect(above, d, 0.0, np.inf)[0]["primitive"][0] == 0
