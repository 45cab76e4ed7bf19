"""Traversal at the limits of accepted imported trees, on every route of the flattened traversal:
queries and explicit paths in few (one launch of whole paths) and many (streamed) paths.
"""

import ctypes as C

import numpy as np
import pytest

from minirender_b200 import _abi, scene as sc

pytestmark = pytest.mark.gpu

NODE = np.dtype([("minimum", "<f4", 3), ("maximum", "<f4", 3), ("first", "<u4"), ("right", "<u4"),
                 ("count", "<u4")])


@pytest.fixture(scope="module")
def api():
    from minirender_b200 import api as a
    return a


def mesh(triangles):
    """MeshData of (n, 3, 3) vertices, each triangle with corners of its own."""
    n = len(triangles)
    normal = np.cross(triangles[:, 1] - triangles[:, 0], triangles[:, 2] - triangles[:, 0])
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    return sc.MeshData(triangles.reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.uint32).reshape(n, 3),
                       np.repeat(normal[:, None], 3, axis=1).astype(np.float32), None)


def imported(api, triangles, tree):
    """The scene of `triangles`, black in a gray environment, under `tree`: a triangle index, or a pair
    of trees."""
    doc = sc.SceneDocument()
    doc.camera = sc.Camera((0, 0, -1.0), (0, 0, 0), vertical_fov_degrees=40.0)
    doc.environment = (0.5, 0.5, 0.5)
    doc.materials = [sc.Material("diffuse", (0, 0, 0), double_sided=True)]
    doc.meshes, doc.objects = [mesh(triangles)], [sc.SceneObject(0, 0)]
    nodes, order = [], []

    def add(t):  # the node's index
        at = len(nodes)
        nodes.append(None)
        if isinstance(t, tuple):
            a = add(t[0])
            b = add(t[1])
            nodes[at] = (np.minimum(nodes[a][0], nodes[b][0]), np.maximum(nodes[a][1], nodes[b][1]), a, b, 0)
        else:
            nodes[at] = (vertices[t].min(0), vertices[t].max(0), len(order), 0, 1)
            order.append(t)
        return at

    vertices = triangles.astype(np.float32)
    add(tree)
    packed, order = np.array(nodes, NODE), np.array(order, np.uint32)
    desc = _abi.BvhDesc(C.cast(packed.ctypes.data, C.POINTER(_abi.BvhNode)), len(packed),
                        order.ctypes.data_as(C.POINTER(C.c_uint32)), len(order))
    return api.Scene(doc.snapshot(), desc)


def axis_rays(n, axis):
    """`n` rays from the origin, `axis` of them along +z (spread over the rays), the others along -z."""
    o, d = np.zeros((n, 3), np.float32), np.zeros((n, 3), np.float32)
    along = np.zeros(n, bool)
    along[::n // axis] = True
    d[:, 2] = np.where(along, 1.0, -1.0)
    keys = np.stack([np.full(n, 3), np.arange(n), np.zeros(n)], 1).astype(np.uint64)
    return o, d, keys, along


PATHS = [1 << 10, 1 << 21]  # one launch of whole paths; streamed, even over few triangles


def nested(covers):
    """Three triangles across the axis at each of 64 nested levels, each level 1.5 times the one inside
    it, as the deepest tree that is accepted: every wide node's nearest child is the rest of the tree
    and its other three are stacked, 189 in all. Where `covers` is false the axis passes the
    triangle by, through its box."""
    inside = np.array([(-1, -1), (3, -1), (-1, 3)], float)
    beside = np.array([(-1, -1.5), (1.5, -1.5), (1.5, 1)], float)
    triangles = []

    def triangle(level, j):
        scale = 1.5 ** (63 - level)
        xy = (inside if covers(level, j) else beside) * scale
        triangles.append(np.column_stack([xy, np.full(3, scale * (1 + 0.05 * j))]))
        return len(triangles) - 1

    tree = (triangle(63, 0), triangle(63, 1))
    tree = ((triangle(62, 0), triangle(62, 1)), tree)
    for level in range(61, -1, -1):
        tree = (((triangle(level, 0), triangle(level, 1)), triangle(level, 2)), tree)
    return np.array(triangles), tree


@pytest.mark.parametrize("paths", PATHS)
@pytest.mark.parametrize("hit", ["innermost", "outermost"])
def test_deepest_tree_fits_the_stacks(api, hit, paths):
    if hit == "innermost":  # every box is entered, the first triangle hit
        triangles, tree = nested(lambda level, j: True)
        target = 0
    else:  # every stacked node is taken back
        triangles, tree = nested(lambda level, j: (level, j) == (0, 2))
        target = len(triangles) - 1
    scene = imported(api, triangles, tree)
    assert scene.statistics()["maximum_depth"] == 64
    o, d, keys, along = axis_rays(paths, 512)
    hits, _ = scene.intersect(o[along], d[along], 0.0, np.inf)
    assert (hits["primitive"] == target).all()
    assert scene.occluded(o[along], d[along], 0.0, np.inf)[0].all()
    tracer = api.PathTracer(scene, api.IntegratorSettings("mis", 1, True, 3))
    radiance, _ = tracer.trace(o, d, 0.0, np.inf, keys)
    np.testing.assert_array_equal(radiance, np.where(along, 0, np.float32(0.5))[:, None].repeat(3, 1))
