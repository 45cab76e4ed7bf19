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


LIMIT = 65536  # node visits and leaves of one ray


def beads(levels, decoys):
    """A tree whose 2^levels - 1 wide nodes the +z axis enters one after the other, each with two
    children of its own beside the axis (four at the bottom), and no triangle. `decoys` bottom leaves
    have boxes that the axis enters: node visits and leaves of an axis ray are 2^levels - 1 + decoys."""
    near = np.array([(4, -0.5), (5, -0.5), (4, 0.5)], float)
    passed = np.array([(-0.4, -0.5), (0.5, -0.5), (0.5, 0.4)], float)
    triangles, left = [], decoys

    def triangle(side):
        xy = passed if side == 0 else near * (side, 1)
        triangles.append(np.column_stack([xy, np.full(3, len(triangles) + 1.0)]))
        return len(triangles) - 1

    def node(level):
        nonlocal left
        if level == 1:
            left, decoy = max(0, left - 1), left > 0
            return (triangle(1), triangle(-1)), (triangle(1), triangle(0 if decoy else -1))
        first = node(level - 1), triangle(1)
        return first, (node(level - 1), triangle(-1))

    tree = node(levels)
    return np.array(triangles), tree


@pytest.fixture(scope="module")
def bead_scenes(api):
    return {decoys: imported(api, *beads(16, decoys)) for decoys in (1, 2)}


@pytest.mark.parametrize("decoys", [1, 2])
@pytest.mark.parametrize("paths", [None, 1 << 10, 1 << 19], ids=["query", "few", "streamed"])
def test_visit_bound_is_the_same_on_every_route(api, bead_scenes, paths, decoys):
    scene = bead_scenes[decoys]
    accepted = (1 << 16) - 1 + decoys <= LIMIT
    o, d, keys, along = axis_rays(paths or 64, 64)
    tracer = api.PathTracer(scene, api.IntegratorSettings("mis", 1, True, 3))

    def calls():
        if paths is None:
            yield lambda: scene.intersect(o, d, 0.0, np.inf)
            yield lambda: scene.occluded(o, d, 0.0, np.inf)
        else:
            yield lambda: tracer.trace(o, d, 0.0, np.inf, keys)

    for call in calls():
        if not accepted:
            with pytest.raises(api.MiniRenderError, match="node-visit bound"):
                call()
            continue
        out, counts = call()
        if paths is None:
            assert counts["bounds_tests"] == 64 * (1 + 4 * ((1 << 16) - 1)) and counts["triangle_tests"] == 64
            assert not (out if out.dtype == bool else out["primitive"] != 0xffffffff).any()
        else:
            np.testing.assert_array_equal(out, np.full((paths, 3), 0.5, np.float32))


@pytest.mark.parametrize("levels", [1, 2, 3, 8])
def test_subtrees_of_several_parents(api, levels):
    """Both children of each of `levels` nodes are the next one, so a walk meets 2^levels - 1 interior
    nodes of which the import holds `levels`: the wide tree has a node for each time one is met."""
    triangles = np.array([[(-1, -1, z), (3, -1, z), (-1, 3, z)] for z in (1.0, 2.0)])
    plain = imported(api, triangles, (0, 1))
    nodes = [((-1, -1, 1), (3, 3, 2), k + 1, k + 1, 0) for k in range(levels - 1)]
    nodes += [((-1, -1, 1), (3, 3, 2), levels, levels + 1, 0),
              ((-1, -1, 1), (3, 3, 1), 0, 0, 1), ((-1, -1, 2), (3, 3, 2), 1, 0, 1)]
    packed, order = np.array(nodes, NODE), np.arange(2, dtype=np.uint32)
    desc = _abi.BvhDesc(C.cast(packed.ctypes.data, C.POINTER(_abi.BvhNode)), len(packed),
                        order.ctypes.data_as(C.POINTER(C.c_uint32)), 2)
    scene = api.Scene(plain.snapshot, desc)
    assert scene.statistics()["leaves"] == 2 ** levels
    rng = np.random.default_rng(2)
    d = np.column_stack([rng.uniform(-1, 1, (1000, 2)), np.ones(1000)])
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    o = np.zeros_like(d)
    np.testing.assert_array_equal(scene.intersect(o, d)[0], plain.intersect(o, d)[0])
    np.testing.assert_array_equal(scene.occluded(o, d)[0], plain.occluded(o, d)[0])


@pytest.mark.parametrize("triangles", [3, 5, 33, 300])
def test_infinite_flat_boxes(api, triangles):
    """Interior boxes without bounds in x and y and of no extent in z have no comparable area: the collapse
    opens them all the same."""
    rng = np.random.default_rng(triangles)
    corners = rng.uniform(-1, 1, (triangles, 3, 2))
    corners = np.concatenate([corners, np.ones((triangles, 3, 1))], 2)

    def halves(begin, end):
        middle = (begin + end) // 2
        return begin if end - begin == 1 else (halves(begin, middle), halves(middle, end))

    plain = imported(api, corners, halves(0, triangles))
    nodes, order, count = plain.export_bvh()
    packed = np.frombuffer(nodes, NODE)[:count].copy()
    inner = packed["count"] == 0
    inner[0] = False  # the scene's bounds
    packed["minimum"][inner, :2], packed["maximum"][inner, :2] = -np.inf, np.inf
    desc = _abi.BvhDesc(C.cast(packed.ctypes.data, C.POINTER(_abi.BvhNode)), count,
                        order.ctypes.data_as(C.POINTER(C.c_uint32)), triangles)
    scene = api.Scene(plain.snapshot, desc)
    d = np.column_stack([rng.uniform(-1, 1, (4000, 2)), np.ones(4000)])
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    o = np.zeros_like(d)
    np.testing.assert_array_equal(scene.intersect(o, d)[0], plain.intersect(o, d)[0])
