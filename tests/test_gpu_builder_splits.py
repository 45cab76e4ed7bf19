"""Every split of a GPU-built tree is the one a plain FP32 sweep over the 33 candidate planes chooses
(src/render/bvh.cpp:131-183): same leaf decisions, same number of primitives on the left, at sizes
around the warp, the small-task limit (256) and the chunk (2,048), with coincident centroids and flat
boxes among them.
"""

import numpy as np
import pytest

from minirender_b200 import scene as sc
from test_gpu_stream import soup

pytestmark = pytest.mark.gpu

F = np.float32
BINS = 12


@pytest.fixture(scope="module")
def api():
    from minirender_b200 import api as a
    return a


def area(lo, hi, scale):
    if np.any(lo > hi):
        return F(0)
    e = (hi - lo) * scale
    return F(2) * ((e[0] * e[1] + e[1] * e[2]) + e[2] * e[0])


def sweep(lo, hi, centroid):
    """(leaf, primitives left of the best plane) of a node, in FP32 with the builder's operations."""
    n = len(lo)
    if n <= 4:
        return True, 0
    node_lo, node_hi = lo.min(0), hi.max(0)
    extent = (node_hi - node_lo).max()
    scale = F(np.ldexp(1.0, -np.frexp(extent)[1])) if extent > 0 else F(1)
    parent = area(node_lo, node_hi, scale)
    best, left_of = F(n), 0
    for axis in range(3):
        c = centroid[:, axis]
        if c.max() == c.min():
            continue
        k = np.minimum(((c - c.min()) / (c.max() - c.min()) * F(BINS)).astype(np.int32), BINS - 1)
        for split in range(BINS - 1):
            left = k <= split
            count = int(left.sum())
            if count in (0, n):
                continue
            cost = F(1) + (area(lo[left].min(0), hi[left].max(0), scale) * F(count)
                           + area(lo[~left].min(0), hi[~left].max(0), scale) * F(n - count)) / parent
            if cost < best:
                best, left_of = cost, count
    return left_of == 0, left_of


def scene_of(kind, count):
    if kind == "soup":
        return soup(count, 0.05, seed=count)
    if kind == "copies":  # many equal centroids
        return soup(max(1, count // 5), 0.05, seed=count, copies=5)
    doc = soup(count, 0.05, seed=count)  # all in one plane
    doc.meshes[0].positions[:, 1] = 0.25
    return doc


@pytest.mark.parametrize("kind", ["soup", "copies", "flat"])
@pytest.mark.parametrize("count", [5, 17, 32, 33, 64, 255, 256, 257, 2048, 2049, 4500])
def test_splits_are_the_sweeps(api, kind, count):
    snapshot = scene_of(kind, count).snapshot()
    nodes, order, _ = api.Scene(snapshot).export_bvh()
    v = snapshot.world_triangles()
    lo, hi = v.min(1), v.max(1)
    third = F(3)
    centroid = (v[:, 0] / third + v[:, 1] / third) + v[:, 2] / third

    def visit(index):
        """Checks the subtree; returns its range in the leaf order."""
        node = nodes[index]
        if node.count:
            begin, end, left = node.first, node.first + node.count, 0
        else:
            begin, middle = visit(node.first)
            also_middle, end = visit(node.right)
            assert middle == also_middle
            left = middle - begin
        prims = order[begin:end]
        with np.errstate(divide="ignore", invalid="ignore"):
            assert sweep(lo[prims], hi[prims], centroid[prims]) == (bool(node.count), left)
        return begin, end

    assert visit(0) == (0, len(lo))
