"""The builder's level passes over more than 1,024 tasks and more than 1,024 chunks, which one block
lists in several passes that carry their counts: every split at such levels is the one that a plain
FP32 sweep over the 33 candidate planes chooses, the leaf order is a permutation and every node's
children divide its range.
"""

import numpy as np
import pytest

from minirender_b200 import scene as sc

pytestmark = pytest.mark.gpu

F = np.float32
BINS, SMALL_TASK, CHUNK, PASS = 12, 256, 2048, 1024
NODE = np.dtype([("minimum", "<f4", 3), ("maximum", "<f4", 3), ("first", "<u4"), ("right", "<u4"),
                 ("count", "<u4")])


def area(lo, hi, scale):
    e = (hi - lo) * scale[..., None]
    return F(2) * ((e[..., 0] * e[..., 1] + e[..., 1] * e[..., 2]) + e[..., 2] * e[..., 0])


def left_counts(lo, hi, centroid, starts, sizes):
    """For nodes over consecutive `sizes` primitives from `starts`: primitives left of the best plane,
    0 where no plane is cheaper than a leaf."""
    nodes = len(sizes)
    node_lo, node_hi = np.minimum.reduceat(lo, starts), np.maximum.reduceat(hi, starts)
    c_lo, c_hi = np.minimum.reduceat(centroid, starts), np.maximum.reduceat(centroid, starts)
    extent = (node_hi - node_lo).max(1)
    scale = np.where(extent > 0, np.ldexp(F(1), -np.frexp(extent)[1]), F(1)).astype(F)
    parent = area(node_lo, node_hi, scale)
    segment = np.repeat(np.arange(nodes), sizes)
    cost = np.full((nodes, 3, BINS - 1), np.inf, F)
    left_of = np.zeros((nodes, 3, BINS - 1), np.int64)
    for axis in range(3):
        span = (c_hi - c_lo)[segment, axis]
        k = ((centroid[:, axis] - c_lo[segment, axis]) / span * F(BINS))
        key = segment * BINS + np.where(span > 0, np.minimum(k, BINS - 1), 0).astype(np.int64)
        order = np.argsort(key, kind="stable")
        bins, first, counts = np.unique(key[order], return_index=True, return_counts=True)
        count = np.zeros(nodes * BINS, np.int64)
        box_lo, box_hi = np.full((nodes * BINS, 3), np.inf, F), np.full((nodes * BINS, 3), -np.inf, F)
        count[bins] = counts
        box_lo[bins], box_hi[bins] = np.minimum.reduceat(lo[order], first), np.maximum.reduceat(hi[order], first)
        count, box_lo, box_hi = (x.reshape(nodes, BINS, -1) for x in (count, box_lo, box_hi))
        left = np.cumsum(count[..., 0], 1)[:, :-1]
        right = np.asarray(sizes)[:, None] - left
        spread = np.broadcast_to(scale[:, None], left.shape)
        l_area = area(np.minimum.accumulate(box_lo, 1)[:, :-1], np.maximum.accumulate(box_hi, 1)[:, :-1], spread)
        r_area = area(np.minimum.accumulate(box_lo[:, ::-1], 1)[:, ::-1][:, 1:],
                      np.maximum.accumulate(box_hi[:, ::-1], 1)[:, ::-1][:, 1:], spread)
        planes = F(1) + (l_area * left.astype(F) + r_area * right.astype(F)) / parent[:, None]
        possible = (left > 0) & (right > 0) & (c_hi > c_lo)[:, axis, None]
        cost[:, axis] = np.where(possible, planes, np.inf)
        left_of[:, axis] = left
    cost, left_of = cost.reshape(nodes, -1), left_of.reshape(nodes, -1)
    best = np.argmin(cost, 1)  # the first of equals
    at = np.arange(nodes)
    splits = (cost[at, best] < np.asarray(sizes).astype(F)) & (np.asarray(sizes) > 4)
    return np.where(splits, left_of[at, best], 0)


def test_levels_of_many_tasks_and_chunks():
    from minirender_b200 import api
    n = 2_200_001
    rng = np.random.default_rng(4)
    v = (rng.uniform(-0.5, 0.5, (n, 1, 3)) + rng.normal(scale=0.004, size=(n, 3, 3))).astype(F)
    normal = np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    doc = sc.SceneDocument()
    doc.materials = [sc.Material()]
    doc.meshes = [sc.MeshData(v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(n, 3),
                              np.repeat(normal[:, None], 3, axis=1).astype(F), None)]
    doc.objects = [sc.SceneObject(0, 0)]
    exported, order, total = api.Scene(doc.snapshot()).export_bvh()
    nodes = np.frombuffer(exported, NODE)[:total]
    assert (np.bincount(order, minlength=n) == 1).all()

    levels = [np.zeros(1, np.int64)]
    while True:
        inner = levels[-1][nodes["count"][levels[-1]] == 0]
        if not len(inner):
            break
        levels.append(np.stack([nodes["first"][inner], nodes["right"][inner]], 1).reshape(-1).astype(np.int64))
    assert sum(map(len, levels)) == total
    begin = nodes["first"].astype(np.int64)
    end = begin + nodes["count"]
    for level in levels[::-1]:
        inner = level[nodes["count"][level] == 0]
        first, right = nodes["first"][inner], nodes["right"][inner]
        assert (end[first] == begin[right]).all()
        begin[inner], end[inner] = begin[first], end[right]
    assert (begin[0], end[0]) == (0, n)

    third = F(3)
    centroid = (v[:, 0] / third + v[:, 1] / third) + v[:, 2] / third
    lo, hi = v.min(1), v.max(1)
    many_chunks, many_tasks = [], []
    for depth, level in enumerate(levels):
        sizes = (end - begin)[level]
        large = sizes[sizes > SMALL_TASK]
        if ((large + CHUNK - 1) // CHUNK).sum() > PASS:
            many_chunks.append(depth)
        if len(large) > PASS:
            many_tasks.append(depth)
    assert many_chunks[:2] == [0, 1] and len(many_tasks) >= 2
    for depth in {0, 1, many_tasks[0], many_tasks[0] + 1, many_tasks[-1], many_tasks[-1] + 1}:
        level = levels[depth]
        sizes = (end - begin)[level]
        starts = np.concatenate([[0], np.cumsum(sizes)[:-1]])
        at = np.arange(sizes.sum()) - np.repeat(starts, sizes) + np.repeat(begin[level], sizes)
        prims = order[at]
        with np.errstate(divide="ignore", invalid="ignore"):
            expected = left_counts(lo[prims], hi[prims], centroid[prims], starts, sizes)
        inner = nodes["count"][level] == 0
        taken = np.where(inner, end[nodes["first"][level] * inner] - begin[level], 0)
        np.testing.assert_array_equal(taken, expected)
