"""The path tracer on both sides of the 1,500 triangles from which it builds wide nodes,
against the CPU restatement's binary traversal, bit for bit: built trees, and above the
limit the trees at the edges of what the wide traversal takes: chains on both sides of
the shader's stack and of the depth it is left to the shader's own traversal, with
leaves of one triangle and of many, and boxes that do not nest or are not finite."""
import numpy as np
import pytest
import torch

from seevr_b200.bvh import BVH
from test_gpu_raytrace_trees import check, scene

pytestmark = pytest.mark.gpu

KEYS = ("node_min", "node_max", "left", "right", "count", "prim_indices")


def mesh(boxes):
    d = scene(boxes)
    a = d.arrays()
    return d, a["vertices"].reshape(-1, 3), a["indices"].reshape(-1, 3)


def chain(verts, tris, groups, left_leaf):
    """A list-shaped tree whose leaves hold the groups of triangles."""
    full = 2 * len(tris) - 1
    mn, mx = np.zeros((full, 3), np.float32), np.zeros((full, 3), np.float32)
    left, right, count = (np.zeros(full, np.uint32) for _ in range(3))
    at = np.concatenate([[0], np.cumsum(groups)])
    for i, n in enumerate(groups):
        leaf = 2 * i if i == len(groups) - 1 else 2 * i + 1
        p = verts[tris[at[i]: at[i + 1]].reshape(-1)]
        mn[leaf], mx[leaf], left[leaf], count[leaf] = p.min(0), p.max(0), at[i], n
        if i < len(groups) - 1:
            p = verts[tris[at[i]:].reshape(-1)]
            mn[2 * i], mx[2 * i] = p.min(0), p.max(0)
            left[2 * i], right[2 * i] = (leaf, 2 * i + 2) if left_leaf else (2 * i + 2, leaf)
    return {"node_min": mn, "node_max": mx, "left": left, "right": right, "count": count,
            "prim_indices": np.arange(len(tris), dtype=np.uint32)}


@pytest.mark.parametrize("ntri", [1499, 1500, 1501, 3000])
def test_built_trees(cuda, ntri):
    d, verts, tris = mesh(ntri // 12 + 1)
    tris = tris[:ntri].copy()
    b = BVH(torch.tensor(verts.reshape(-1)).cuda(), torch.tensor(tris.view(np.int32).reshape(-1)).cuda())
    b.build(ntri)
    tree = {k: b[k].cpu().numpy() for k in KEYS}
    b.deinit()
    check(d, verts, tris, {k: v.view(np.uint32) if v.dtype == np.int32 else v for k, v in tree.items()})


@pytest.mark.parametrize("left_leaf", [True, False])
@pytest.mark.parametrize("ones", [2, 28, 29, 30, 31, 47, 48, 49])
def test_chains(cuda, left_leaf, ones):
    d, verts, tris = mesh(126)
    check(d, verts, tris, chain(verts, tris, [1] * ones + [len(tris) - ones], left_leaf))


@pytest.mark.parametrize("groups", [12, 30, 36])
def test_leaves_of_many(cuda, groups):
    d, verts, tris = mesh(126)
    per = len(tris) // groups
    check(d, verts, tris, chain(verts, tris, [per] * (groups - 1) + [len(tris) - per * (groups - 1)], True))


@pytest.mark.parametrize("value", [0.5, np.inf])
def test_boxes_left_to_the_binary_tree(cuda, value):
    d, verts, tris = mesh(126)
    tree = chain(verts, tris, [1] * 20 + [len(tris) - 20], True)
    tree["node_max"][4, 0] -= np.float32(value)  # smaller than its children, or not finite
    check(d, verts, tris, tree)
