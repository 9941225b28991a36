"""The path tracer's wide traversal against the CPU restatement's binary one, bit
for bit, on trees at the edges of what it takes: one to five triangles, leaves of
several triangles, a chain that the shader's 32-entry stack truncates (which only
the shader's own traversal reproduces), chains on both sides of the limit, and
boxes that do not nest."""
import numpy as np
import pytest
import torch

import pyoracle
from seevr_b200 import Data
from seevr_b200 import _lib as L
from seevr_b200.bvh import BVH
from seevr_b200.raytrace import Raytracer

pytestmark = pytest.mark.gpu

W, H = 40, 30
CAM = np.array([0.0, 2.5, 6.0, 0.0, -0.25, -1.0, 1.0, 0.0, 0.0, 0.0, 1.0, -0.25], np.float32)


def scene(n):
    """n boxes in front of the camera."""
    d = Data()
    m = d.add_material((0.8, 0.6, 0.4), 0.4, 0.0, (0.2, 0.2, 0.2), 0.0, 1000.0)
    rng = np.random.default_rng(n)
    for _ in range(n):
        c = (rng.uniform(-2, 2), rng.uniform(0.3, 2), rng.uniform(-3, 1))
        d.add_box(c, (0.4, 0.4, 0.4), (1, 1, 1), 0.5, 0.2, m)
    return d


def check(d, verts, tris, tree):
    """Renders on the GPU and with the restatement over the same tree (a dict of
    numpy arrays)."""
    a = d.arrays()
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x).reshape(-1).view(
        np.int32 if x.dtype == np.uint32 else x.dtype)).cuda()
    bvh = {"vertices": t(verts), "indices": t(tris), **{k: t(v) for k, v in tree.items()}}
    rt = Raytracer(d, bvh, W, H)
    rt.t["tri_geom"] = t(a["tri_geom"][: len(tris)])
    got = rt.render(CAM[0:3], CAM[3:6], CAM[6:9], CAM[9:12], len(tris)).cpu().numpy()
    ref = pyoracle.raytrace(verts, tris, tree["node_min"], tree["node_max"], tree["left"],
                            tree["right"], tree["count"], tree["prim_indices"], a["tri_geom"],
                            a["geom_material"], a["mat_albedo"], a["mat_roughness"],
                            a["mat_metallic"], a["mat_emission"], a["mat_ior"], CAM, W, H, 0,
                            L.lib.seevr_raytrace_fov_scale(), threads=4)
    assert np.array_equal(got, ref)
    return got


def chain(verts, tris, left_leaf, per_leaf=1):
    """A list-shaped tree: every inner node has a leaf on one side and the rest on
    the other (the right one where left_leaf)."""
    groups = [list(range(i, min(i + per_leaf, len(tris)))) for i in range(0, len(tris), per_leaf)]
    n = 2 * len(groups) - 1
    full = 2 * len(tris) - 1  # the arrays' size
    mn, mx = np.zeros((full, 3), np.float32), np.zeros((full, 3), np.float32)
    left, right, count = (np.zeros(full, np.uint32) for _ in range(3))
    box = lambda g: (verts[tris[g].reshape(-1)].min(0), verts[tris[g].reshape(-1)].max(0))
    inner = lambda i: 2 * i           # node of groups[i:]; the last one is a leaf
    for i, g in enumerate(groups):
        leaf = inner(i) if i == len(groups) - 1 else 2 * i + 1
        mn[leaf], mx[leaf] = box(g)
        left[leaf], count[leaf] = g[0], len(g)
        if i < len(groups) - 1:
            mn[inner(i)], mx[inner(i)] = box(sum(groups[i:], []))
            a, b = (leaf, inner(i + 1)) if left_leaf else (inner(i + 1), leaf)
            left[inner(i)], right[inner(i)] = a, b
    assert n <= full
    return {"node_min": mn, "node_max": mx, "left": left, "right": right, "count": count,
            "prim_indices": np.arange(len(tris), dtype=np.uint32)}


@pytest.mark.parametrize("ntri", [1, 2, 3, 4, 5, 12])
def test_few_triangles(cuda, ntri):
    d = scene(1)
    a = d.arrays()
    verts = a["vertices"].reshape(-1, 3)
    tris = a["indices"].reshape(-1, 3)[-ntri:].copy()
    b = BVH(torch.tensor(verts.reshape(-1)).cuda(), torch.tensor(tris.view(np.int32).reshape(-1)).cuda())
    b.build(ntri)
    tree = {}
    for k in ("node_min", "node_max", "left", "right", "count", "prim_indices"):
        x = b[k].cpu().numpy()
        tree[k] = x.view(np.uint32) if x.dtype == np.int32 else x
    b.deinit()
    check(d, verts, tris, tree)


@pytest.mark.parametrize("left_leaf", [True, False])
@pytest.mark.parametrize("groups, per_leaf", [(29, 1), (30, 1), (31, 1), (32, 1), (34, 1), (48, 1),
                                              (49, 1), (50, 1), (12, 5)])
def test_chains(cuda, left_leaf, groups, per_leaf):
    d = scene(6)
    a = d.arrays()
    verts, tris = a["vertices"].reshape(-1, 3), a["indices"].reshape(-1, 3)
    tris = tris[: groups * per_leaf]
    img = check(d, verts, tris, chain(verts, tris, left_leaf, per_leaf))
    assert np.isfinite(img).all()


def test_boxes_that_do_not_nest(cuda):
    d = scene(4)
    a = d.arrays()
    verts, tris = a["vertices"].reshape(-1, 3), a["indices"].reshape(-1, 3)[:24]
    tree = chain(verts, tris, True)
    tree["node_max"][4, 0] -= 0.5  # a parent smaller than its children
    check(d, verts, tris, tree)
