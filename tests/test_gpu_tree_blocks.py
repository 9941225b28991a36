"""The bottom-up tree over blocks of 1,024 leaves against the oracle's Karras
hierarchy, bit for bit: leaf counts on both sides of a block and of several, so
many that the blocks' subtrees do not fit one block (600,000), spread, clustered
and equal Morton codes (ties by position), and boxes as the unions of their
children's."""
import numpy as np
import pytest

import pyoracle
from seevr_b200.bvh import BVH

pytestmark = pytest.mark.gpu


def triangles(n, kind):
    rng = np.random.default_rng(n)
    c = rng.uniform(-10, 10, (n, 1, 3))
    if kind == "equal":
        c[:] = c[0]
    elif kind == "clustered":
        c = np.round(c / 5) * 5 + rng.uniform(0, 1e-3, c.shape) * (rng.uniform(size=(n, 1, 1)) < 0.1)
    tri = (c + (0 if kind == "equal" else 1) * rng.uniform(-0.01, 0.01, (n, 3, 3))
           + np.array([[0, 0, 0], [0.1, 0, 0], [0, 0.1, 0.1]])).astype(np.float32)
    return tri


@pytest.mark.parametrize("n, kind", [(n, k) for n in (2, 3, 31, 1023, 1024, 1025, 2048, 2049, 70000)
                                     for k in ("spread", "clustered", "equal")] + [(600000, "spread")])
def test_tree(cuda, n, kind):
    import torch

    tri = triangles(n, kind)
    v = torch.from_numpy(tri.reshape(-1, 3)).to(cuda)
    idx = torch.arange(3 * n, dtype=torch.int32, device=cuda).reshape(n, 3)
    bvh = BVH(v, idx)
    for _ in range(2):  # the second build starts from the first one's flags
        bvh.build(n)
    torch.cuda.synchronize()
    g = lambda k: bvh[k].cpu().numpy()
    cen = ((tri[:, 0] + tri[:, 1]) + tri[:, 2]) / np.float32(3.0)
    codes, _ = pyoracle.morton(cen)
    s, perm = pyoracle.radix_sort(codes)
    assert np.array_equal(g("morton")[:n].view(np.uint32), s)
    assert np.array_equal(g("prim_indices")[:n].view(np.uint32), perm)
    left, right, parent = pyoracle.karras(s)
    nodes = 2 * n - 1
    assert np.array_equal(g("left")[: n - 1].view(np.uint32), left[: n - 1])
    assert np.array_equal(g("right")[: n - 1].view(np.uint32), right[: n - 1])
    assert np.array_equal(g("parent")[:nodes].view(np.uint32), parent)
    assert np.array_equal(g("left")[n - 1: nodes], np.arange(n))
    assert (g("count")[n - 1: nodes] == 1).all() and (g("count")[: n - 1] == 0).all()
    assert (g("flags")[: n - 1] == 2).all()
    nmin = g("node_min")[: 3 * nodes].reshape(nodes, 3)
    nmax = g("node_max")[: 3 * nodes].reshape(nodes, 3)
    lt = tri[perm.astype(np.int64)]
    assert np.array_equal(nmin[n - 1:], lt.min(axis=1)) and np.array_equal(nmax[n - 1:], lt.max(axis=1))
    L, R = left[: n - 1].astype(np.int64), right[: n - 1].astype(np.int64)
    assert np.array_equal(nmin[: n - 1], np.minimum(nmin[L], nmin[R]))
    assert np.array_equal(nmax[: n - 1], np.maximum(nmax[L], nmax[R]))
    bvh.deinit()
