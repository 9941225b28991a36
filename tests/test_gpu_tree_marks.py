"""The triangle tree on vertices with NaN bits of every kind, the one among them that
marks a box as not yet arrived: the build ends, and its links and numbers are those
for a quiet NaN in the same places."""
import numpy as np
import pytest

from seevr_b200.bvh import BVH

pytestmark = pytest.mark.gpu

MARK = 0xFFA5C3E1


@pytest.mark.parametrize("n", [2, 1500, 9000])
@pytest.mark.parametrize("bits", [MARK, 0x7F800001, 0x7FFFFFFF])
def test_nan_bits(cuda, n, bits):
    import torch

    rng = np.random.default_rng(n)
    tri = rng.uniform(-10, 10, (n, 3, 3)).astype(np.float32)
    at = rng.uniform(size=n) < 0.3
    at[:2] = True

    def build(value):
        v = tri.copy()
        v.view(np.uint32)[at, 0, 1] = value
        bvh = BVH(torch.from_numpy(v.reshape(-1, 3)).to(cuda),
                  torch.arange(3 * n, dtype=torch.int32, device=cuda))
        bvh.build(n)
        out = {k: bvh[k].cpu().numpy() for k in ("left", "right", "parent", "prim_indices",
                                                 "node_min", "node_max")}
        bvh.deinit()
        return out

    a, b = build(bits), build(0x7FC00000)
    assert np.isnan(b["node_min"]).any()
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=a[k].dtype == np.float32), k
