"""The LBVH broadphase's rows of static bodies against the all-pairs lists: as many
static bodies as have a block each, more (the write pass traverses again), one with
a partner in every word of the bitmap, and scenes too large for the bitmap."""
import numpy as np
import pytest

from helpers import DT, G, read_back
from seevr_b200 import BROADPHASE_LBVH, Caps, Data, Physics, make_params

pytestmark = pytest.mark.gpu


def scene(statics, n):
    d = Data()
    g = d.add_material((.5, .5, .5), .5, 0, (0, 0, 0), 0, 0)
    m = d.add_material((.8, .2, .2), .4, 0, (0, 0, 0), 0, 1000)
    side = 2.0 * int(np.ceil(np.sqrt(n)))
    for k in range(statics):  # slabs, each under a strip of the bodies
        w = side / statics
        d.add_box((w * (k + 0.5), -0.25, side / 2), (w / 2, 0.25, side / 2), (1, 1, 1), 0.5, 0.2, g)
    rng = np.random.default_rng(n)
    xy = rng.permutation(int(side // 2) ** 2)[:n]
    for i in xy:
        d.add_box((2.0 * (i % int(side // 2)) + 1, 0.45, 2.0 * (i // int(side // 2)) + 1), (0.5, 0.5, 0.5),
                  (1, 1, 1), 0.5, 0.2, m)
    return d


def lists(d, cuda, broadphase, frames=1):
    buf = d.upload(cuda, Caps.for_data(d))
    ph = Physics(buf, make_params(pgs_iterations=2, flags=4, broadphase=broadphase))
    for _ in range(frames):
        ph.step(buf.num_bodies, 0, buf.num_hull_verts, 2, DT, G)
    out = read_back(buf)
    ph.deinit()
    return out


@pytest.mark.parametrize("statics, n", [(1, 1), (1, 40), (1, 2000), (8, 700), (9, 700), (30, 1500)])
def test_static_rows(cuda, statics, n):
    d = scene(statics, n)
    a, b = lists(d, cuda, 0), lists(d, cuda, BROADPHASE_LBVH)
    assert a["num_pairs"] >= n
    for k in ("num_pairs", "num_contacts"):
        assert a[k] == b[k]
    for k in ("pairs", "pos", "vel", "lambda"):
        assert np.array_equal(a[k], b[k]), k


def test_beyond_the_bitmap(cuda):
    """361,201 bodies: the general pass, against rows found on the host."""
    d = Data.towers(seed=0, towers=11287, height=32, spacing=2.0, overlap=0.004)
    b = lists(d, cuda, BROADPHASE_LBVH)
    assert d.num_bodies > 360000
    rows = b["pairs"][b["pairs"][:, 0] == 0][:, 1]
    lo, hi = b["aabb_min"], b["aabb_max"]
    near = np.all((lo[0] <= hi) & (lo <= hi[0]), axis=1)
    near[0] = False
    assert len(rows) >= 11287 and (np.diff(rows.astype(np.int64)) > 0).all()
    # (the boxes are those of the last substep's broadphase)
    assert np.array_equal(np.flatnonzero(near), rows)
