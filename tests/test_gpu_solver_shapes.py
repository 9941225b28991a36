"""The bundle solver's launch shapes against the sequential loop, bit for bit: one
bundle above 512 bodies among few and among many (eight warps, four), the same in
scene groups, and contact lists that do not fit a block's shared memory (a heap of
boxes has several contacts per body)."""
import numpy as np
import pytest

from helpers import DT, G, read_back
from seevr_b200 import SOLVER_SEQUENTIAL, SOLVER_WAVEFRONT, Caps, Data, Physics, make_params

pytestmark = pytest.mark.gpu

KEYS = ("pos", "quat", "vel", "omega", "lambda", "c_a", "c_b")


def heaps(sizes, pitch=1.01):
    """Scenes of `sizes` boxes each, in cubes of boxes that touch."""
    d = Data()
    ground = d.add_material((.5, .5, .5), .5, 0, (0, 0, 0), 0, 0)
    m = d.add_material((.8, .2, .2), .4, 0, (0, 0, 0), 0, 1000)
    for n in sizes:
        d.begin_scene()
        d.add_box((0, -0.25, 0), (100, 0.25, 100), (1, 1, 1), 0.5, 0.2, ground)
        side = max(2, round(n ** (1 / 3)))
        for i in range(n):
            d.add_box((pitch * (i % side) + 0.003 * (i % 7), 0.499 + 0.99 * (i // side**2),
                       pitch * (i // side % side) + 0.003 * (i % 5)), (0.5, 0.5, 0.5), (1, 1, 1),
                      0.5, 0.2, m)
    return d


def run(d, cuda, solver, groups=1, bundle=0, frames=2, pgs=6):
    buf = d.upload(cuda, Caps.for_data(d, pairs_per_body=24.0, contacts_per_body=12.0))
    ph = Physics(buf, make_params(pgs_iterations=pgs, solver=solver, flags=4, bundle_bodies=bundle))
    if groups > 1:
        ph.set_tuning(scene_groups=groups, bundle_bodies=bundle)
    for _ in range(frames):
        ph.step(buf.num_bodies, 0, buf.num_hull_verts, 10, DT, G)
    out = read_back(buf)
    ph.deinit()
    return out


@pytest.mark.parametrize("sizes, groups, bundle", [
    ([600, 40, 300], 1, 0), ([600] + [9] * 11200, 1, 64), ([700, 300, 300, 900, 80, 500], 3, 1000),
    ([20] * 90, 4, 100), ([120] * 12, 1, 128), ([250] * 6, 1, 256), ([1000], 1, 0), ([27] * 30, 2, 1000)])
def test_shapes(cuda, sizes, groups, bundle):
    d = heaps(sizes)
    a = run(d, cuda, SOLVER_SEQUENTIAL, groups, bundle)
    b = run(d, cuda, SOLVER_WAVEFRONT, groups, bundle)
    assert a["num_contacts"] > 0.4 * sum(sizes)
    for k in KEYS:
        assert np.isfinite(a[k]).all() and np.array_equal(a[k], b[k]), k
