"""Bundles with more than two contacts per lane, swept level by level, against the
sequential loop, bit for bit: columns of boxes (every contact chained, as many contacts
as boxes) on both sides of the limit for two, four and eight warps, with levels of one
contact, of a few and of more than a block's threads, one and several iterations, and
records in shared memory, in part and not at all (heaps in 1,024-body bundles)."""
import numpy as np
import pytest

from helpers import DT, G, read_back
from seevr_b200 import SOLVER_COLORED, SOLVER_SEQUENTIAL, SOLVER_WAVEFRONT, Caps, Data, Physics, make_params

pytestmark = pytest.mark.gpu

KEYS = ("pos", "quat", "vel", "omega", "lambda", "c_a", "c_b")


def scene(boxes):
    """boxes: per scene, the centres."""
    d = Data()
    ground = d.add_material((.5, .5, .5), .5, 0, (0, 0, 0), 0, 0)
    m = d.add_material((.8, .2, .2), .4, 0, (0, 0, 0), 0, 1000)
    for at in boxes:
        d.begin_scene()
        d.add_box((0, -0.25, 0), (200, 0.25, 200), (1, 1, 1), 0.5, 0.2, ground)
        for p in at:
            d.add_box(tuple(map(float, p)), (0.5, 0.5, 0.5), (1, 1, 1), 0.5, 0.2, m)
    return d


def columns(n, height):
    return [(1.5 * (i // height % 40) - 30 + 0.02 * (i % height % 3), 0.499 + 0.998 * (i % height),
             1.5 * (i // height // 40)) for i in range(n)]


def heap(n):
    side = round(n ** (1 / 3))
    return [(1.01 * (i % side) + 0.003 * (i % 7), 0.499 + 0.99 * (i // side**2),
             1.01 * (i // side % side) + 0.003 * (i % 5)) for i in range(n)]


def run(d, cuda, solver, pgs, groups=1, bundle=0, frames=1):
    buf = d.upload(cuda, Caps.for_data(d, pairs_per_body=24.0, contacts_per_body=12.0))
    ph = Physics(buf, make_params(pgs_iterations=pgs, solver=solver, flags=4, bundle_bodies=bundle))
    if groups > 1:
        ph.set_tuning(scene_groups=groups, bundle_bodies=bundle)
    for _ in range(frames):
        ph.step(buf.num_bodies, 0, buf.num_hull_verts, 10, DT, G)
    out = read_back(buf)
    ph.deinit()
    return out


def same(a, b):
    for k in KEYS:
        assert np.isfinite(a[k]).all() and np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("pgs", [1, 2, 9])
@pytest.mark.parametrize("n, height", [
    (128, 2), (129, 2), (129, 43), (200, 200), (255, 5),  # two warps: above 128 contacts
    (256, 4), (257, 4), (500, 2), (500, 250), (511, 7),  # four: above 256
    (512, 8), (513, 8), (1000, 2), (1000, 500), (1023, 11)])  # eight: above 512
def test_columns(cuda, n, height, pgs):
    d = scene([columns(n, height)])
    a, b = (run(d, cuda, s, pgs) for s in (SOLVER_SEQUENTIAL, SOLVER_WAVEFRONT))
    assert a["num_contacts"] >= n
    same(a, b)


@pytest.mark.parametrize("sizes, groups, bundle", [
    ([216] * 8, 1, 256), ([125] * 8, 1, 512), ([1000] * 3, 3, 1024), ([343, 64, 27, 512] * 3, 4, 1024),
    ([64] * 60, 4, 1024), ([8] * 300, 1, 1024)])
def test_heaps(cuda, sizes, groups, bundle):
    d = scene([heap(n) for n in sizes])
    a, b = (run(d, cuda, s, 5, groups, bundle, frames=3) for s in (SOLVER_SEQUENTIAL, SOLVER_WAVEFRONT))
    assert a["num_contacts"] > sum(sizes) // 2
    same(a, b)


def test_more_than_32_colours(cuda):
    """A plate with 40 boxes on it has no 32 colours: the bundle goes in contact order."""
    d = scene([columns(500, 4)])
    m = d.add_material((.8, .2, .2), .4, 0, (0, 0, 0), 0, 1000)
    d.add_box((0, 0.249, 40), (5.5, 0.25, 3), (1, 1, 1), 0.5, 0.2, m)
    for i in range(40):
        d.add_box((1.05 * (i % 10) - 4.7, 0.996, 40 + 1.2 * (i // 10) - 2), (0.5, 0.5, 0.5), (1, 1, 1),
                  0.5, 0.2, m)
    a, b = (run(d, cuda, s, 5) for s in (SOLVER_SEQUENTIAL, SOLVER_COLORED))
    assert a["num_contacts"] >= 540
    same(a, b)
