"""The bundle solver's dataflow order against the sequential loop (mode
SEQUENTIAL, one thread, contacts in index order), bit for bit, over bundle
sizes on both sides of each launch shape (1, 2, 4 and 8 warps), contacts per
lane (one, several), and scenes whose contacts are all lone, all chained or
none; and the update's fallback to the built-in divisions (bodies so heavy
that the normal mass leaves the branch-free range)."""
import numpy as np
import pytest

from helpers import DT, G, read_back
from seevr_b200 import SOLVER_SEQUENTIAL, SOLVER_WAVEFRONT, Caps, Data, Physics, make_params

pytestmark = pytest.mark.gpu

KEYS = ("pos", "quat", "vel", "omega", "lambda", "c_a", "c_b")


def run(d, cuda, solver, frames, pgs, bundle=0, edit=None):
    buf = d.upload(cuda, Caps.for_data(d))
    if edit:
        edit(buf.tensors)
    ph = Physics(buf, make_params(pgs_iterations=pgs, solver=solver, flags=4, bundle_bodies=bundle))
    for _ in range(frames):
        ph.step(buf.num_bodies, 0, buf.num_hull_verts, 10, DT, G)
    out = read_back(buf)
    ph.deinit()
    return out


def both(d, cuda, frames, pgs, bundle=0, edit=None):
    a = run(d, cuda, SOLVER_SEQUENTIAL, frames, pgs, bundle, edit)
    b = run(d, cuda, SOLVER_WAVEFRONT, frames, pgs, bundle, edit)
    for k in KEYS:
        assert np.array_equal(a[k], b[k], equal_nan=True), k
    return a


def column(n, height):
    """n bodies in columns of `height` just above each other: chains."""
    d = Data()
    ground = d.add_material((.5, .5, .5), .5, 0, (0, 0, 0), 0, 0)
    m = d.add_material((.8, .2, .2), .4, 0, (0, 0, 0), 0, 1000)
    d.add_box((0, -0.25, 0), (50, 0.25, 50), (1, 1, 1), 0.5, 0.2, ground)
    for i in range(n):
        c, k = divmod(i, height)
        d.add_box((1.5 * (c % 12) - 9 + 0.02 * (k % 3), 0.499 + 0.998 * k, 1.5 * (c // 12) - 9),
                  (0.5, 0.5, 0.5), (1, 1, 1), 0.5, 0.2, m)
    return d


@pytest.mark.parametrize("bodies, height", [(1, 1), (31, 1), (33, 2), (127, 4), (129, 3), (255, 5),
                                            (300, 8), (511, 4), (700, 6), (1000, 10)])
def test_chains_equal_the_sequential_loop(cuda, bodies, height):
    a = both(column(bodies, height), cuda, frames=2, pgs=7)
    assert a["num_contacts"] >= bodies // 2


@pytest.mark.parametrize("bundle", [64, 128, 200, 512, 1000])
def test_batches_equal_the_sequential_loop(cuda, bundle):
    d = Data.batch(num_scenes=24, min_bodies=8, max_bodies=160, seed_base=31)
    a = both(d, cuda, frames=60, pgs=5, bundle=bundle)
    assert a["num_contacts"] > 50


def test_masses_outside_the_branch_free_range(cuda):
    def heavy(t):  # 1e-20 kg^-1: the normal mass is far below 1e-12
        for k in ("body_inv_mass", "body_inv_inertia"):
            t[k][6:60] *= 1e-20

    both(column(40, 4), cuda, frames=2, pgs=5, edit=heavy)


def test_no_iterations(cuda):
    a = both(column(40, 4), cuda, frames=1, pgs=0)
    assert a["num_contacts"] > 0 and not a["lambda"].any()
