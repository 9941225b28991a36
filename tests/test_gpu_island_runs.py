"""Runs of islands (scenes above 1,024 bodies), bit for bit: in contact order
against the sequential loop, in colour order against the warp-per-island kernel
(which a giant-island threshold of 1,024 contacts selects).  Islands of one
contact, below, at and above a run's window of 128 contacts, above the 1,024
contacts a run takes (128 in contact order), and a body with more than 32 contacts (no 32 colours)
among others in one run."""
import numpy as np
import pytest

from helpers import DT, G, read_back
from seevr_b200 import (BROADPHASE_LBVH, SOLVER_COLORED, SOLVER_SEQUENTIAL, SOLVER_WAVEFRONT, Caps,
                        Data, Physics, make_params)

pytestmark = pytest.mark.gpu

KEYS = ("pos", "quat", "vel", "omega", "lambda", "c_a", "c_b")
N = 1200


def ground(d):
    m = d.add_material((.5, .5, .5), .5, 0, (0, 0, 0), 0, 0)
    d.add_box((0, -0.25, 0), (200, 0.25, 200), (1, 1, 1), 0.5, 0.2, m)
    return d.add_material((.8, .2, .2), .4, 0, (0, 0, 0), 0, 1000)


def boxes(d, m, n, height, x0=0.0):
    for i in range(n):
        c, k = divmod(i, height)
        d.add_box((x0 + 1.5 * (c % 40) - 30 + 0.02 * (k % 3), 0.499 + 0.998 * k, 1.5 * (c // 40) - 25),
                  (0.5, 0.5, 0.5), (1, 1, 1), 0.5, 0.2, m)


def columns(height):
    d = Data()
    boxes(d, ground(d), N, height)
    return d


def sheet(cols, rows):
    """Boxes side by side, all in one island, and single ones beside it."""
    d = Data()
    m = ground(d)
    boxes(d, m, N, 2, x0=80.0)
    for i in range(cols * rows):
        d.add_box((0.999 * (i % cols) - 30, 0.499, 0.999 * (i // cols) - 20), (0.5, 0.5, 0.5),
                  (1, 1, 1), 0.5, 0.2, m)
    return d


def plates(n):
    """Plates with 40 boxes on each, between columns of two."""
    d = Data()
    m = ground(d)
    for p in range(n):
        d.add_box((12.0 * p - 60, 0.249, 60), (5.5, 0.25, 3), (1, 1, 1), 0.5, 0.2, m)
        for i in range(40):
            d.add_box((12.0 * p - 60 + 1.05 * (i % 10) - 4.7, 0.996, 60 + 1.2 * (i // 10) - 2),
                      (0.5, 0.5, 0.5), (1, 1, 1), 0.5, 0.2, m)
        boxes(d, m, 8, 2, x0=80.0 * (p % 2))
    boxes(d, m, N, 3, x0=170.0)
    return d


def run(d, cuda, solver, giant=0, frames=2, pgs=6, broadphase=0):
    buf = d.upload(cuda, Caps.for_data(d))
    ph = Physics(buf, make_params(pgs_iterations=pgs, solver=solver, flags=4, broadphase=broadphase))
    if giant:
        ph.set_tuning(giant_island_contacts=giant)
    for _ in range(frames):
        ph.step(buf.num_bodies, 0, buf.num_hull_verts, 10, DT, G)
    out = read_back(buf)
    ph.deinit()
    return out


SCENES = {"lone": lambda: columns(1), "pairs": lambda: columns(2), "40": lambda: columns(40),
          "120": lambda: columns(120), "400": lambda: columns(400), "sheet": lambda: sheet(12, 10),
          "wide sheet": lambda: sheet(30, 24), "plates": lambda: plates(3)}


@pytest.mark.parametrize("name", SCENES)
def test_contact_order(cuda, name):
    d = SCENES[name]()
    a, b = run(d, cuda, SOLVER_SEQUENTIAL), run(d, cuda, SOLVER_WAVEFRONT)
    assert a["num_contacts"] > 400
    for k in KEYS:
        assert np.array_equal(a[k], b[k], equal_nan=True), k


def test_three_sort_passes(cuda):
    """67,201 bodies: the islands' roots no longer fit two 8-bit digits."""
    d = Data.towers(seed=0, towers=2100, height=32, spacing=2.0, overlap=0.004)
    a, b = (run(d, cuda, s, frames=1, broadphase=BROADPHASE_LBVH)
            for s in (SOLVER_SEQUENTIAL, SOLVER_WAVEFRONT))
    assert a["num_contacts"] > 60000
    for k in KEYS:
        assert np.array_equal(a[k], b[k], equal_nan=True), k


# (the wide sheet's island is above the lowered threshold: the reference run would
# solve it grid-wide, in other colours)
@pytest.mark.parametrize("name", [n for n in SCENES if n != "wide sheet"])
def test_colour_order(cuda, name):
    d = SCENES[name]()
    a, b = run(d, cuda, SOLVER_COLORED, giant=1024), run(d, cuda, SOLVER_COLORED)
    assert a["num_contacts"] > 400
    for k in KEYS:
        assert np.array_equal(a[k], b[k], equal_nan=True), k
