"""Contacts whose two geoms belong to one body (geom_body_idx not one to one): contact
and colour order against the sequential loop (mode SEQUENTIAL), which reads both sides
at each update and writes side b last, bit for bit.  Boxes two by two, the upper one's
geom on the lower one's body: in free fall (each such contact alone at its body) and on
the ground (two contacts at each body); tall columns whose geoms share bodies in twos
(chains).  Bundles of every block size, lanes with one and with several contacts, and
islands (above 1,024 bodies).  Colour order is compared over one substep of the boxes
two by two, where it is contact order: the ground's contacts come first and take one
colour, the others the next."""
import numpy as np
import pytest

from helpers import DT, G, read_back
from seevr_b200 import (SOLVER_COLORED, SOLVER_SEQUENTIAL, SOLVER_WAVEFRONT, Caps, Data, Physics,
                        make_params)

pytestmark = pytest.mark.gpu

KEYS = ("pos", "quat", "vel", "omega", "lambda", "c_a", "c_b")


def scene(n, height, y):
    d = Data()
    ground = d.add_material((.5, .5, .5), .5, 0, (0, 0, 0), 0, 0)
    m = d.add_material((.8, .2, .2), .4, 0, (0, 0, 0), 0, 1000)
    d.add_box((0, -0.25, 0), (200, 0.25, 200), (1, 1, 1), 0.5, 0.2, ground)
    for i in range(n):
        c, k = divmod(i, height)
        b = d.add_box((1.5 * (c % 40) - 30 + 0.02 * (k % 3), y + 0.98 * k, 1.5 * (c // 40) - 25),
                      (0.5, 0.5, 0.5), (1, 1, 1), 0.5, 0.2, m)
        d.set_body_vel(b, (0.1 * (i % 3), 0.0, 0.2), (0.3, 0.1 * (i % 5), -0.2))
    return d


def owners(n):
    g = np.arange(n + 1)
    g[2::2] -= 1  # bodies 1 and 2, 3 and 4, ...: the odd one's
    return g.astype(np.uint32)


def run(d, cuda, geom_body, solver, substeps):
    buf = d.upload(cuda, Caps.for_data(d))
    buf["geom_body_idx"][: len(geom_body)] = buf["geom_body_idx"].new_tensor(geom_body.astype(np.int32))
    ph = Physics(buf, make_params(pgs_iterations=6, solver=solver, flags=4))
    ph.step(buf.num_bodies, 0, buf.num_hull_verts, substeps, DT * substeps / 10, G)
    out = read_back(buf)
    ph.deinit()
    return out


@pytest.mark.parametrize("solver", [SOLVER_WAVEFRONT, SOLVER_COLORED])
@pytest.mark.parametrize("bodies, height, y", [
    (2, 2, 9.0), (60, 2, 9.0), (400, 2, 9.0), (1200, 2, 9.0),
    (20, 2, 0.49), (120, 2, 0.49), (240, 2, 0.49), (400, 2, 0.49), (900, 2, 0.49), (1200, 2, 0.49),
    (64, 16, 0.49), (500, 20, 0.49), (1000, 100, 0.49), (1200, 100, 0.49)])
def test_both_sides_one_body(cuda, solver, bodies, height, y):
    if solver == SOLVER_COLORED and height > 2:
        pytest.skip("colour order is not contact order here")
    d, geom_body = scene(bodies, height, y), owners(bodies)
    a, b = (run(d, cuda, geom_body, s, 1 if solver == SOLVER_COLORED else 10)
            for s in (SOLVER_SEQUENTIAL, solver))
    same = geom_body[a["c_a"]] == geom_body[a["c_b"]]
    assert same.sum() >= bodies // 2 and (a["lambda"][same] > 0).any()
    for k in KEYS:
        assert np.isfinite(a[k]).all() and np.array_equal(a[k], b[k]), k
