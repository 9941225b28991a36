"""Arguments outside the ranges of the branch-free root and divisions, against the CPU
oracle, which has only the built-in ones, bit for bit: normal and tangential masses
below and above the divisors' range, approach and slip speeds so small or large that a
numerator or the slip's square leaves its range, and a slip with one tiny component.
Columns of boxes (chained contacts) and boxes one by one (lone contacts)."""
import numpy as np
import pytest

import pyoracle
from helpers import DT, read_back
from seevr_b200 import SOLVER_COLORED, SOLVER_SEQUENTIAL, SOLVER_WAVEFRONT, Caps, Physics, make_params
from test_gpu_solver_flow import column

pytestmark = pytest.mark.gpu

KEYS = ("pos", "quat", "vel", "omega", "lambda", "c_a", "c_b")


def masses(f):
    def edit(a):
        for k in ("body_inv_mass", "body_inv_inertia"):
            a[k][6:60] *= np.float32(f)
    return edit


def speeds(v, w=(0.0, 0.0, 0.0)):
    def edit(a):
        a["body_vel"][1:] = np.asarray(v, np.float32)
        a["body_omega"][1:] = np.asarray(w, np.float32)
    return edit


CASES = {  # edit, gravity, what shows that a range is left
    "heavy": (masses(1e-20), -9.81, lambda a, m, v: m.min() < 1e-12),
    "light": (masses(1e18), -9.81, lambda a, m, v: m.max() > 1e12),
    "slow": (speeds((3e-27, -5e-27, 1e-27)), 0.0, lambda a, m, v: 0 < abs(v).max() < 1e-25),
    "fast slip": (speeds((3e13, -1.0, 1e12)), 0.0, lambda a, m, v: abs(v).max() ** 2 > 1e24),
    "fast": (speeds((0.0, -4e25, 0.0)), 0.0, lambda a, m, v: abs(v).max() > 1e25),
    "one tiny component": (speeds((1e-30, -0.5, 1.5)), 0.0, lambda a, m, v: 0 < abs(v[1:, 0]).max() < 1e-25),
}


@pytest.mark.parametrize("bodies, height", [(40, 4), (24, 1), (300, 3)])
@pytest.mark.parametrize("solver", [SOLVER_WAVEFRONT, SOLVER_COLORED, SOLVER_SEQUENTIAL])
@pytest.mark.parametrize("case", CASES)
def test_against_the_oracle(cuda, case, solver, bodies, height):
    if solver == SOLVER_COLORED and height > 1:
        pytest.skip("colour order is not contact order here")
    edit, g, leaves = CASES[case]
    d = column(bodies, height)
    a = d.arrays()
    edit(a)
    caps = Caps.for_data(d)
    gravity = (0.0, g, 0.0)
    want = pyoracle.run(a, frames=1, substeps=1, dt=DT / 10, gravity=gravity, pgs_iterations=5,
                        max_pairs=caps.max_pairs, max_contacts=caps.max_contacts, slop=0.1)
    m = a["body_inv_mass"]
    assert want["num_contacts"] >= bodies and leaves(a, m[want["c_a"]] + m[want["c_b"]], a["body_vel"])
    assert all(np.isfinite(want[k]).all() for k in ("vel", "omega", "lambda"))
    buf = d.upload(cuda, caps)
    for k in ("body_inv_mass", "body_inv_inertia", "body_vel", "body_omega"):
        x = a[k].reshape(-1)
        buf[k][: x.size].copy_(buf[k].new_tensor(x))
    ph = Physics(buf, make_params(pgs_iterations=5, solver=solver, flags=4, slop=0.1))
    ph.step(buf.num_bodies, 0, buf.num_hull_verts, 1, DT / 10, gravity)
    got = read_back(buf)
    ph.deinit()
    for k in KEYS:
        assert np.array_equal(got[k], want[k].astype(got[k].dtype)), k
