"""The LBVH broadphase with a single body, static or not: no pairs, whatever an
earlier step with more bodies left in the handle."""
import pytest

from helpers import DT, G
from seevr_b200 import BROADPHASE_LBVH, Caps, Data, Physics, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("static", [True, False])
def test_one_body(cuda, static):
    d = Data()
    m = d.add_material((.5, .5, .5), .5, 0, (0, 0, 0), 0, 0 if static else 1000)
    d.add_box((0, -0.25, 0), (30, 0.25, 30), (1, 1, 1), 0.5, 0.2, m)
    b = d.add_material((.8, .2, .2), .4, 0, (0, 0, 0), 0, 1000)
    for i in range(100):
        d.add_box((1.2 * (i % 10) - 6, 0.49, 1.2 * (i // 10) - 6), (0.5, 0.5, 0.5), (1, 1, 1), 0.5, 0.2, b)
    buf = d.upload(cuda, Caps.for_data(d))
    ph = Physics(buf, make_params(flags=4, broadphase=BROADPHASE_LBVH))
    ph.step(buf.num_bodies, 0, buf.num_hull_verts, 1, DT / 10, G)
    assert ph.read_counters()[0] >= 100
    ph.step(1, 0, buf.num_hull_verts, 1, DT / 10, G)
    assert ph.read_counters() == (0, 0)
    ph.deinit()
