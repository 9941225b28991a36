"""A sort whose look-backs give up (wait limit 0): the step ends with a timeout and
stays within its buffers, and the handle, its limit restored, steps like a fresh one.
The body tree's sort (30-bit codes, four passes) and the islands' (two and three
passes); and a tree of more blocks than run at once, where a wait of the first ones
gives up while others begin."""
import numpy as np
import pytest

from helpers import DT, G, read_back
from seevr_b200 import BROADPHASE_LBVH, Caps, Data, Physics, SeevrError, make_params
from seevr_b200 import _lib as L

pytestmark = pytest.mark.gpu

ROWS = ("body_pos", 3), ("body_quat", 4), ("body_vel", 3), ("body_omega", 3)


@pytest.mark.parametrize("towers, height", [(200, 60), (1200, 60), (5200, 60)])
def test_sorts_that_give_up(cuda, towers, height):
    import torch

    d = Data.towers(seed=0, towers=towers, height=height, spacing=2.0, overlap=0.004)
    caps = Caps.for_data(d)
    buf = d.upload(cuda, caps)
    nb, nhv = buf.num_bodies, buf.num_hull_verts
    params = make_params(pgs_iterations=4, flags=4, broadphase=BROADPHASE_LBVH)
    ph = Physics(buf, params)
    ph.step(nb, 0, nhv, 2, DT, G)
    saved = {k: buf[k][: n * nb].clone() for k, n in ROWS}
    ph.set_wait_limit(0)
    outcomes = []
    for _ in range(6):
        try:
            ph.step(nb, 0, nhv, 2, DT, G)
            outcomes.append(L.OK)
        except SeevrError as e:
            outcomes.append(e.status)
    assert set(outcomes) <= {L.OK, L.ERR_TIMEOUT} and L.ERR_TIMEOUT in outcomes, outcomes
    ph.set_wait_limit(1 << 22)

    def again(buf, ph):
        for k, v in saved.items():
            buf[k][: v.numel()].copy_(v)
        torch.cuda.synchronize()
        ph.step(nb, 0, nhv, 2, DT, G)
        out = read_back(buf)
        ph.deinit()
        return out

    a = again(buf, ph)
    buf2 = d.upload(cuda, caps)
    b = again(buf2, Physics(buf2, params))
    assert a["num_contacts"] > towers * height // 2
    for k in ("pos", "quat", "vel", "omega", "pairs", "lambda", "c_a", "c_b"):
        assert np.array_equal(a[k], b[k]), k
