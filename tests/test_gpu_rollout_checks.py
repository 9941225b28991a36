"""What a rollout does before its first substep: in bounds-check mode the caller's
index arrays are checked before anything reads through them, and without the hull
range binding the ranges are derived before the lookups' aliases are found."""
import os

import pytest

from helpers import DT, G
from seevr_b200 import Caps, Data, Physics, SeevrError, make_params
from seevr_b200 import _lib as L
from seevr_b200.grad import rollout

pytestmark = pytest.mark.gpu

ROWS = ("body_pos", 3), ("body_quat", 4), ("body_vel", 3), ("body_omega", 3)


def handle(buf, check=False, **kw):
    if check:
        os.environ["SEEVR_CHECK"] = "1"  # read when the handle is created
    try:
        return Physics(buf, make_params(pgs_iterations=5, flags=4), **kw)
    finally:
        os.environ.pop("SEEVR_CHECK", None)


def settled(cuda):
    import torch

    d = Data.rollout(num_scenes=8, bodies=24, seed_base=5)
    buf = d.upload(cuda, Caps.for_data(d))
    ph = handle(buf)
    for _ in range(75):
        ph.step(buf.num_bodies, 0, buf.num_hull_verts, 10, DT, G)
    assert ph.read_counters()[1] > 0
    ph.deinit()
    torch.cuda.synchronize()
    return buf, {k: buf[k][: n * buf.num_bodies].clone() for k, n in ROWS}


def put(buf, state):
    import torch

    for k, v in state.items():
        buf[k][: v.numel()].copy_(v)
    torch.cuda.synchronize()


@pytest.mark.parametrize("check, ranges", [(True, True), (False, False), (True, False)])
def test_a_first_rollout_equals_frames(cuda, check, ranges):
    import torch

    buf, state = settled(cuda)
    ph = handle(buf)
    for _ in range(10):
        ph.step(buf.num_bodies, 0, buf.num_hull_verts, 1, DT / 10, G)
    want = [buf[k][: v.numel()].clone() for k, v in state.items()]
    ph.deinit()
    put(buf, state)
    ph = handle(buf, check, use_hull_range=ranges)
    got = rollout(ph, frames=1)
    for x, y in zip(want, got):
        assert torch.equal(x, y.reshape(-1))
    assert ph.read_flags() == 0
    ph.deinit()


@pytest.mark.parametrize("array", ["hull_range", "geom_body_idx", "support_offset"])
def test_bad_indices_are_reported_first(cuda, array):
    import torch

    buf, state = settled(cuda)
    body = int(buf.scene_body_offset[3]) + 2
    ph = handle(buf, check=True)
    saved = buf[array].clone()
    if array == "hull_range":
        buf[array][2 * body + 1] = buf.num_hull_verts + 5
    elif array == "geom_body_idx":
        buf[array][body] = int(buf.scene_body_offset[5])
    else:
        buf[array][body] = buf["support_lookup"].numel() - 10
    torch.cuda.synchronize()
    with pytest.raises(SeevrError) as e:
        rollout(ph, frames=1)
    assert e.value.status == L.ERR_INVALID_ARGUMENT
    assert "bounds check" in str(e.value) and f"index {body}" in str(e.value), str(e.value)
    for k, v in state.items():
        assert torch.equal(v, buf[k][: v.numel()]), k
    buf[array].copy_(saved)
    torch.cuda.synchronize()
    rollout(ph, frames=1)
    ph.deinit()
