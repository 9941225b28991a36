"""Rollouts under another default dtype of torch: the checkpoints, which the library
writes through a raw pointer, are float32 all the same, and states and gradients are
those under the usual default."""
import pytest

from helpers import DT, G
from seevr_b200 import Caps, Data, Physics, make_params
from seevr_b200.grad import rollout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["float64", "bfloat16", "float16"])
def test_default_dtype(cuda, name):
    import torch

    d = Data.rollout(num_scenes=4, bodies=16, seed_base=7)
    buf = d.upload(cuda, Caps.for_data(d))
    nb = buf.num_bodies
    ph = Physics(buf, make_params(pgs_iterations=5, flags=4))
    for _ in range(75):
        ph.step(nb, 0, buf.num_hull_verts, 10, DT, G)
    torch.cuda.synchronize()
    x = [buf[k][: n * nb].clone().reshape(nb, n)
         for k, n in (("body_pos", 3), ("body_quat", 4), ("body_vel", 3), ("body_omega", 3))]

    def grads():
        vel = x[2].clone().requires_grad_()
        out = rollout(ph, x[0], x[1], vel, x[3], frames=1, substeps=4)
        assert out[0].grad_fn.ckpt.dtype == torch.float32
        assert out[0].grad_fn.ckpt.shape == (4, 13 * nb)
        (out[0].square().sum() + out[1].sum()).backward()
        return [*(y.detach() for y in out), vel.grad]

    want = grads()
    default = torch.get_default_dtype()
    torch.set_default_dtype(getattr(torch, name))
    try:
        got = grads()
    finally:
        torch.set_default_dtype(default)
    for a, b in zip(want, got):
        assert a.dtype == b.dtype == torch.float32 and torch.equal(a, b)
    ph.deinit()
