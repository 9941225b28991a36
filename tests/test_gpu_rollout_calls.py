"""The rollout calls against the calls for single substeps, bit for bit: states
and checkpoints of seevr_physics_rollout against step_async, gradients of
seevr_physics_adjoint_rollout against seevr_physics_adjoint_substep from the same
checkpoints; one and several substeps, with and without the frame graph, on the
default and another stream."""
import ctypes as C

import numpy as np
import pytest

from helpers import G
from seevr_b200 import Caps, Data, Physics, make_params
from seevr_b200 import _lib as L

pytestmark = pytest.mark.gpu

DT = 1.0 / 600.0
ROWS = ("body_pos", 3), ("body_quat", 4), ("body_vel", 3), ("body_omega", 3)


@pytest.mark.parametrize("steps, graph, side", [(1, False, False), (7, False, False), (7, True, False),
                                                (7, False, True)])
def test_calls(cuda, steps, graph, side):
    import torch

    d = Data.rollout(num_scenes=60, bodies=24, seed_base=5)
    buf = d.upload(cuda, Caps.for_data(d))
    nb, nhv, t = buf.num_bodies, buf.num_hull_verts, buf.tensors
    ph = Physics(buf, make_params(pgs_iterations=5, flags=4 | (2 if graph else 0)))
    for _ in range(75):  # bodies in contact
        ph.step(nb, 0, nhv, 10, 10 * DT, G)
    torch.cuda.synchronize()
    state = lambda: torch.cat([t[k][: n * nb] for k, n in ROWS])
    start = state()

    def put(x):
        for (k, n), part in zip(ROWS, torch.split(x, [n * nb for _, n in ROWS])):
            t[k][: n * nb].copy_(part)
        torch.cuda.synchronize()

    want = []
    for _ in range(steps):
        want.append(state())
        ph.step_async(nb, 0, nhv, 1, DT, G, frames=1)
        torch.cuda.synchronize()
    end = state()
    assert ph.read_counters()[1] > 10
    put(start)
    ckpt = torch.zeros(steps, 13 * nb, device=cuda)
    torch.cuda.synchronize()
    st = torch.cuda.Stream(cuda).cuda_stream if side else 1
    L.check(L.lib.seevr_physics_rollout(ph._h, nb, nhv, steps, DT, L.fptr(G, 3), ckpt.data_ptr(),
                                        C.c_void_p(st)))
    torch.cuda.synchronize()
    assert torch.equal(ckpt, torch.stack(want)) and torch.equal(state(), end)

    def grads():
        rng = np.random.default_rng(1)
        g = [torch.from_numpy(rng.standard_normal(n * nb)).to(cuda) for _, n in ROWS]
        g.append(torch.zeros(nb, dtype=torch.float64, device=cuda))
        torch.cuda.synchronize()
        return g, L.AdjointGrads(*[x.data_ptr() for x in g])

    a, ga = grads()
    for k in reversed(range(steps)):
        put(ckpt[k])
        L.check(L.lib.seevr_physics_adjoint_substep(ph._h, nb, nhv, DT, L.fptr(G, 3), C.byref(ga)))
    b, gb = grads()
    L.check(L.lib.seevr_physics_adjoint_rollout(ph._h, nb, nhv, steps, DT, L.fptr(G, 3),
                                                ckpt.data_ptr(), C.byref(gb)))
    for x, y in zip(a, b):
        assert torch.equal(x, y) and torch.isfinite(x).all()
    ph.deinit()
