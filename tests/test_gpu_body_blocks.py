"""The body stage's bodies per block against the oracle, bit for bit: body
counts on both sides of the block sizes' edges (8 per block up to 4,736
bodies, 16 above), with small and large hulls."""
import pytest

import pyoracle
from helpers import DT, G, assert_bit_exact, gpu_run
from seevr_b200 import Caps, Data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scenes, lo, hi", [(1, 1, 1), (1, 7, 7), (1, 8, 8), (1, 9, 9), (591, 7, 7),
                                            (592, 7, 7), (593, 7, 7), (40, 230, 250)])
def test_body_counts(cuda, scenes, lo, hi):
    d = Data.batch(num_scenes=scenes, min_bodies=lo, max_bodies=hi, seed_base=3)
    caps = Caps.for_data(d)
    ref = pyoracle.run(d.arrays(), frames=1, substeps=3, dt=DT, gravity=G, pgs_iterations=2,
                       max_pairs=caps.max_pairs, max_contacts=caps.max_contacts)
    assert_bit_exact(gpu_run(d, cuda, substeps=3, pgs=2, caps=caps), ref)
