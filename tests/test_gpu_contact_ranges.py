"""Each bundle's run of contacts, taken from the offsets of the pair rows and of
the pairs' contacts, bit for bit against the oracle: bundles with and without
contacts, and lists cut by the pair or the contact capacity, past which a
bundle owns nothing."""
import dataclasses

import pytest

import pyoracle
from helpers import DT, G, assert_bit_exact, gpu_run
from seevr_b200 import Caps, Data, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cut", [{}, {"max_pairs": 40}, {"max_pairs": 1}, {"max_contacts": 11},
                                 {"max_contacts": 1}])
@pytest.mark.parametrize("bundle", [1, 150])
def test_ranges(cuda, cut, bundle):
    d = Data.batch(num_scenes=24, min_bodies=1, max_bodies=120, seed_base=31)
    caps = dataclasses.replace(Caps.for_data(d), **cut)
    ref = pyoracle.run(d.arrays(), frames=50, substeps=10, dt=DT, gravity=G, pgs_iterations=3,
                       max_pairs=caps.max_pairs, max_contacts=caps.max_contacts)
    assert ref["num_contacts"] > 11 or cut
    got = gpu_run(d, cuda, frames=50, pgs=3, caps=caps,
                  params=make_params(pgs_iterations=3, bundle_bodies=bundle))
    assert_bit_exact(got, ref)
