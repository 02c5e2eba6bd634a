"""GPU test of the seed-table build over target lengths around its work units
(8-base words, CTA ranges, sort tiles), any step, both shapes, masked and N
bases, and of rebuilding larger, smaller and sparser tables over one another:
the device table equals the oracle's."""
import numpy as np
import pytest

import oracle
from segalign_b200 import SeedFilter, build_sub_mat
from tests.helpers import random_text

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,span,weight", [("12of19", 19, 12), ("110111", 6, 5)])
def test_table_over_lengths_and_steps(built, shape, span, weight):
    p = oracle.params(shape=shape)
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos(shape)
    sf.initialize_processor(False, 10_000, span, build_sub_mat(910), 910, 3000, False)
    rng = np.random.default_rng(5)
    for n, step, lower in ((300_001, 1, 0.02), (span + 1, 1, 0.0), (span + 9, 1, 0.0), (2055, 1, 0.01), (2_100_007, 1, 0.0),
                           (4096 + span, 1, 0.05), (50_000, 3, 0.02), (50_003, 7, 0.0), (9000, 1, 1.0), (700_000, 2, 0.001)):
        T = random_text(rng, n, lower=lower, nfrac=0.001 if n > 1000 else 0.0)
        sf.send_ref_write_request(T)
        sf.generate_seed_pos_table(None, step, span, weight)
        it, pt = sf.get_seed_pos_table()
        want_i, want_p = oracle.build_table(T, p, step)
        assert np.array_equal(it, want_i) and np.array_equal(pt, want_p), (n, step, lower)
