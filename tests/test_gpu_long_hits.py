"""GPU test of the statistic `long_hits`: it counts hits, also where both sides
of a hit pass the lane cap and where the queue is full."""
import numpy as np
import pytest

import oracle
from segalign_b200 import SeedFilter, build_sub_mat, host_seeds
from tests.helpers import compare_segments, random_text

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("queue", [1 << 20, 5, 1])
def test_hits_with_two_long_sides_count_once(built, queue, monkeypatch):
    rng = np.random.default_rng(41)
    T = random_text(rng, 12_000)
    Q = random_text(rng, 1000) + T[4000:7000] + random_text(rng, 1000)
    p = oracle.params()
    idx, pos = oracle.build_table(T, p)
    monkeypatch.setenv("SA_LONG_CAP", str(queue))
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos("12of19")
    sf.initialize_processor(False, 10_000, 19, build_sub_mat(910), 910, 3000, False)
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.send_query_write_request(Q, 0)
    for k in (1, 2, 33, 200):
        # every k-th part of the copy's middle: words left out, so that no chains form
        seeds = np.concatenate([host_seeds(Q, j, j + 1) for j in np.linspace(1400, 3400, k).astype(int)])
        want, st = oracle.seed_and_filter(p, oracle.encode(T), oracle.encode(Q), idx, pos, seeds, False)
        assert st["survivors"] == k  # the hits of the copy, which ends 350 bases or more away; two others are chance hits
        compare_segments(sf.seed_and_filter(seeds, False, 0), want, f"{k} hits")
        cs = sf.last_call_stats()
        assert cs["long_hits"] == k and cs["tiles"] == st["tiles_right"] + st["tiles_left"], k
    monkeypatch.delenv("SA_LONG_CAP")
    sf.initialize_processor(False, 10_000, 19, build_sub_mat(910), 910, 3000, False)
