"""GPU tests of a plain call's lookup at the sizes where its split can go wrong: words per thread, per CTA round and
per grid, whole and ragged, every seed word and not, with one MAX_HITS iteration and several."""
import numpy as np
import pytest

import oracle
from segalign_b200 import SeedFilter, build_sub_mat, host_seeds
from tests.helpers import compare_segments, random_text

pytestmark = pytest.mark.gpu

WORDS = [1, 3, 4, 5, 591, 592, 593, 2047, 2048, 2049, 148 * 2048 - 3, 148 * 2048 + 5]


@pytest.fixture(scope="module")
def setup(built):
    rng = np.random.default_rng(11)
    T = np.frombuffer(random_text(rng, 4_000), dtype=np.uint8).copy()
    Q = np.frombuffer(random_text(rng, 24_500), dtype=np.uint8).copy()
    for k in range(6):  # copies of target pieces, one of them twice
        Q[4_000 * k + 10:4_000 * k + 210] = T[600 * (k // 2):600 * (k // 2) + 200]
    T, Q = T.tobytes(), Q.tobytes()
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos("12of19")
    sf.initialize_processor(True, 30_000, 19, build_sub_mat(910), 910, 3000, False)
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.send_query_write_request(Q, 0)
    return sf, T, Q, host_seeds(Q, 0, len(Q) - 19, "12of19", True)


@pytest.mark.parametrize("n", WORDS)
@pytest.mark.parametrize("max_hits", [0, 50])
def test_words_of_a_call(setup, n, max_hits):
    sf, T, Q, words = setup
    assert len(words) > WORDS[-1]
    at = min(100, len(words) - n)
    seeds = words[at:at + n]
    p = oracle.params(transition=True, max_hits=max_hits or (1 << 40))
    idx, pos = oracle.build_table(T, p)
    want, st = oracle.seed_and_filter(p, oracle.encode(T), oracle.encode(Q), idx, pos, seeds, False)
    assert max_hits == 0 or n < 2047 or st["num_iter"] > 1
    sf.set_max_hits(max_hits)
    try:
        compare_segments(sf.seed_and_filter(seeds, False, 0), want, f"{n} words")
    finally:
        sf.set_max_hits(0)
    cs = sf.last_call_stats()
    assert cs["num_hits"] == st["num_hits"] and cs["survivors"] == st["survivors"]
    assert cs["tiles"] == st["tiles_right"] + st["tiles_left"]
