"""GPU tests of the HSP sort at the sizes where it changes form: one record, a
tile and one more or less, and runs that do not fill a merge pass.  With a
threshold below every seed's score and entropy off, each hit of random
sequences is an HSP, so the record count is the hit count of the seeds chosen."""
import numpy as np
import pytest

import oracle
from segalign_b200 import SeedFilter, build_sub_mat, host_revcomp, host_seeds
from tests.helpers import compare_segments, random_text

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 31, 33, 1023, 1024, 1025, 2049, 4097, 32_768, 32_769)


@pytest.fixture(scope="module")
def setup(built):
    rng = np.random.default_rng(21)
    T, Q = random_text(rng, 2_200_000, gc=0.5), random_text(rng, 400_000, gc=0.5)
    p = oracle.params(hspthresh=600, noentropy=True)
    idx, pos = oracle.build_table(T, p)
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos("12of19")
    sf.initialize_processor(False, 700_000, 19, build_sub_mat(910), 910, 600, True)
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.send_query_write_request(Q, 0)
    sf.rm_send_query_write_request()
    return dict(T=T, Q=Q, p=p, idx=idx, pos=pos, sf=sf)


def _prefix(seeds, n, count):
    """The shortest prefix of the seeds with at least n HSPs (all of them if there are fewer)."""
    lo, hi = 1, len(seeds)
    while lo < hi:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if count(seeds[:mid]) >= n else (mid + 1, hi)
    return seeds[:lo]


@pytest.mark.parametrize("n", SIZES)
def test_plain_and_batched(setup, n):
    sf, p = setup["sf"], setup["p"]
    R, C = oracle.encode(setup["T"]), oracle.encode(setup["Q"])
    run = lambda s: oracle.seed_and_filter(p, R, C, setup["idx"], setup["pos"], s, False)[0]  # noqa: E731
    seeds = _prefix(host_seeds(setup["Q"], 0, len(setup["Q"]) - 19), n, lambda s: len(run(s)) - 1)
    want = run(seeds)
    assert len(want) - 1 == n
    compare_segments(sf.seed_and_filter(seeds, False, 0), want, f"{n} records")
    if len(seeds) <= 1 << 18:  # that entry point's limit
        compare_segments(sf.seed_and_filter_noalloc(seeds, False, 0), want, f"{n} records, no allocation")
    j = (seeds & np.uint64(0xffffffff)).astype(np.int64)
    cut = int(j[len(j) // 3])
    got = sf.seed_and_filter_batch([(0, 0, 0, cut), (0, 0, cut, int(j[-1]) + 1)])
    for g, s in zip(got, (seeds[j < cut], seeds[j >= cut])):
        if len(s):
            compare_segments(g, run(s), f"{n} batched")


@pytest.mark.parametrize("rev,exclude", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("n", [k for k in SIZES if k < 4000])
def test_repeat_masker(setup, n, rev, exclude):
    sf, T = setup["sf"], setup["T"]
    R = oracle.encode(T)
    C = oracle.rc_codes(R) if rev else R
    text = host_revcomp(T) if rev else T
    lo, hi = (100_000, 650_000) if rev else (330_000, 700_000)  # the main diagonal's last seeds lie in the window
    p = oracle.params(hspthresh=600, noentropy=True, rm_exclude_diag=exclude)
    run = lambda s: oracle.seed_and_filter(p, R, C, setup["idx"], setup["pos"], s, rev, 1, lo, hi)[0]  # noqa: E731
    seeds = host_seeds(text, 0, 330_010)
    if n < 1000:
        seeds = seeds[::-1][:20_000][::-1].copy()
    seeds = _prefix(seeds, n, lambda s: len(run(s)) - 1)
    sf.set_rm_exclude_diagonal(exclude)
    try:
        compare_segments(sf.rm_seed_and_filter(seeds, rev, lo, hi), run(seeds), f"{n} rm rev={rev} exclude={exclude}")
    finally:
        sf.set_rm_exclude_diagonal(False)


@pytest.fixture(scope="module")
def large(built):
    rng = np.random.default_rng(22)
    T, Q = random_text(rng, 2_200_000, gc=0.5), random_text(rng, 1_150_000, gc=0.5)
    p = oracle.params(hspthresh=600, noentropy=True)
    idx, pos = oracle.build_table(T, p)
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos("12of19")
    sf.initialize_processor(False, 1_200_000, 19, build_sub_mat(910), 910, 600, True)
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.send_query_write_request(Q, 0)
    R, C = oracle.encode(T), oracle.encode(Q)
    return sf, host_seeds(Q, 0, len(Q) - 19), lambda s: oracle.seed_and_filter(p, R, C, idx, pos, s, False)[0]


@pytest.mark.parametrize("n", [8191, 8192, 8193, 65_535, 65_536, 65_537, 131_071, 131_072, 131_073])
def test_limits_of_rank_passes(large, n):
    """One, two and three passes of eight runs each, and the merge passes above them."""
    sf, words, run = large
    seeds = _prefix(words, n, lambda s: len(run(s)) - 1)
    want = run(seeds)
    assert len(want) - 1 == n
    compare_segments(sf.seed_and_filter(seeds, False, 0), want, f"{n} records")
