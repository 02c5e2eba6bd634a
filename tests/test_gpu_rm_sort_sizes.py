"""GPU test of a repeat-masker call's sorts at the limits of their passes (one
tile, one, two and three rank passes, merge passes), the sizes being those of the
HSP set before the diagonal unique, which removes some: lists equal the oracle's."""
import numpy as np
import pytest

import oracle
from segalign_b200 import SeedFilter, build_sub_mat, host_revcomp, host_seeds
from tests.helpers import compare_segments, random_text

pytestmark = pytest.mark.gpu

HALF = 1_600_000
LO, HI = HALF + 100, 2 * HALF - 100  # target window: seeds of the first half do not meet the main diagonal


def _diverged(rng, text):
    """A copy in which blocks of 60 bases stay, each with a weaker seed match 7 changed bases before it (the HSP of
    that one goes on into the block, whose own HSP ends there) and 150 random bases after it."""
    other = np.zeros(256, dtype=np.uint8)
    other[list(b"ACGT")] = list(b"TGCA")
    free = np.array([3, 5, 6, 9, 10])  # five of the seven bases that 12of19 leaves open
    copy = text.copy()
    for at in range(0, len(text) - 236, 236):
        copy[at + free] = other[text[at + free]]
        copy[at + 19:at + 26] = other[text[at + 19:at + 26]]
        copy[at + 86:at + 236] = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, 150)]
    return copy


def _prefix(seeds, n, count):
    """The shortest prefix of the seeds with at least n HSPs."""
    lo, hi, c_lo, c_hi = 0, len(seeds), 0, count(seeds)
    assert c_hi >= n
    while hi - lo > 1:  # HSPs come evenly: guess the place, a little to either side in turn
        guess = lo + int((hi - lo) * (n - c_lo) / (c_hi - c_lo))
        guess += 40 if n - c_lo > c_hi - n else -40
        mid = min(max(guess, lo + 1), hi - 1) if hi - lo > 64 else (lo + hi) // 2
        c = count(seeds[:mid])
        if c >= n:
            hi, c_hi = mid, c
        else:
            lo, c_lo = mid, c
    return seeds[:hi]


@pytest.fixture(scope="module")
def setup(built):
    rng = np.random.default_rng(71)
    first = np.frombuffer(random_text(rng, HALF, gc=0.5), dtype=np.uint8)
    T = first.tobytes() + _diverged(rng, first).tobytes()
    p = oracle.params(hspthresh=600, noentropy=True)
    idx, pos = oracle.build_table(T, p)
    # the table of the window alone: a plain call on it has the HSPs of the call before the diagonal unique
    keep = (pos + 19 >= LO) & (pos + 19 <= HI)
    cnt = np.concatenate([[0], np.cumsum(keep)])
    widx, wpos = cnt[idx].astype(np.uint32), pos[keep]
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos("12of19")
    sf.initialize_processor(False, 1_700_000, 19, build_sub_mat(910), 910, 600, True)
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.rm_send_query_write_request()
    R = oracle.encode(T)
    sides = {}
    for rev in (False, True):
        text = host_revcomp(T) if rev else T
        C = oracle.rc_codes(R) if rev else R
        a = HALF if rev else 0  # the other half's reverse complement comes first there
        seeds = host_seeds(text, a, a + HALF - 30)
        sides[rev] = (seeds, C)
    return dict(sf=sf, p=p, R=R, sides=sides, table=(idx, pos), window=(widx, wpos))


@pytest.mark.parametrize("n,rev,exclude", [(n, False, False) for n in (1024, 1025, 8192, 8193, 65_536, 65_537, 131_072,
                                                                       131_073)] +
                         [(n, rev, not rev) for n in (1025, 8193, 131_073) for rev in (False, True)])
def test_sizes_of_the_set(setup, n, rev, exclude):
    sf, p, R = setup["sf"], setup["p"], setup["R"]
    seeds, C = setup["sides"][rev]
    before = lambda s: oracle.seed_and_filter(p, R, C, *setup["window"], s, False)[0][1:]  # noqa: E731
    seeds = _prefix(seeds, n, lambda s: len(before(s)))
    assert len(before(seeds)) == n
    pe = oracle.params(hspthresh=600, noentropy=True, rm_exclude_diag=exclude)
    want = oracle.seed_and_filter(pe, R, C, *setup["table"], seeds, rev, 1, LO, HI)[0]
    # the unique removes some; on the minus strand, whose query starts are flipped, HSPs that hold others have other diagonals
    assert rev or len(want) - 1 < n
    sf.set_rm_exclude_diagonal(exclude)
    try:
        compare_segments(sf.rm_seed_and_filter(seeds, rev, LO, HI), want, f"{n} in the set, rev={rev}")
    finally:
        sf.set_rm_exclude_diagonal(False)
