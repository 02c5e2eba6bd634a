"""GPU tests of scans with scores and X-drops far from the default table's: the
end of a sequence ends every scan whatever these are.  HSP lists and the
statistics of every hit equal the oracle's."""
import numpy as np
import pytest

import oracle
from segalign_b200 import SeedFilter, build_sub_mat, host_revcomp, host_seeds
from tests.helpers import compare_segments, random_text

pytestmark = pytest.mark.gpu


def _filter(p, sub, xdrop, hspthresh):
    """A filter with these scores, and the oracle's parameters set alike."""
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos("12of19")
    sf.initialize_processor(False, 20_000, 19, sub, xdrop, hspthresh, bool(p.noentropy))
    p.sub_mat[:] = [int(x) for x in sub]
    p.xdrop, p.hspthresh = xdrop, hspthresh
    return sf


def _pair(rng, n):
    """A target and a query of its pieces, from like to unlike."""
    t = np.frombuffer(random_text(rng, n), dtype=np.uint8).copy()
    q = t.copy()
    for k in range(0, n, 300):
        m = rng.random(len(q[k:k + 300])) < 0.3 * k / n
        q[k:k + 300][m] = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, int(m.sum()))]
    return t.tobytes(), q.tobytes()


def _check_calls(sf, p, T, Q, calls, what):
    """Plain calls and one batched call on the windows `calls` of both strands."""
    idx, pos = oracle.build_table(T, p)
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.send_query_write_request(Q, 0)
    R, units, wants, total = oracle.encode(T), [], [], 0
    for rev in (False, True):
        text = host_revcomp(Q) if rev else Q
        for a, b in calls:
            seeds = host_seeds(text, a, b)
            want, st = oracle.seed_and_filter(p, R, oracle.encode(text), idx, pos, seeds, rev)
            compare_segments(sf.seed_and_filter(seeds, rev, 0), want, f"{what} {(rev, a, b)}")
            cs = sf.last_call_stats()
            assert cs["tiles"] == st["tiles_right"] + st["tiles_left"], (what, rev, a, b)
            assert cs["survivors"] == st["survivors"] and cs["hits_extended"] == st["hits_extended"], (what, rev, a, b)
            units.append((0, int(rev), a, b))
            wants.append(want)
            total += st["tiles_right"] + st["tiles_left"]
    for u, got, want in zip(units, sf.seed_and_filter_batch(units), wants):
        compare_segments(got, want, f"{what} unit {u}")
    assert sf.last_call_stats()["tiles"] == total, what
    return wants


@pytest.mark.parametrize("xdrop", [1 << 25, 1 << 28, 1 << 30, 2_000_000_000, 2**31 - 1])
@pytest.mark.parametrize("lane_cap", [64, 8192])
def test_scans_that_only_a_sequence_end_stops(built, xdrop, lane_cap):
    """lane_cap 64: the warp kernel ends them; 8192: the lanes do."""
    T, Q = _pair(np.random.default_rng(31), 3001)
    p = oracle.params()
    sf = _filter(p, build_sub_mat(910), xdrop, 3000)
    saved = sf.get_tuning()
    sf.set_tuning(lane_cap=lane_cap)
    try:
        L = len(Q) - 19
        wants = _check_calls(sf, p, T, Q, ((0, L), (700, 1200), (L - 40, L)), f"xdrop {xdrop} lane_cap {lane_cap}")
        assert sum(len(w) - 1 for w in wants) > 0
    finally:
        sf.set_tuning(lane_cap=saved["lane_cap"])


@pytest.mark.parametrize("end", [-9100, -911, -910, -100, 0, 60])
@pytest.mark.parametrize("xdrop", [910, 3000])
def test_scores_of_codes_past_the_ends(built, end, xdrop):
    """Hits next to both ends of both sequences: what a table gives for the code
    that fills the padding (E) is never counted, in lists or in tiles."""
    T, Q = _pair(np.random.default_rng(32), 2011)
    p = oracle.params()
    sub = build_sub_mat(910).reshape(8, 8)
    sub[7, :] = sub[:, 7] = end
    sf = _filter(p, sub.reshape(-1), xdrop, 2200)
    for t, q in ((T, Q), (T[:150], Q[:131]), (T[700:], Q[700:1100]), (T[:411], T[303:411]), (T[1900:], T[1900:]),
                 (T[77:120], T[77:120])):
        L = len(q) - 19
        _check_calls(sf, p, t, q, ((0, L), (0, min(L, 70)), (max(0, L - 70), L)), f"E {end} xdrop {xdrop} {len(t)}x{len(q)}")


@pytest.mark.parametrize("bits", [24, 26])
def test_large_scores_in_the_warp_kernel(built, bits):
    """Scores whose sums over 8 bases pass 2^28, totals below 2^31; every hit passes the lane cap."""
    rng = np.random.default_rng(33)
    T = np.frombuffer(random_text(rng, 6000, gc=0.5), dtype=np.uint8)
    Q = np.frombuffer(random_text(rng, 4000, gc=0.5), dtype=np.uint8).copy()
    for k in range(0, 4000, 40):
        at = int(rng.integers(0, 5900))
        Q[k + 9:k + 31] = T[at:at + 22]
    sub = np.full((8, 8), -(1 << bits), dtype=np.int32)
    np.fill_diagonal(sub[:4, :4], 1 << bits)
    p = oracle.params(noentropy=True)
    sf = _filter(p, sub.reshape(-1), 3 << bits, 14 << bits)
    saved = sf.get_tuning()
    sf.set_tuning(lane_cap=8, step_bases=8)
    try:
        L = len(Q) - 19
        wants = _check_calls(sf, p, T.tobytes(), Q.tobytes(), ((0, L), (L // 2, L)), f"scores of 2^{bits}")
        assert len(wants[0]) - 1 > 50 and max(int(w["score"].max()) for w in wants) < 31 << bits
    finally:
        sf.set_tuning(lane_cap=saved["lane_cap"], step_bases=saved["step_bases"])
