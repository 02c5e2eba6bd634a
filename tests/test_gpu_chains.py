"""GPU tests of the sweep and of chains (hits of one diagonal scanned once):
HSP lists and the statistics of every hit (tiles, survivors, hits extended) equal
the oracle's on sequences full of same-diagonal hits, at the places where a
chain starts, breaks or must not form: diverged copies, exact and tandem
repeats, soft-masked and N bases inside the window, sequence ends, call and
block limits, repeat-masker windows, seed lists and tables that do not hold
every window, and MAX_HITS iterations."""
import numpy as np
import pytest

import oracle
from segalign_b200 import SeedFilter, build_sub_mat, host_revcomp, host_seeds
from tests.helpers import compare_segments, random_text

pytestmark = pytest.mark.gpu

SPAN = {"12of19": (19, 12), "14of22": (22, 14), "110111": (6, 5)}


def _texts(seed, n=24_000):
    """A target with tandem arrays and exact repeats, and a query of its pieces at 0-35% divergence."""
    rng = np.random.default_rng(seed)
    t = np.frombuffer(random_text(rng, n), dtype=np.uint8).copy()
    for period, at, length in ((1, 500, 90), (2, 900, 200), (7, 2000, 700), (31, 4000, 1500), (170, 7000, 3400)):
        unit = t[at:at + period].copy()
        t[at:at + length] = np.tile(unit, length // period + 1)[:length]
    t[12_000:14_600] = t[15_000:17_600]  # one exact copy, across blocks of 1024
    q = t.copy()
    for k in range(0, n, 1500):  # pieces from no to strong divergence
        m = rng.random(1500) < 0.35 * (k / n)
        piece = q[k:k + 1500]
        m = m[:len(piece)]
        piece[m] = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, int(m.sum()))]
    for s in (t, q):
        for _ in range(25):
            at, k = int(rng.integers(0, n)), int(rng.integers(1, 40))
            s[at:at + k] |= 0x20
        s[rng.integers(0, n, 12)] = ord("N")
    return t.tobytes(), q.tobytes()


def _filter(shape="12of19", transition=False, xdrop=910, hspthresh=3000, noentropy=False, chunk=60_000):
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos(shape)
    sf.initialize_processor(transition, chunk, SPAN[shape][0], build_sub_mat(xdrop), xdrop, hspthresh, noentropy)
    return sf


def _check(sf, got, want, st, what):
    compare_segments(got, want, what)
    cs = sf.last_call_stats()
    assert cs["tiles"] == st["tiles_right"] + st["tiles_left"], what
    assert cs["survivors"] == st["survivors"], what
    assert cs["hits_extended"] == st["hits_extended"] and cs["num_hits"] == st["num_hits"], what


@pytest.mark.parametrize("shape,transition,xdrop,hspthresh,noentropy", [
    ("12of19", False, 910, 3000, False), ("12of19", True, 910, 3000, False), ("12of19", False, 700, 2200, True),
    ("14of22", True, 1500, 3000, False), ("110111", False, 910, 2000, False), ("12of19", False, 100_000, 3000, False),
    ("12of19", False, 699, 3000, False)])
def test_calls_and_batches(built, shape, transition, xdrop, hspthresh, noentropy):
    T, Q = _texts(3, 6_000 if shape == "110111" else 24_000)
    span, weight = SPAN[shape]
    p = oracle.params(xdrop=xdrop, hspthresh=hspthresh, noentropy=noentropy, shape=shape,
                      transition=transition)
    idx, pos = oracle.build_table(T, p)
    sf = _filter(shape, transition, xdrop, hspthresh, noentropy)
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, span, weight)
    sf.send_query_write_request(Q, 0)
    R, L = oracle.encode(T), len(Q) - span
    units, wants, surv = [], [], 0
    for rev in (False, True):
        text = host_revcomp(Q) if rev else Q
        codes = oracle.encode(text)
        for a, b in ((0, L), (1, 1030), (1030, 1031), (2040, 5001), (L - 700, L)):
            a, b = max(0, min(a, L - 1)), max(1, min(b, L))
            seeds = host_seeds(text, a, b, shape, transition)
            if not len(seeds):
                continue
            want, st = oracle.seed_and_filter(p, R, codes, idx, pos, seeds, rev)
            _check(sf, sf.seed_and_filter(seeds, rev, 0), want, st, f"call {(rev, a, b)}")
            units.append((0, int(rev), a, b))
            wants.append(want)
            surv += st["survivors"]
    for u, got, want in zip(units, sf.seed_and_filter_batch(units), wants):
        compare_segments(got, want, f"unit {u}")
    assert sf.last_call_stats()["survivors"] == surv


@pytest.mark.parametrize("lane_cap,step", [(64, 8), (512, 32)])
def test_long_queue_and_steps(built, lane_cap, step):
    """Chains whose first hit goes to the warp kernel, and other step lengths."""
    T, Q = _texts(5)
    p = oracle.params()
    idx, pos = oracle.build_table(T, p)
    sf = _filter()
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.send_query_write_request(Q, 0)
    saved = sf.get_tuning()
    sf.set_tuning(lane_cap=lane_cap, step_bases=step)
    try:
        seeds = host_seeds(Q, 0, len(Q) - 19)
        want, st = oracle.seed_and_filter(p, oracle.encode(T), oracle.encode(Q), idx, pos, seeds, False)
        _check(sf, sf.seed_and_filter(seeds, False, 0), want, st, "long queue")
        assert sf.last_call_stats()["long_hits"] > 0
    finally:
        sf.set_tuning(lane_cap=saved["lane_cap"], step_bases=saved["step_bases"])


@pytest.mark.parametrize("cap", [32, 2048, 20_000])
def test_list_overflow_and_segments(built, cap, monkeypatch):
    """A list too small for a call's hits (the call runs again without the sweep), and a batched pass
    of more hits than four lists (segments)."""
    T, Q = _texts(13)
    p = oracle.params()
    idx, pos = oracle.build_table(T, p)
    monkeypatch.setenv("SA_LIST_CAP", str(cap))
    sf = _filter()
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.send_query_write_request(Q, 0)
    R, C = oracle.encode(T), oracle.encode(Q)
    units, wants, surv = [], [], 0
    for a, b in ((0, len(Q) - 19), (18_500, 19_400), (3, 700)):
        seeds = host_seeds(Q, a, b)
        want, st = oracle.seed_and_filter(p, R, C, idx, pos, seeds, False)
        _check(sf, sf.seed_and_filter(seeds, False, 0), want, st, f"call {(cap, a, b)}")
        units.append((0, 0, a, b))
        wants.append(want)
        surv += st["survivors"]
    for u, got, want in zip(units, sf.seed_and_filter_batch(units), wants):
        compare_segments(got, want, f"unit {u}")
    assert sf.last_call_stats()["survivors"] == surv
    monkeypatch.delenv("SA_LIST_CAP")
    _filter()


def test_hits_that_are_not_every_seed_match(built):
    """Words left out, repeated, reordered or shifted, sparse tables (step 3, a host table with positions left out),
    a table of another target, and MAX_HITS iterations: every hit is scanned for itself."""
    T, Q = _texts(7)
    p = oracle.params()
    idx, pos = oracle.build_table(T, p)
    R, C = oracle.encode(T), oracle.encode(Q)
    sf = _filter()
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.send_query_write_request(Q, 0)
    full = host_seeds(Q, 0, len(Q) - 19)
    moved = full.copy()
    moved[5000] = (moved[5000] >> np.uint64(32) << np.uint64(32)) | (moved[5000] + np.uint64(1) & np.uint64(0xffffffff))
    for what, seeds in (("left out", np.delete(full, slice(9, None, 7))), ("twice", np.concatenate([full, full[4000:4100]])),
                        ("reversed", full[::-1].copy()), ("another key", np.where(np.arange(len(full)) == 6000, full[10], full)),
                        ("moved", moved), ("last word missing inside", np.delete(full, len(full) - 2))):
        want, st = oracle.seed_and_filter(p, R, C, idx, pos, seeds, False)
        _check(sf, sf.seed_and_filter(seeds, False, 0), want, st, what)
    sf.set_max_hits(4000)
    try:
        pm = oracle.params(max_hits=4000)
        want, st = oracle.seed_and_filter(pm, R, C, idx, pos, full, False)
        assert st["num_iter"] > 1
        _check(sf, sf.seed_and_filter(full, False, 0), want, st, "iterations")
        # a batched unit has at most 16 iterations
        seeds = host_seeds(Q, 0, 2100)
        want, st = oracle.seed_and_filter(pm, R, C, idx, pos, seeds, False)
        assert 1 < st["num_iter"] <= 16
        compare_segments(sf.seed_and_filter_batch([(0, 0, 0, 2100)])[0], want, "iterations, batched")
    finally:
        sf.set_max_hits(0)
    sf.generate_seed_pos_table(None, 3, 19, 12)
    i3, p3 = oracle.build_table(T, p, 3)
    want, st = oracle.seed_and_filter(p, R, C, i3, p3, full, False)
    _check(sf, sf.seed_and_filter(full, False, 0), want, st, "step 3")
    keep = np.random.default_rng(1).random(len(pos)) < 0.8
    cnt = np.add.reduceat(np.concatenate([keep, [False]]), np.minimum(np.concatenate([[0], idx[:-1]]), len(pos)))
    cnt[np.diff(np.concatenate([[0], idx])) == 0] = 0
    ik = np.cumsum(cnt).astype(np.uint32)
    sf.send_seed_pos_table(ik, pos[keep])
    want, st = oracle.seed_and_filter(p, R, C, ik, pos[keep], full, False)
    _check(sf, sf.seed_and_filter(full, False, 0), want, st, "host table")


@pytest.mark.parametrize("transition", [False, True])
def test_repeat_masker_windows(built, transition):
    """Self alignment: the main diagonal is one match, cut by the window, masked bases and the chunk."""
    T, _ = _texts(11)
    p = oracle.params(transition=transition, rm_exclude_diag=True)
    idx, pos = oracle.build_table(T, p)
    sf = _filter(transition=transition)
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.rm_send_query_write_request()
    sf.set_rm_exclude_diagonal(True)
    R = oracle.encode(T)
    RC = oracle.rc_codes(R)
    try:
        for rev in (False, True):
            text = host_revcomp(T) if rev else T
            for a, b, lo, hi in ((0, len(T) - 19, 0, len(T)), (3000, 9000, 4111, 12_345), (11_000, 17_000, 12_100, 16_001)):
                seeds = host_seeds(text, a, b, "12of19", transition)
                want, st = oracle.seed_and_filter(p, R, RC if rev else R, idx, pos, seeds, rev, 1, lo, hi)
                _check(sf, sf.rm_seed_and_filter(seeds, rev, lo, hi), want, st, f"rm {(rev, a, b, lo, hi)}")
    finally:
        sf.set_rm_exclude_diagonal(False)
