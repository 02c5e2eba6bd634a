"""GPU test of single calls with more hits than one sweep's list is sure to hold:
their sweep runs in segments, once where the number of seed words tells it
beforehand and a second time where it does not; lists and statistics equal the
oracle's, and the kernel launches are those of such runs."""
import numpy as np
import pytest

import oracle
from segalign_b200 import SeedFilter, build_sub_mat, host_seeds
from tests.helpers import compare_segments, random_text

pytestmark = pytest.mark.gpu

SHAPE, SPAN, WEIGHT = "110111", 6, 5


def _setup(T, Q, chunk):
    p = oracle.params(shape=SHAPE)
    idx, pos = oracle.build_table(T, p)
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos(SHAPE)
    sf.initialize_processor(False, chunk, SPAN, build_sub_mat(910), 910, 3000, False)
    sf.send_ref_write_request(T)
    sf.generate_seed_pos_table(None, 1, SPAN, WEIGHT)
    sf.send_query_write_request(Q, 0)
    seeds = host_seeds(Q, 0, len(Q) - SPAN, SHAPE)
    want, st = oracle.seed_and_filter(p, oracle.encode(T), oracle.encode(Q), idx, pos, seeds, False)
    assert 1 < len(want) <= 1024  # one sort kernel
    return sf, seeds, want, st


def _run_launches(hits, cap):
    """Kernels of one run: lookup 3; sweep, scans and finish per segment; long hits."""
    return 3 + 3 * -(-hits // (4 * cap)) + 1


def _check(sf, call, seeds, want, st, launches):
    l0 = sf.kernel_launches()
    got = call(seeds, False, 0)
    assert sf.kernel_launches() - l0 == launches + 1  # and the sort
    compare_segments(got, want, "segments")
    return st["tiles_right"] + st["tiles_left"], st["survivors"]


@pytest.mark.parametrize("cap,gc,known", [(1024, 0.36, True), (4096, 0.36, True), (12_000, 0.25, False)])
def test_plain_call(built, cap, gc, known, monkeypatch):
    rng = np.random.default_rng(51)
    T, Q = random_text(rng, 6000, gc=gc), random_text(rng, 6000, gc=gc)
    Q = Q[:2000] + T[3000:3300] + Q[2300:]
    monkeypatch.setenv("SA_LIST_CAP", str(cap))
    sf, seeds, want, st = _setup(T, Q, 10_000)
    assert (len(seeds) * (len(T) - SPAN) / 4 ** WEIGHT > 4 * cap) == known and st["num_hits"] > 4 * cap
    launches = 1 + _run_launches(st["num_hits"], cap)  # a slot's first call clears its HSP set
    if not known:
        launches += 3 + 3 + 1 + 1  # a run whose list was too small, and the set cleared again
    stats = _check(sf, sf.seed_and_filter, seeds, want, st, launches)
    cs = sf.last_call_stats()
    assert (cs["tiles"], cs["survivors"]) == stats and cs["num_hits"] == st["num_hits"]
    monkeypatch.delenv("SA_LIST_CAP")
    sf.initialize_processor(False, 10_000, SPAN, build_sub_mat(910), 910, 3000, False)


def test_no_allocation_call(built):
    rng = np.random.default_rng(52)
    T, Q = random_text(rng, 200_000, gc=0.5), random_text(rng, 10_000, gc=0.5)
    Q = Q[:2000] + T[3000:3300] + Q[2300:]
    sf, seeds, want, st = _setup(T, Q, 20_000)
    sf.seed_and_filter_noalloc(seeds[:1], False, 0)  # leaves the HSP set empty
    _check(sf, sf.seed_and_filter_noalloc, seeds, want, st, _run_launches(st["num_hits"], 1 << 17))
