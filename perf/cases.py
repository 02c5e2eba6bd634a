"""Workloads that time the seed-filter path through its public entry points.

Each case is one thing a user of the library has it do, over the range of sizes
it is used at: single SeedAndFilter calls (a contig, a 250 kbp chunk, chunks
with transitions), batched calls over the windows of a query, a query from host
text to HSP lists, the C++ seeder's concurrent calls, serving requests, a new
target block, and repeat-masker calls and whole self-alignments.

Sequences are the synthetic genomes of ``segalign_b200.synth``.  A target
belongs to its case, as an assembly stays resident while queries stream past
it; the query is a stretch of the workload's query that the seed picks.  Where
a call brings its own target, the seed makes that too.
The library holds one target and eight query buffers per process, so states of
one case share the target and own a query buffer each.

A pass gathers its HSP lists, as a program that goes on with them does, into an
array the program keeps: rows of four int32 (target start, query start, length,
score), the lists back to back, each call's list with the call's header row
first, and the lists' lengths beside them.
"""
from __future__ import annotations

import os
import weakref

import numpy as np
import torch

from segalign_b200 import SeedFilter, build_sub_mat, host_revcomp, host_seeds, synth

# The workload families of segalign_b200.synth: 1 = 1 Mbp x 1 Mbp with inserted
# segments, 2 = genome scale (GC 36%, 12% repeats), 4 = repeat-rich (GC 41%, 45% repeats).
SPAN = {"12of19": 19, "14of22": 22}
WEIGHT = {"12of19": 12, "14of22": 14}
FULL = {1: 1_000_000, 2: 100_000_000, 4: 600_000_000}

BASE = dict(family=2, target=100_000_000, shape="12of19", transition=False, xdrop=910, hspthresh=3000,
            noentropy=False, slots=2)


def listed():
    def case(name, kind, **kw):
        return {**BASE, **kw, "name": name, "kind": kind}

    return [
        # a short contig against a bacterial-size target: the smallest call, all latency
        case("call_contig", "call", family=1, target=1_000_000, positions=881, rev=False),
        # the default chunk of the seeder against the 1 Mbp test pair
        case("call_chunk_1mbp", "call", family=1, target=1_000_000, positions=250_000, rev=False),
        # the default chunk against the 100 Mbp genome, minus strand
        case("call_chunk_genome", "call", positions=250_000, rev=True),
        # an odd chunk with one transition allowed per seed (13 words per position), repeat-rich target
        case("call_transition", "call", family=4, target=30_000_000, transition=True, positions=100_003, rev=False),
        # many small ragged windows: the batched form with little work per unit; the heavier seed
        # shape, other thresholds and entropy off
        case("batch_windows_14of22", "batch", target=10_000_000, shape="14of22", xdrop=800, hspthresh=2600,
             noentropy=True, query=700_001, units=61, uneven=True),
        # windows of very uneven length over a long query, both strands: the largest
        case("batch_uneven_genome", "batch", query=24_000_000, units=40, uneven=True),
        # a new query from host text to HSP lists (upload, keys, batched call)
        case("query_batch_genome", "query_batch", query=2_500_003, units=20, uneven=False),
        # a new query through the C++ seeder: concurrent plain calls on 16 host threads
        case("seeder_genome", "seeder", query=5_000_000, slots=12),
        # serving: six requests of 20 kbp to 1 Mbp submitted together
        case("serve_mix", "serve", query=2_000_000, requests=6),
        # a new target block: upload, seed table, and the first chunk on it
        case("target_block", "target_block", target=20_000_003, positions=50_000, rev=False),
        # repeat-masker call on one chunk of a repeat-rich sequence, windowed
        case("rm_call", "rm_call", family=4, target=30_000_000, positions=60_001, rev=False),
        # repeat-masker self-alignment of a whole sequence, from host text to coverage runs
        case("rm_whole", "rm_seeder", family=4, target=1_500_000, slots=4),
    ]


def draw(rng):
    def logint(a, b):
        return int(round(a * (b / a) ** rng.random()))

    kind = rng.choice(["call", "call", "call", "batch", "batch", "query_batch", "seeder", "serve", "target_block",
                       "rm_call", "rm_seeder"])
    family = rng.choice([1, 2, 2, 4])
    transition = rng.random() < 0.25
    c = dict(BASE, kind=kind, family=family, transition=transition,
             target=logint(60_000, 1_000_000) if family == 1 else logint(1_000_000, 40_000_000),
             shape=rng.choice(["12of19", "12of19", "12of19", "14of22"]), xdrop=rng.choice([910, 910, 700, 1200]),
             hspthresh=rng.choice([3000, 3000, 2500, 4000]), noentropy=rng.random() < 0.2)
    if kind in ("call", "target_block", "rm_call"):
        c.update(positions=logint(300, 60_000 if transition or kind == "rm_call" else 250_000), rev=rng.random() < 0.5)
        c["positions"] = min(c["positions"], c["target"] // 2)
    if kind == "target_block":
        c["target"] = min(c["target"], 20_000_000)
    if kind in ("batch", "query_batch"):
        c.update(query=logint(30_000, 1_000_000 if transition or family == 4 else 6_000_000), units=rng.randint(1, 60),
                 uneven=rng.random() < 0.5)
    if kind == "seeder":
        c.update(query=logint(30_000, 600_000 if transition or family == 4 else 5_000_000), slots=12)
    if kind == "serve":
        c.update(query=logint(200_000, 600_000 if transition or family == 4 else 3_000_000), requests=rng.randint(1, 12))
    if kind == "rm_seeder":
        c.update(family=4, target=logint(300_000, 2_000_000), transition=False, slots=4)
    return c


# ---- inputs --------------------------------------------------------------

def _windows(rng, length, span, units, uneven):
    """`units` windows of seed positions over both strands of a query, in seeder order."""
    last = length - span
    per = max(1, units // 2)
    if uneven:
        w = np.exp(rng.random(per) * np.log(200.0))
        cut = np.concatenate([[0], np.cumsum(w) / w.sum()])
    else:
        cut = np.linspace(0, 1, per + 1)
    cut = [int(x * last) for x in cut]
    fw = [(0, a, b) for a, b in zip(cut, cut[1:])]
    rc = [(1, last - b, last - a) for a, b in zip(cut, cut[1:])]
    return (fw + rc)[:units] if units > 1 else fw[:1]


# ---- the process's library ------------------------------------------------

_lib = dict(sf=None, config=None, target=None, workload=None, workload_key=None, serving=False, rm=None)
_owners: list = [None] * 8


class State:
    def __init__(self, case, sf):
        self.case, self.sf = case, sf


def _workload(case):
    key = (case["family"], case["target"])
    if _lib["workload_key"] != key:
        _lib["workload"] = synth.make(case["family"], scale=case["target"] / FULL[case["family"]])
        _lib["workload_key"] = key
    return _lib["workload"]


def _query(case, rng, n):
    """A stretch of n bases of the workload's query (at most nine tenths of it)."""
    q = _workload(case).query
    n = min(n, len(q) * 9 // 10)
    at = int(rng.integers(0, len(q) - n + 1))
    return q[at:at + n]


def _library(case):
    """The library set up for the case: processor parameters, and the resident target with its table."""
    config = tuple(case[k] for k in ("shape", "transition", "xdrop", "hspthresh", "noentropy", "slots"))
    if _lib["sf"] is None:
        _lib["sf"] = SeedFilter()
    sf = _lib["sf"]
    if _lib["serving"] and (_lib["config"] != config or _lib["target"] != (case["family"], case["target"])
                            or case["kind"] != "serve"):
        sf.serve_stop()
        _lib["serving"] = False
    if _lib["config"] != config:
        if _lib["config"] is not None:
            sf.shutdown_processor()
        os.environ["SA_SLOTS_PER_GPU"] = str(case["slots"])
        sf.initialize_interface(1)
        sf.generate_shape_pos(case["shape"])
        sf.initialize_processor(case["transition"], 250_000, SPAN[case["shape"]], build_sub_mat(case["xdrop"]),
                                case["xdrop"], case["hspthresh"], case["noentropy"])
        _lib["config"], _lib["target"] = config, None
    if case["kind"] in ("target_block", "rm_seeder"):
        _lib["target"] = None  # each pass brings its own target
    elif _lib["target"] != (case["family"], case["target"]):
        sf.send_ref_write_request(_workload(case).target)
        sf.generate_seed_pos_table(None, 1, SPAN[case["shape"]], WEIGHT[case["shape"]])
        _lib["target"] = (case["family"], case["target"])
        _lib["rm"] = None
    if case["kind"] == "rm_call" and _lib["rm"] is None:
        sf.rm_send_query_write_request()
        _lib["rm"] = True
    sf.set_rm_exclude_diagonal(case["kind"].startswith("rm_"))
    return sf


def _buffer(state):
    for b, o in enumerate(_owners):
        if o is None or o() is None:
            _owners[b] = weakref.ref(state)
            return b
    raise RuntimeError("eight states of a case are alive at once")


def _seeds(case, text, rng, n):
    """Seed words of n positions somewhere in text, as the host seeder builds them (at least one)."""
    span = SPAN[case["shape"]]
    n = min(n, len(text) - span)
    at = int(rng.integers(0, len(text) - span - n + 1))
    return host_seeds(text, at, at + n, case["shape"], case["transition"]), at, at + n


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, span = case["kind"], SPAN[case["shape"]]
    sf = _library(case)
    s = State(case, sf)
    if kind == "target_block":
        w = synth.make(case["family"], seed=seed, scale=case["target"] / FULL[case["family"]])
        s.target = w.target
        query = w.query[:max(case["positions"] + span, min(len(w.query), 1_000_000))]
    elif kind == "rm_seeder":
        s.text = synth.make(case["family"], seed=seed, scale=case["target"] / FULL[case["family"]]).target
        return s
    elif kind == "rm_call":
        text = _workload(case).target
        text = host_revcomp(text) if case["rev"] else text
        s.seeds, a, b = _seeds(case, text, rng, case["positions"])
        # a window of a fifth of the sequence around the chunk (the driver's neighbour windows)
        mid, L = (a + b) // 2, len(text)
        mid = L - 1 - mid if case["rev"] else mid
        s.window = (max(0, mid - L // 10), min(L, mid + L // 10))
        return s
    else:
        n = case["query"] if "query" in case else max(4 * case["positions"], 100_000)
        query = _query(case, rng, n)
    if kind == "serve":
        # requests of log-uniform length cut from the query
        w = np.exp(rng.random(case["requests"]) * np.log(50.0))
        cut = [int(x) for x in np.concatenate([[0], np.cumsum(w) / w.sum()]) * len(query)]
        s.requests = [query[a:b] for a, b in zip(cut, cut[1:]) if b - a > 64]
        if not _lib["serving"]:
            sf.serve_start(interval_size=10_000_000, interval_overlap=50_000, chunk_size=250_000, strands=3)
            _lib["serving"] = True
        return s
    s.buffer = _buffer(s)
    s.query = query
    if kind in ("query_batch", "seeder"):
        if kind == "query_batch":
            s.units = [(s.buffer, r, a, b) for r, a, b in _windows(rng, len(query), span, case["units"],
                                                                   case["uneven"])]
        return s
    sf.send_query_write_request(query, s.buffer)
    if kind == "batch":
        s.units = [(s.buffer, r, a, b) for r, a, b in _windows(rng, len(query), span, case["units"], case["uneven"])]
        sf.refresh_query_keys(s.buffer)
    else:
        s.seeds = _seeds(case, host_revcomp(query) if case["rev"] else query, rng, case["positions"])[0]
    return s


def _room(case):
    """Rows the program keeps for a pass's lists: well above what these sequences give."""
    n = case.get("positions") or 2 * case.get("query", case["target"])
    return 40_000 + int(n * (3.0 if case["family"] == 4 else 0.25 if case["target"] > 50_000_000 else 1.0))


def _gather(s, lists):
    """The lists (arrays of 16-byte records) into the state's array, and their lengths."""
    if not hasattr(s, "rows"):
        s.rows = torch.zeros((_room(s.case), 4), dtype=torch.int32)
        s.lengths = torch.zeros(64, dtype=torch.int64)
    at = 0
    for i, x in enumerate(lists):
        n = len(x)
        if n:
            s.rows[at:at + n].copy_(torch.from_numpy(x.view(np.int32).reshape(-1, 4)))
        s.lengths[i] = n
        at += n
    return [s.rows, s.lengths]


def run(s):
    c, sf = s.case, s.sf
    kind = c["kind"]
    if kind == "call":
        return _gather(s, [sf.seed_and_filter(s.seeds, c["rev"], s.buffer)])
    if kind == "batch":
        return _gather(s, sf.seed_and_filter_batch(s.units))
    if kind == "query_batch":
        sf.send_query_write_request(s.query, s.buffer)
        return _gather(s, sf.seed_and_filter_batch(s.units))
    if kind == "seeder":
        sf.send_query_write_request(s.query, s.buffer)
        fw, rc, _ = sf.seeder_run(s.query, buffer=s.buffer, strand=3, num_threads=16, interval_size=10_000_000,
                                  chunk_size=250_000, interval_overlap=50_000, shape=c["shape"],
                                  transition=c["transition"])
        return _gather(s, [fw, rc])
    if kind == "serve":
        ids = [sf.serve_submit(q) for q in s.requests]
        return _gather(s, [x for i in ids for x in sf.serve_wait(i)[:2]])
    if kind == "target_block":
        sf.send_ref_write_request(s.target)
        sf.generate_seed_pos_table(None, 1, SPAN[c["shape"]], WEIGHT[c["shape"]])
        return _gather(s, [sf.seed_and_filter(s.seeds, c["rev"], s.buffer)])
    if kind == "rm_call":
        return _gather(s, [sf.rm_seed_and_filter(s.seeds, c["rev"], *s.window)])
    runs, _ = sf.rm_seeder_run(s.text, lastz_interval_size=max(100_000, len(s.text) // 4 // 1000 * 1000),
                               num_threads=4, chunk_size=250_000, shape=c["shape"], transition=c["transition"])
    return _gather(s, [runs])


def work(case):
    """Bytes: texts or packed sequences and seed words once, one index pair per seed word, one table
    position per expected hit, and the target bases that the hits' 32-base windows touch, once.
    Operations: an add and a maximum for the 64 bases that the shortest scans of a hit cover."""
    S = 1 + WEIGHT[case["shape"]] if case["transition"] else 1
    kind, T = case["kind"], case["target"]
    n = case.get("positions") or 2 * case.get("query", T)
    if case.get("units") == 1:
        n //= 2
    words = n * S
    hits = words * max(T, 1) / 4.0 ** WEIGHT[case["shape"]]
    if kind == "rm_call":
        hits *= 0.2
    b = 8.0 * words + 4.0 * hits + min(32.0 * hits, T / 2.0) + n
    if kind in ("call", "rm_call", "target_block", "seeder"):
        b += 8.0 * words
    if kind in ("target_block", "rm_seeder"):
        b += 1.5 * T + 4.0 * T + 4.0 * 4 ** WEIGHT[case["shape"]]
    return {"bytes": float(b), "flops": float(hits * 128)}
