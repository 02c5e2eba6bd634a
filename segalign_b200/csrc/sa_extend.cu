// sa_extend.cu — ungapped X-drop extension of every seed hit, HSP keep/score
// (entropy adjustment) and survivor compaction.
//
// Reference: find_hsps (src/seed_filter.cu:204-624; repeat-masker variant
// repeat_masker_src/seed_filter.cu:249-688) and compress_output (:626-652;
// rm :690-721).  The reference runs one warp per hit over 32-base tiles with
// four shuffle scans per tile.  Its result does not depend on the tile width.
// For each direction it is defined per position:
//   S(o) = running score, M(o) = max(0, max S up to o),
//   stop at the first o with M(o) - S(o) > xdrop or at the sequence edge,
//   best = max over o < stop, pos = first o reaching best (right: -1 if
//   best == 0; left: 0).
// This file computes the same quantities in two phases:
//   phase A, for scores and steps that sa_sweep_params admits: sa_k_sweep scores
//     the bases near every hit, which finishes the chance hits, and drops hits
//     whose HSP another hit of the diagonal gives; sa_k_scan goes on with the
//     others' sides; sa_k_finish counts and keeps.
//   phase A, general form (sa_k_extend_lane): one hit per lane.  A warp keeps its 32 lanes
//     busy by handing out the next hits of its tile, in order, to lanes that
//     finish.  Hits are expanded on the fly from the compacted seed
//     list.  The short random-hit extensions that dominate the hit count
//     finish here in a few steps.
//   phase B (sa_k_extend_warp): hits whose extension passes `lane_cap` bases in
//     one direction move to a queue and are redone by a warp per side,
//     256 bases per step.  Each lane scans 8 bases; warp scans carry the
//     running sum and maximum.
// Kept HSPs, with their dedup scope, go into the call's set of distinct HSPs
// (SaHashSet), which the dedup stage compacts and sorts.
#include <algorithm>
#include <climits>
#include <mutex>

#include "sa_launch.h"
#include "sa_radix.cuh"

#define SA_FULL 0xffffffffu
#define SA_LANE_TABLES 256  // lane kernel: the 64-entry score table

struct SaExtK {
    const uint32_t* ref;
    uint32_t ref_len;
    const uint32_t* pos_table;
    SaSeedList cs;
    const SaUnit* units;
    SaCounters* ctr;
    SaLongHit* long_q;
    uint64_t long_cap;
    SaHashSet hset;
    uint32_t seed_size;
    int32_t xdrop, hspthresh, noentropy;
    uint32_t lane_cap;
    uint32_t tile_hits;
    uint32_t substeps;  // steps per lane-kernel iteration (at most)
    uint32_t switch_now;  // 1: a lane starts its left side in the step after its right side ends
    uint32_t windowed;    // 1: hits outside their unit's rm window are dropped from the tiles
    // chains of hits on one diagonal (see there); chain = 0: every hit is scanned
    uint32_t chain;
    uint32_t gap;         // largest distance to the hit before
    int32_t match, swing; // smallest match score, and that minus the lowest mismatch score
    uint32_t mismatches;  // as many mismatches in a row cannot stop a scan
    uint32_t shift[16];   // shape positions, the first one again in the unused places
    uint4* list;          // hits the sweep leaves to the scans, two words of 16 bytes each:
                          // {rl, ql, scope, unit | SA_CHAIN_NEXT}, {SaSwept}
    uint64_t list_cap;    // 0: no sweep
    uint4* scanned;       // per list record and side (right, left): {best, its offset (-1: best is 0), start and
                          // depth of the step that stops}
};

// Largest compacted seed c in [0, nnz) with E[c] <= h (E strictly increasing,
// E[0] == 0 <= h).  Warp-cooperative 32-ary search; all lanes get the result.
__device__ __forceinline__ uint64_t sa_warp_find_seed(const uint64_t* __restrict__ E, uint64_t nnz, uint64_t h) {
    const int lane = threadIdx.x & 31;
    uint64_t lo = 0, hi = nnz;
    while (hi - lo > 32) {
        uint64_t step = (hi - lo + 31) / 32;
        uint64_t probe = lo + (uint64_t)lane * step;
        bool ok = probe < hi && E[probe] <= h;
        uint32_t m = __ballot_sync(SA_FULL, ok);
        uint64_t k = 31 - __clz(m);
        uint64_t nlo = lo + k * step;
        hi = (nlo + step < hi) ? nlo + step : hi;
        lo = nlo;
    }
    uint64_t probe = lo + lane;
    bool ok = probe < hi && E[probe] <= h;
    uint32_t m = __ballot_sync(SA_FULL, ok);
    return lo + (31 - __clz(m));
}

// Entropy factor and keep/score of one HSP (src/seed_filter.cu:580-621).
// c[] are the match counts per base over the HSP, already summed.
__device__ __forceinline__ void sa_keep_score(int total, int ext, const int* cnt, bool entropy_branch,
                                              int hspthresh, int* keep, int* score) {
    if (!entropy_branch) {
        // E = 1.0: (int)((double)(float)total * 1.0) == (int)(float)total, score == total
        *keep = (int)(float)total >= hspthresh;
        *score = total;
        return;
    }
    double E = 1.0;  // entropy[warp_id] = 1.0f
    {
        short c0 = (short)cnt[0], c1 = (short)cnt[1], c2 = (short)cnt[2], c3 = (short)cnt[3];
        if ((int)c0 + (int)c1 + (int)c2 + (int)c3 >= 20) {
            double n = (double)(ext + 1);
            double e = 0.0;
            // one log at a time (same accumulation order): keeps the register peak low
#pragma unroll 1
            for (int b = 0; b < 4; ++b) {
                const short cb = b == 0 ? c0 : b == 1 ? c1 : b == 2 ? c2 : c3;
                double q = (double)cb / n;
                double lg = (cb != 0) ? log((double)cb / n) : 0.0;
                e = fma(q, lg, e);
            }
            E = -e / (double)logf(4.0f);
        }
    }
    *keep = (int)(((double)(float)total) * E) >= hspthresh;
    *score = E > 0 ? (int)((double)total * E) : 0;
}

__device__ __forceinline__ bool sa_entropy_branch(const SaExtK& a, int total) {
    return !a.noentropy && total >= a.hspthresh && total <= 3 * a.hspthresh;
}

// ---------------------------------------------------------------------------
// Phase A: one hit per lane.
//
// A warp takes tiles of consecutive hits from a global counter and expands
// each tile once into shared memory ({ref_loc, query_loc, scope, unit} per
// hit).  At the top of every iteration the lanes without a hit take the next
// records of the tile, in order, and start them in the same iteration.
// Both directions of a hit run the same rightward scan: the left
// extension from (rl, ql) is the right extension from (ref_len - rl,
// qlen - ql) in the reversed copies that follow every packed sequence, so
// lanes in different directions execute the same instructions.  A step
// scores STEP bases as 8-base windows; the target and query words of the
// next step are loaded while the current one is scored.
//
// Fast scoring form.  Inside a step, scores are kept relative to the best
// score at the step start and packed with the base index k (0..STEP-1):
//     P(k) = SCALE * (S(k) - best_in) + (STEP - 1 - k),   SCALE = 2 * STEP,
// so a running max over P yields the best score together with the FIRST base
// that reached it; the best carried in from earlier steps enters as
// STEP, which no base of the step ties.  The X-drop stop test runs once
// per 8-base window: with m = the window's minimum score and b = the best
// score at the window's end, a base of the window stops the scan iff
// b - m > xdrop, provided 7 * max(0, max_sub) <= xdrop (max_sub = largest
// substitution score).  If b was reached at or before the minimum's base,
// that base itself has best - S = b - m; otherwise b - m is a climb over at
// most 7 bases, <= xdrop, and no base has best - S above b - m.  The same
// bound shows that no base after a stop in the window can raise the best
// (that takes a climb of more than xdrop), so the window's best is the best
// at the stop.  Bases past the sequence end score -(xdrop + 1): the first of
// them stops the scan.  The test runs on the packed values themselves:
// with B = SCALE * b + i (i in 0..STEP) and min = SCALE * m + j (j in
// 0..STEP-1), b - m > xdrop  <=>  B - min > SCALE * xdrop + STEP.
// Parameters outside the bound use the exact form, which tests every base.
// ---------------------------------------------------------------------------
// Byte b of lo (hi) = byte offset ((q << 3) | r) * 4 of the score of base 2b
// (2b+1) in a 64-entry int table; codes are 0..7, so a byte never carries.
__device__ __forceinline__ void sa_merge8(uint32_t rw, uint32_t qw, uint32_t& lo, uint32_t& hi) {
    lo = ((qw & 0x07070707u) << 5) | ((rw & 0x07070707u) << 2);
    hi = (((qw >> 4) & 0x07070707u) << 5) | (((rw >> 4) & 0x07070707u) << 2);
}

__device__ __forceinline__ int sa_tbl(const char* tblb, uint32_t lo, uint32_t hi, int kk) {
    const uint32_t byte = __byte_perm((kk & 1) ? hi : lo, 0, 0x4440 | (kk >> 1));
    return *reinterpret_cast<const int*>(tblb + byte);
}

// Fast form, one 8-base window.  P = packed running score, B = packed
// running best; `at` takes B at the end of each window up to and including
// the one that stops; `stop` is set by that window.  EDGE: bases at
// off0 + k >= avail score `neg`.
template <bool EDGE>
__device__ __forceinline__ void sa_window_fast(const char* tblb, uint32_t lo, uint32_t hi, uint32_t off0,
                                               uint32_t avail, int neg, uint32_t T, int& P, int& B, int& at,
                                               bool& stop) {
    int mn = INT_MAX;
    // Bases in pairs: the running best and minimum take both prefixes of a
    // pair with one 3-input max / min (DPX on sm_90 and later).
#pragma unroll
    for (int kk = 0; kk < 8; kk += 2) {
        int t0 = sa_tbl(tblb, lo, hi, kk);
        int t1 = sa_tbl(tblb, lo, hi, kk + 1);
        if (EDGE && off0 + kk >= avail) t0 = neg;
        if (EDGE && off0 + kk + 1 >= avail) t1 = neg;
        const int P0 = P + t0;
        P = P0 + t1;
        B = __vimax3_s32(B, P0, P);
        mn = __vimin3_s32(mn, P0, P);
    }
    if (!stop) at = B;
    stop = stop || (uint32_t)(B - mn) > T;
}

// Exact form, one 8-base window at step-relative indices k0..k0+7: S =
// running score, best = running maximum (from 0), pk = step-relative index
// of the last strict increase of best, alive cleared at the first base with
// best - S > xdrop or (EDGE) at off0 + k >= avail.
template <bool EDGE>
__device__ __forceinline__ void sa_window_exact(const char* tblb, uint32_t lo, uint32_t hi, int k0, uint32_t off0,
                                                uint32_t avail, int xdrop, int& S, int& best, int& pk, bool& alive) {
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
        const int sc = sa_tbl(tblb, lo, hi, kk);
        if (EDGE && off0 + kk >= avail) alive = false;
        S += sc;
        const bool up = alive && S > best;
        best = up ? S : best;
        pk = up ? k0 + kk : pk;
        alive = alive && (best - S <= xdrop);
    }
}

// ---------------------------------------------------------------------------
// Chains: hits of one diagonal that give the same HSP are scanned once.
//
// Let T be the running sum of substitution scores along a diagonal, and a hit
// at p scan right from p and left from p.  Take hits p' < p of one diagonal.
// If T(p) > T(y) for all y in [p', p) and the scan from p' does not stop before
// p, the right scan from p' has its best at or after p; from p on both scans
// see the same maxima, so they stop at the same base and end the HSP at the
// same base.  Likewise on the left if some x <= p' has T(x) < T(y) for all y in
// (x, p] and the scan from p does not stop before x.  Both hold: one HSP, one
// score, the same stops.  A hit p is therefore dropped when its nearest
// predecessor p' on the diagonal is at most `gap` bases back and the two
// conditions hold on the 32 bases before p with every match scored `match`
// (the smallest match score) and every mismatch at its lowest: such sums are
// lower bounds, so what they show positive is positive (sa_chain_joined).  At
// most `mismatches` of the 32 may differ: then no drop exceeds xdrop and no
// scan stops among them.
//
// Which hits there are is read off the two sequences: the table holds every
// window of the target, the call's seeds every window of [j_lo, j_hi)
// (checked by the lookup; else ctr->chain_bad), so a hit ends at p exactly if
// the shape's positions match in the seed_size bases before p (one transition
// allowed when the call has them).  Whether p is dropped depends on those 32
// bases and on fixed limits only (predecessors lie in p's block of
// SA_CHAIN_BLOCK query positions, which bounds a chain's length, and in the
// call's window), so the hit that starts a chain finds the dropped ones
// that follow it by the same test (sa_chain_members) and counts their tiles and
// survivors: the call's statistics stay those of every hit scanned.
//
// The sweep (below) finishes hits that stop early with a low total; such a hit
// counts no others.  As p' has p's total, and stops delta bases further right
// and delta fewer left, p sees whether the sweep finishes p': not if p itself
// has not stopped in the sweep's 32 bases right, nor if both of p's scans
// have stopped there and the total is high (else p would be finished).  In the
// remaining case, stopped right and not left, p is not dropped.  Near a
// sequence end (sa_sweep_margin) no hit is.
//
// On the genome workload 13-16% of the hits are dropped, with them a third to
// two fifths of all 32-base scan steps (they are the hits inside long HSPs);
// on repeat-rich targets half the steps, in a self-alignment nine of ten.
// ---------------------------------------------------------------------------
#define SA_CHAIN_BLOCK 1024u
#define SA_CHAIN_NEXT 0x80000000u  // unit bit: a hit follows on the diagonal within `gap` bases
#define SA_CHAIN_DROP 0x40000000u  // unit bit, inside the sweep: what it saw of the hit allows dropping it
#define SA_CHAIN_GAP 13u           // largest `gap`
#define SA_SWEEP_RIGHT 32u         // bases the sweep scores right and left of a hit
#define SA_SWEEP_LEFT 64u

// Bit 4k of v (k = 0..7) -> bit 24 + k of the result (lower bits are left over).
__device__ __forceinline__ uint32_t sa_nibble_bits(uint32_t v) {
    return ((v | (v >> 3)) & 0x03030303u) * 0x01041040u;
}

__device__ __forceinline__ uint32_t sa_join_bits(uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3) {
    return __byte_perm(__byte_perm(b0, b1, 0x0073), __byte_perm(b2, b3, 0x0073), 0x5410);
}

// Match and transition bits of 8 bases, as sa_nibble_bits gives them.
template <bool TRANS>
__device__ __forceinline__ void sa_match_bits(uint32_t rw, uint32_t qw, uint32_t& m, uint32_t& t) {
    const uint32_t d = rw ^ qw, d1 = d >> 1, d2 = d >> 2;
    m = sa_nibble_bits(~(d | d1 | d2) & 0x11111111u);
    t = TRANS ? sa_nibble_bits(d1 & ~d & ~d2 & 0x11111111u) : 0u;  // codes differ by 2: A-G, C-T
}

// Bit b = 1: a seed match starts at bit b + off of the 64-base masks
// (m0, m1: matches; t0, t1: transitions).  off + shape position <= 32.
template <bool TRANS>
__device__ __forceinline__ uint32_t sa_seed_bits(const SaExtK& a, int kmer, uint32_t m0, uint32_t m1, uint32_t t0,
                                                 uint32_t t1, uint32_t off) {
    uint32_t all = ~0u, one = 0;
    if (!TRANS) {
#pragma unroll
        for (int i = 0; i < 16; ++i) all &= __funnelshift_rc(m0, m1, off + a.shift[i]);
        return all;
    }
    for (int i = 0; i < kmer; ++i) {
        const uint32_t m = __funnelshift_rc(m0, m1, off + a.shift[i]), t = __funnelshift_rc(t0, t1, off + a.shift[i]);
        one = (one & m) | (all & t);
        all &= m;
    }
    return all | one;
}

// The two conditions on the 32 bases before p, predecessor `delta` bases back.
// mis bit k: base p - 32 + k differs.  c(o) = match * o - swing * (mismatches
// among the o bases before p) bounds T(p) - T(p - o) from below: c(o) > 0 for
// 1 <= o <= delta, and a new maximum of c at some o >= delta.
__device__ __forceinline__ bool sa_chain_joined(const SaExtK& a, uint32_t mis, uint32_t delta) {
    uint32_t r = __brev(mis);  // bit i: base p - 1 - i
    if ((uint32_t)__popc(r) > a.mismatches) return false;
    const uint32_t before = r & ((1u << (delta - 1)) - 1u), upto = r & ((1u << delta) - 1u);
    int near = max(0, a.match * (int)(delta - 1) - a.swing * __popc(before));  // max of c below delta
    const int last = max(a.match * (int)delta - a.swing * __popc(upto), a.match * 32 - a.swing * __popc(r));
    int c0 = a.match;  // c(i) = match * i + c0 - match before the k-th mismatch, c0 falling by swing each time
    for (; r; r &= r - 1) {
        const int i = __ffs(r) - 1;
        const int c = a.match * i + c0 - a.match;  // before the mismatch at o = i + 1
        if (i < (int)delta) {
            near = max(near, c);
            if (c + a.match - a.swing <= 0) return false;
        } else if (c > near) {
            return true;
        }
        c0 -= a.swing;
    }
    return last > near;
}

// Whether the sweep's windows of a hit and of those up to SA_CHAIN_GAP bases
// either way lie inside both sequences.
__device__ __forceinline__ bool sa_sweep_margin(const SaExtK& a, const SaUnit& U, uint32_t rl, uint32_t ql) {
    return min(rl, ql) >= SA_SWEEP_LEFT + SA_CHAIN_GAP && (uint64_t)rl + SA_SWEEP_RIGHT + SA_CHAIN_GAP <= a.ref_len &&
           (uint64_t)ql + SA_SWEEP_RIGHT + SA_CHAIN_GAP <= U.q_len;
}

// One hit the sweep has not finished: 0 = scan it, 1 = dropped, SA_CHAIN_NEXT =
// scan it, and a hit follows within `gap` bases.
template <bool TRANS>
__device__ __forceinline__ uint32_t sa_chain_test(const SaExtK& a, int kmer, const SaUnit& U, uint32_t rl, uint32_t ql,
                                                  bool may_drop) {
    const uint32_t S = a.seed_size, own = 32 - S, j = ql - S;
    uint32_t back = min(min(a.gap, j & (SA_CHAIN_BLOCK - 1)), min(j - U.j_lo, rl - S - 1));  // position 0 is not in the table
    uint32_t ahead = min(a.gap, U.j_hi - 1 - j);
    if (U.flags & 1u) {
        back = min(back, rl - U.rm_lo);
        ahead = min(ahead, U.rm_hi - rl);
    }
    // 48 bases from p - 32
    const uint32_t* __restrict__ pr = a.ref + (int)(rl >> 3) - 4;
    const uint32_t* __restrict__ pq = U.q_packed + (int)(ql >> 3) - 4;
    const uint32_t sr = (rl & 7u) * 4u, sq = (ql & 7u) * 4u;
    uint32_t r[7], q[7], m[6], t[6], any = 0;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        r[k] = __ldg(pr + k);
        q[k] = __ldg(pq + k);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const uint32_t rw = __funnelshift_r(r[k], r[k + 1], sr), qw = __funnelshift_r(q[k], q[k + 1], sq);
        if (k < 4) any |= rw | qw;
        sa_match_bits<TRANS>(rw, qw, m[k], t[k]);
    }
    const uint32_t m0 = sa_join_bits(m[0], m[1], m[2], m[3]), m1 = __byte_perm(m[4], m[5], 0x0073) & 0xffffu;
    const uint32_t t0 = TRANS ? sa_join_bits(t[0], t[1], t[2], t[3]) : 0u;
    const uint32_t t1 = TRANS ? __byte_perm(t[4], t[5], 0x0073) & 0xffffu : 0u;
    const uint32_t H = sa_seed_bits<TRANS>(a, kmer, m0, m1, t0, t1, 0);  // bit own: this hit
    const uint32_t prev = (H & ((1u << own) - 1u)) >> (own - back) << (own - back);
    if (may_drop && prev && !(any & 0x44444444u) && sa_chain_joined(a, ~m0, own - (31 - __clz(prev)))) return 1;
    return ((H >> own >> 1) & ((1u << ahead) - 1u)) ? SA_CHAIN_NEXT : 0u;
}

// ---------------------------------------------------------------------------
// The sweep: 32 consecutive hits per warp, one per lane, all in step.  Each is
// scored over the 32 bases right of it and the 64 left of it (the seed and as
// many again).  A hit whose scans both stop there with a total below hspthresh
// is done: it adds its tiles and leaves nothing else.  These are the chance
// hits, four of five on the genome workload.  The others gather in a buffer
// per warp; full batches of them take the chain test, and those it does not
// drop go to `list`, for the scans (sa_k_scan).
//
// Why apart from the lane kernel: a chance hit's work there was the hand-out,
// two direction set-ups and the bookkeeping of an iteration, most of it run
// for a few lanes of a warp; here it is straight-line code for all 32.  Both
// directions come from one window of the forward sequence: four aligned
// 16-byte loads of the target (a scattered load costs an L1 wavefront per
// lane, whatever its width), and query words that consecutive hits share.
//
// Bound by the L1 data pipe (83%: 96 table lookups and 128 wavefronts of target
// loads in about 250 per round), with the ALU pipe and issue at 70%.  On a 2.5 Mbp query
// against the 100 Mbp genome (60.2 M hits, both strands, one B200): every hit in
// the lane kernel 5.65 ms; sweep 2.04, scans 0.73, finish 0.51 ms, together 3.29 between events
// (with the lane kernel after the sweep 3.75, and 4.79 without chains).  The chain test on all hits as they were
// scored, with the rounds split evenly over the warps, made the sweep 2.33 ms.
// Lane phase of 24 Mbp: 55.0 -> 30.8 ms.
// ---------------------------------------------------------------------------
// What the sweep leaves of a hit, for the scans to go on from: per
// direction the best score (low half) and best - score (high half) after the
// direction's sweep, and in `rest` the offsets of the first bases reaching the
// bests (a byte each) and these flags.  A direction that has stopped leaves its
// result.
#define SA_SWEPT_SEEN 0x10000u     // else nothing is scored yet: both directions start anew
#define SA_SWEPT_STOP_R 0x20000u
#define SA_SWEPT_STOP_L 0x40000u
#define SA_SWEPT_TILE_2 0x80000u   // the left scan stopped in its second 32-base tile
#define SA_SWEPT_LONG 0x100000u    // the hit went to the long queue (set by sa_k_scan)
#define SA_SWEPT_FULL 0x200000u    // a side passed the cap and found the queue full

// One 8-base window of a scan, from its first base on (REV: from base 7
// down), in the lane kernel's packed form with SA_SWEEP_LEFT in place of STEP
// (SCALE = 2 * SA_SWEEP_LEFT): P running score, B running best, `at` B at the
// end of the windows up to and including the one that stops.
#define SA_SWEEP_SH 7  // log2(SCALE)
template <bool REV>
__device__ __forceinline__ void sa_sweep_window(const char* tblb, uint32_t rw, uint32_t qw, uint32_t T, int& P, int& B,
                                                int& at, bool& stop) {
    uint32_t lo, hi;
    sa_merge8(rw, qw, lo, hi);
    int mn = INT_MAX;
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const int P0 = P + sa_tbl(tblb, lo, hi, REV ? 7 - k : k);
        P = P0 + sa_tbl(tblb, lo, hi, REV ? 6 - k : k + 1);
        B = __vimax3_s32(B, P0, P);
        mn = __vimin3_s32(mn, P0, P);
    }
    if (!stop) at = B;
    stop = stop || (uint32_t)(B - mn) > T;
}

// Best score, best - score and best's offset of a direction after its sweep.
__device__ __forceinline__ uint32_t sa_swept_word(int P, int at) {
    const int best = at >> SA_SWEEP_SH;
    return (uint32_t)best | ((uint32_t)(best - (P >> SA_SWEEP_SH)) << 16);
}

__device__ __forceinline__ uint32_t sa_swept_pos(int at) {
    const uint32_t low = at & ((1 << SA_SWEEP_SH) - 1);
    return low == SA_SWEEP_LEFT ? 0u : SA_SWEEP_LEFT - 1 - low;
}

#define SA_SWEEP_BUF 128  // unfinished hits a warp gathers

template <bool TRANS>
__global__ void __launch_bounds__(256, 4)
sa_k_sweep(const __grid_constant__ SaExtK a, const __grid_constant__ SaParams P, uint64_t h_begin, uint64_t h_end) {
    __shared__ int tbl[64];
    __shared__ uint4 s_buf[8][SA_SWEEP_BUF], s_swept[8][SA_SWEEP_BUF];
    if (threadIdx.x < 64) tbl[threadIdx.x] = (P.sub_mat[(threadIdx.x & 7) * 8 + (threadIdx.x >> 3)] << SA_SWEEP_SH) - 1;
    __syncthreads();
    const char* tblb = reinterpret_cast<const char*>(tbl);
    sa_wait_prior();
    SaCounters* const ctr = a.ctr;
    const uint64_t H = min((uint64_t)ctr->num_hits, h_end), nnz = ctr->nnz;
    if (ctr->error || h_begin >= H) return;
    const bool chains = a.chain && !ctr->chain_bad;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = sa_lanemask_lt();
    uint4* const buf = s_buf[threadIdx.x >> 5];
    uint4* const swept = s_swept[threadIdx.x >> 5];
    uint32_t nbuf = 0, tiles = 0, ext = 0;
    const uint32_t T = (uint32_t)a.xdrop * (2 * SA_SWEEP_LEFT) + SA_SWEEP_LEFT;
    // chain test of the buffered hits, 32 at a time; those left, moved to the
    // buffer's front, go to the list
    auto write_out = [&]() {
        __syncwarp();
        uint32_t kept = nbuf;
        if (chains) {
            kept = 0;
            for (uint32_t i0 = 0; i0 < nbuf; i0 += 32) {
                const bool on = i0 + lane < nbuf;
                uint4 v = make_uint4(0, 0, 0, 0), x = v;
                uint32_t f = 1;
                if (on) {
                    v = buf[i0 + lane];
                    x = swept[i0 + lane];
                    const bool may_drop = v.w & SA_CHAIN_DROP;
                    v.w &= ~SA_CHAIN_DROP;
                    f = sa_chain_test<TRANS>(a, P.kmer_size, a.units[v.w], v.x, v.y, may_drop);
                }
                const uint32_t m = __ballot_sync(SA_FULL, f != 1);
                if (f != 1) {
                    v.w |= f;
                    buf[kept + __popc(m & lt)] = v;
                    swept[kept + __popc(m & lt)] = x;
                }
                kept += __popc(m);
                __syncwarp();
            }
        }
        nbuf = 0;
        if (!kept) return;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&ctr->list_count, (unsigned long long)kept);
        at = __shfl_sync(SA_FULL, at, 0);
        for (uint32_t i = lane; i < 2 * kept; i += 32)
            if (at + (i >> 1) < a.list_cap) a.list[2 * at + i] = (i & 1) ? swept[i >> 1] : buf[i >> 1];
        __syncwarp();
    };
    const uint64_t first = h_begin / 32, rounds = (H + 31) / 32 - first;  // h_begin is a multiple of 32
    // Runs of rounds are handed out by a counter (the warps' speeds differ with
    // their hits); a run's first seed is searched for once.  32 rounds where
    // there are enough for every warp to take eight runs.
    const uint64_t run = max((uint64_t)1, min((uint64_t)32, rounds / ((uint64_t)gridDim.x * 64)));
    while (true) {
        unsigned long long k0 = 0;
        if (lane == 0) k0 = atomicAdd(&ctr->sweep_cursor, 1ull);
        const uint64_t r0 = (uint64_t)__shfl_sync(SA_FULL, k0, 0) * run;
        if (r0 >= rounds) break;
        const uint64_t r1 = first + min(r0 + run, rounds);
        uint64_t c = sa_warp_find_seed(a.cs.E, nnz, 32 * (first + r0));
        for (uint64_t r = first + r0; r < r1; ++r) {
            const uint64_t t = 32 * r, h = t + lane;
            // the hit's seed: c, and one more for each seed that starts by then
            const uint64_t ahead = c + 1 + lane < nnz ? a.cs.E[c + 1 + lane] - t : ~0ull;
            const uint32_t starts = __reduce_or_sync(SA_FULL, ahead < 32 ? 1u << (uint32_t)ahead : 0u);
            bool left = false;
            uint4 rec = make_uint4(0, 0, 0, 0), x = rec;
            if (h < H) {
                const uint64_t k = c + __popc(starts & ((2u << lane) - 1u));
                const uint32_t rl = __ldg(a.pos_table + a.cs.lo[k] + (uint32_t)(h - a.cs.E[k])) + a.seed_size;  // find_hits :192
                const uint32_t ql = a.cs.qpos[k] + a.seed_size;                                               // find_hits :176
                const uint32_t unit = a.cs.unit[k];
                rec = make_uint4(rl, ql, a.cs.scope[k], unit);
                const SaUnit U = a.units[unit];
                // rm: hits outside [ref_start, ref_end] are never extended
                // (repeat_masker_src/seed_filter.cu:237-243, 304-333)
                bool live = !(U.flags & 1u) || (rl >= U.rm_lo && rl <= U.rm_hi);
                // Coordinates past either sequence end (a caller-supplied table or
                // seed beyond the sequences) are rejected, not read.
                if (rl > a.ref_len || ql > U.q_len) {
                    atomicCAS(&ctr->error, 0ull, 5ull);
                    live = false;
                }
                if (live) {
                    ++ext;
                    // bases [rl - 64, rl + 32) of both sequences as 12 words
                    const uint32_t* __restrict__ pq = U.q_packed + (int)(ql >> 3) - 8;
                    uint32_t rw[16], qw[13];
#pragma unroll
                    for (int i = 0; i < 13; ++i) qw[i] = __ldg(pq + i);
                    const uint4* __restrict__ pr = reinterpret_cast<const uint4*>(a.ref) + (int)(rl >> 5) - 2;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint4 v = __ldg(pr + i);
                        rw[4 * i] = v.x;
                        rw[4 * i + 1] = v.y;
                        rw[4 * i + 2] = v.z;
                        rw[4 * i + 3] = v.w;
                    }
                    if (rl & 8u) {
#pragma unroll
                        for (int i = 0; i < 15; ++i) rw[i] = rw[i + 1];
                    }
                    if (rl & 16u) {
#pragma unroll
                        for (int i = 0; i < 13; ++i) rw[i] = rw[i + 2];
                    }
                    const uint32_t sr = (rl & 7u) * 4u, sq = (ql & 7u) * 4u;
                    int p = SA_SWEEP_LEFT, B = SA_SWEEP_LEFT, at = 0;
                    bool stop_r = false, stop_l = false;
#pragma unroll
                    for (int i = 8; i < 12; ++i)
                        sa_sweep_window<false>(tblb, __funnelshift_r(rw[i], rw[i + 1], sr),
                                               __funnelshift_r(qw[i], qw[i + 1], sq), T, p, B, at, stop_r);
                    x.x = sa_swept_word(p, at);
                    x.z = sa_swept_pos(at);
                    const int best_r = at >> SA_SWEEP_SH;
                    p = B = SA_SWEEP_LEFT;
                    uint32_t tl = 0;
#pragma unroll
                    for (int i = 7; i >= 0; --i) {
                        sa_sweep_window<true>(tblb, __funnelshift_r(rw[i], rw[i + 1], sr),
                                              __funnelshift_r(qw[i], qw[i + 1], sq), T, p, B, at, stop_l);
                        if (i == 4) tl = stop_l ? 2 : 3;  // tiles of both scans, if they stop
                    }
                    x.y = sa_swept_word(p, at);
                    // where a window reaches past a sequence end, it holds scores of padding: neither scan
                    // has stopped, and both start anew (what else is passed on is not looked at)
                    const bool inside = min(rl, ql) >= SA_SWEEP_LEFT && (uint64_t)rl + SA_SWEEP_RIGHT <= a.ref_len &&
                                        (uint64_t)ql + SA_SWEEP_RIGHT <= U.q_len;
                    stop_r = stop_r && inside;
                    stop_l = stop_l && inside;
                    left = !stop_r || !stop_l || (int)(float)(best_r + (at >> SA_SWEEP_SH)) >= a.hspthresh;
                    x.z |= (sa_swept_pos(at) << 8) | (inside ? SA_SWEPT_SEEN : 0u) | (stop_r ? SA_SWEPT_STOP_R : 0u) |
                           (stop_l ? SA_SWEPT_STOP_L : 0u) | (tl == 3 ? SA_SWEPT_TILE_2 : 0u);
                    if (!left) tiles += tl;
                    if (!(stop_r && !stop_l) && sa_sweep_margin(a, U, rl, ql)) rec.w |= SA_CHAIN_DROP;
                }
            }
            if (!chains) rec.w &= ~SA_CHAIN_DROP;
            const uint32_t m = __ballot_sync(SA_FULL, left);
            if (left) {
                buf[nbuf + __popc(m & lt)] = rec;
                swept[nbuf + __popc(m & lt)] = x;
            }
            nbuf += __popc(m);
            if (nbuf > SA_SWEEP_BUF - 32) write_out();
            c += __popc(starts) + (__any_sync(SA_FULL, ahead == 32) ? 1 : 0);
        }
    }
    if (nbuf) write_out();
    unsigned long long sum = tiles, e = ext;
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        sum += __shfl_xor_sync(SA_FULL, sum, s);
        e += __shfl_xor_sync(SA_FULL, e, s);
    }
    if (lane == 0 && e) {
        atomicAdd(&ctr->base_steps, sum);
        atomicAdd(&ctr->extended, e);
    }
}

// Match, transition and non-ACGT bits of 32 bases from word pr[0] and pq[0]
// (shifted by sr, sq bits); the words after the 32 bases' first four are left in
// rl, ql, which hold those first words on entry.
__device__ __forceinline__ void sa_masks32(const uint32_t* __restrict__ pr, const uint32_t* __restrict__ pq, uint32_t sr,
                                           uint32_t sq, uint32_t& rl, uint32_t& ql, uint32_t& m, uint32_t& t,
                                           uint32_t& bad) {
    uint32_t mm[4], tt[4], bb[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t rn = __ldg(pr + k + 1), qn = __ldg(pq + k + 1);
        const uint32_t rw = __funnelshift_r(rl, rn, sr), qw = __funnelshift_r(ql, qn, sq);
        rl = rn;
        ql = qn;
        sa_match_bits<true>(rw, qw, mm[k], tt[k]);
        bb[k] = sa_nibble_bits(((rw | qw) >> 2) & 0x11111111u);
    }
    m = sa_join_bits(mm[0], mm[1], mm[2], mm[3]);
    t = sa_join_bits(tt[0], tt[1], tt[2], tt[3]);
    bad = sa_join_bits(bb[0], bb[1], bb[2], bb[3]);
}

// The dropped hits that follow the scanned hit (rl, ql) of `unit` (high: its
// total is at least hspthresh): their number and the tiles of their scans.
// stop_r, stop_l: offsets at which the hit's right and left scans stop; a hit d
// bases on stops at stop_r - d and stop_l + d.
struct SaChain {
    unsigned long long tiles;
    uint32_t n;
};

__device__ __forceinline__ SaChain sa_chain_members(const SaExtK& a, const SaParams& P, uint32_t unit, uint32_t rl,
                                                 uint32_t ql, uint32_t stop_r, uint32_t stop_l, bool high) {
    const SaUnit U = a.units[unit];
    unsigned long long tiles = 0;
    const uint32_t S = a.seed_size, j = ql - S;
    uint32_t ahead = U.j_hi - 1 - j;
    if (U.flags & 1u) ahead = min(ahead, U.rm_hi - rl);
    const uint32_t* __restrict__ pr = a.ref + (int)(rl >> 3) - 4;
    const uint32_t* __restrict__ pq = U.q_packed + (int)(ql >> 3) - 4;
    const uint32_t sr = (rl & 7u) * 4u, sq = (ql & 7u) * 4u;
    uint32_t n = 0, last = 0, m0, t0, b0, wr = __ldg(pr), wq = __ldg(pq);
    sa_masks32(pr, pq, sr, sq, wr, wq, m0, t0, b0);
    for (uint32_t c = 0; c + 1 - last <= a.gap; c += 32) {
        uint32_t m1, t1, b1;
        pr += 4;
        pq += 4;
        sa_masks32(pr, pq, sr, sq, wr, wq, m1, t1, b1);
        if ((m0 & m1) == ~0u && !(b0 | b1) && last == c && c + 32 <= ahead && stop_r >= c + 64 &&
            ((j + c) & (SA_CHAIN_BLOCK - 1)) + 32 < SA_CHAIN_BLOCK && sa_sweep_margin(a, U, rl + c + 1, ql + c + 1) &&
            sa_sweep_margin(a, U, rl + c + 32, ql + c + 32)) {
            // 64 matching bases: each of the next 32 positions ends a dropped hit.  Over
            // 32 consecutive d, (stop_r - d) >> 5 sums to stop_r - c - 32 and (stop_l + d) >> 5 to stop_l + c + 1.
            n += 32;
            tiles += (unsigned long long)(stop_r - c - 32) + (stop_l + c + 1) + 64;
            last = c + 32;
        } else {
            // bit i - 1: a match ends c + i bases on
            uint32_t hits = P.transition ? sa_seed_bits<true>(a, P.kmer_size, m0, m1, t0, t1, 33 - S)
                                         : sa_seed_bits<false>(a, P.kmer_size, m0, m1, t0, t1, 33 - S);
            for (; hits; hits &= hits - 1) {
                const uint32_t i = __ffs(hits), d = c + i, delta = d - last;
                if (d > ahead || delta > a.gap || delta > ((j + d) & (SA_CHAIN_BLOCK - 1)) ||
                    (stop_r - d < SA_SWEEP_RIGHT && (!high || stop_l + d >= SA_SWEEP_LEFT)) ||
                    !sa_sweep_margin(a, U, rl + d, ql + d) || __funnelshift_rc(b0, b1, i) || !sa_chain_joined(a, ~__funnelshift_rc(m0, m1, i), delta))
                    return {tiles, n};
                ++n;
                tiles += ((stop_r - d) >> 5) + ((stop_l + d) >> 5) + 2;
                last = d;
            }
        }
        m0 = m1;
        t0 = t1;
        b0 = b1;
    }
    return {tiles, n};
}

// sa_chain_members by a warp, 32 bases per lane: whether a hit goes on with the
// chain depends on the hit before it, at most a.gap (< 32) bases back, so a lane
// needs the last one of the lane below only; and a chain ends with its block of
// SA_CHAIN_BLOCK positions.  All lanes get the result.
__device__ __forceinline__ SaChain sa_warp_chain_members(const SaExtK& a, const SaParams& P, uint32_t unit, uint32_t rl,
                                                         uint32_t ql, uint32_t stop_r, uint32_t stop_l, bool high) {
    static_assert(SA_CHAIN_BLOCK <= 32 * 32, "a chain fits the warp");
    const SaUnit U = a.units[unit];
    const int lane = threadIdx.x & 31;
    const uint32_t S = a.seed_size, j = ql - S, c = 32 * lane;
    uint32_t ahead = U.j_hi - 1 - j;
    if (U.flags & 1u) ahead = min(ahead, U.rm_hi - rl);
    uint32_t hits = 0, m0 = 0, m1 = 0, b0 = 0, b1 = 0;  // hits bit i - 1: a match ends c + i bases on
    // a block that starts past either sequence's end holds no hit of the chain and is not read
    if (c <= ahead && c <= a.ref_len - rl) {
        const uint32_t sr = (rl & 7u) * 4u, sq = (ql & 7u) * 4u;
        const uint32_t* __restrict__ pr = a.ref + (int)(rl >> 3) - 4 + (c >> 3);
        const uint32_t* __restrict__ pq = U.q_packed + (int)(ql >> 3) - 4 + (c >> 3);
        uint32_t t0, t1, wr = __ldg(pr), wq = __ldg(pq);
        sa_masks32(pr, pq, sr, sq, wr, wq, m0, t0, b0);
        sa_masks32(pr + 4, pq + 4, sr, sq, wr, wq, m1, t1, b1);
        hits = P.transition ? sa_seed_bits<true>(a, P.kmer_size, m0, m1, t0, t1, 33 - S)
                            : sa_seed_bits<false>(a, P.kmer_size, m0, m1, t0, t1, 33 - S);
    }
    const uint32_t below = __shfl_up_sync(SA_FULL, hits, 1);
    uint32_t last = lane ? c - __clz(below) : 0, n = 0;
    unsigned long long tiles = 0;
    bool ended = (lane && !below) || !hits;
    if (!ended)
        for (uint32_t h = hits; h; h &= h - 1) {
            const uint32_t i = __ffs(h), d = c + i, delta = d - last;
            if (d > ahead || delta > a.gap || delta > ((j + d) & (SA_CHAIN_BLOCK - 1)) ||
                (stop_r - d < SA_SWEEP_RIGHT && (!high || stop_l + d >= SA_SWEEP_LEFT)) ||
                !sa_sweep_margin(a, U, rl + d, ql + d) || __funnelshift_rc(b0, b1, i) ||
                !sa_chain_joined(a, ~__funnelshift_rc(m0, m1, i), delta)) {
                ended = true;
                break;
            }
            ++n;
            tiles += ((stop_r - d) >> 5) + ((stop_l + d) >> 5) + 2;
            last = d;
        }
    const uint32_t em = __ballot_sync(SA_FULL, ended);
    if (em && lane > __ffs(em) - 1) n = tiles = 0;  // the chain ends below
    n = __reduce_add_sync(SA_FULL, n);
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) tiles += __shfl_xor_sync(SA_FULL, tiles, s);
    return {tiles, n};
}

// Where a scan of the fast form stops, to the base, from offset o where best -
// score is `depth` on.  sr, sq: the scan's first bases in R and Q; SH: log2 of the
// table's score scale.
template <int SH>
__device__ __forceinline__ uint32_t sa_stop_offset(const char* tblb, const uint32_t* __restrict__ R,
                                                const uint32_t* __restrict__ Q, uint32_t sr, uint32_t sq,
                                                uint32_t avail, int xdrop, uint32_t o, uint32_t depth) {
    int S = -(int)depth, best = 0;
    const uint32_t* __restrict__ pr = R + (sr >> 3) + (o >> 3);  // o is a multiple of 8
    const uint32_t* __restrict__ pq = Q + (sq >> 3) + (o >> 3);
    uint32_t r0 = __ldg(pr), q0 = __ldg(pq);
    while (true) {
        const uint32_t r1 = __ldg(++pr), q1 = __ldg(++pq);
        const uint32_t rw = __funnelshift_r(r0, r1, (sr & 7u) * 4u), qw = __funnelshift_r(q0, q1, (sq & 7u) * 4u);
        r0 = r1;
        q0 = q1;
        uint32_t lo, hi;
        sa_merge8(rw, qw, lo, hi);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (o + k >= avail) return avail;
            S += (sa_tbl(tblb, lo, hi, k) + 1) >> SH;
            best = max(best, S);
            if (best - S > xdrop) return o + k;
        }
        o += 8;
    }
}

// Keep test of one candidate HSP per lane (total >= hspthresh): entropy factor
// from the per-base match counts over the HSP when the total is in the entropy
// range (src/seed_filter.cu:580-621), then insertion of the kept ones into the
// call's set of distinct HSPs (rm: query start flipped on the reverse strand,
// repeat_masker_src/seed_filter.cu:704-707).  r: {ref_start, query_start (before
// the rm flip), len, scope}; the candidate counts as `hits` survivors.  Called
// by the whole warp.  LOOKUP: look it up in the set first (sa_set_query: the
// query start of its key).
__device__ __forceinline__ uint32_t sa_set_query(const SaExtK& a, uint32_t flags, const uint4& r) {
    return (flags & 2u) ? a.ref_len - 1 - (r.y + r.z) : r.y;
}

template <bool LOOKUP>
__device__ __forceinline__ void sa_keep_candidates(const SaExtK& a, bool on, uint4 r, int total, uint32_t unit,
                                                   uint32_t hits) {
    const int lane = threadIdx.x & 31;
    int keep = 0, score = 0;
    bool known = false;
    uint32_t qs = 0;
    if (on) {
        const SaUnit U = a.units[unit];
        const int ext = (int)r.z;
        qs = sa_set_query(a, U.flags, r);
        // A candidate whose key the set already holds was kept with this same
        // key (the scope fixes the unit, so the same bases): it is a survivor,
        // and its match counts, logs and insertion are skipped.
        known = LOOKUP && sa_hash_contains(a.hset, a.ctr->hash_mask, r.w, r.x, qs, r.z);
        if (known) {
            keep = 1;
        } else {
            int cnt[4] = {0, 0, 0, 0};
            const bool eb = sa_entropy_branch(a, total);
            if (eb) sa_count_matches_span(a.ref, r.x, U.q_packed, r.y, (int64_t)ext + 1, cnt);
            sa_keep_score(total, ext, cnt, eb, a.hspthresh, &keep, &score);
        }
    }
    const uint32_t kept = __reduce_add_sync(SA_FULL, keep ? hits : 0u);
    if (lane == 0 && kept) atomicAdd(&a.ctr->surv_count, (unsigned long long)kept);
    unsigned long long claimed = ~0ull;
    if (keep && !known)
        claimed = sa_hash_insert(a.hset, a.ctr->hash_mask, r.w, r.x, qs, r.z, score, &a.ctr->hash_overflow);
    sa_hash_note_used(a.hset, &a.ctr->hash_used, claimed);
}

// Keep test of `n` (<= 32) ring candidates from slot `head` on, one per lane, by
// the whole warp; leaves the slots free for reuse.
__device__ __forceinline__ void sa_flush_candidates(const SaExtK& a, const uint4* s_em, const uint2* s_ex,
                                                    uint32_t head, uint32_t n) {
    const int lane = threadIdx.x & 31;
    const bool on = (uint32_t)lane < n;
    uint4 r = make_uint4(0, 0, 0, 0);
    uint2 x = make_uint2(0, 0);
    if (on) {
        const uint32_t slot = (head + lane) & 63u;
        r = s_em[slot];
        x = s_ex[slot];
    }
    __syncwarp();  // slots are rewritten by later appends
    sa_keep_candidates<true>(a, on, r, (int)x.x, x.y, 1);
}

// Dynamic shared memory of the lane kernel for `tile` hits per warp tile.
static size_t sa_lane_smem(uint32_t tile) {
    return SA_LANE_TABLES + 8 * (size_t)tile * 16 + 8 * (size_t)(tile + 1) * 8 + 8 * 64 * 16 + 8 * 64 * 8;
}

template <int MIN_CTAS, int STEP, bool EXACT>
__global__ void __launch_bounds__(256, MIN_CTAS)
sa_k_extend_lane(const __grid_constant__ SaExtK a, const __grid_constant__ SaParams P) {
    constexpr int NW = STEP / 8;                  // 8-base windows per step
    constexpr int SCALE = 2 * STEP;               // packed score scale (fast form)
    constexpr int SH = STEP == 8 ? 4 : STEP == 16 ? 5 : 6;  // log2(SCALE)
    static_assert(STEP == 8 || STEP == 16 || STEP == 32, "8-, 16- or 32-base steps");
    // Read-ahead: the last step reads up to 2 * NW + 1 words past the last base.
    static_assert(2 * NW + 2 <= SA_PADW, "padding shorter than the read-ahead");
    // Shared memory: score table (64 ints), then per warp: tile records,
    // tile E window, and a 64-entry ring of candidate HSPs awaiting the keep
    // test and insertion.
    extern __shared__ __align__(16) unsigned char sa_smem[];
    const uint32_t TILE = a.tile_hits;
    // entry (q << 3) | r: target code r vs query code q.  Codes 0..3 use
    // entries 0..27 only, one per bank: lookups of A/C/G/T pairs never conflict.
    int* tbl = reinterpret_cast<int*>(sa_smem);
    if (threadIdx.x < 64) {
        const int sc = P.sub_mat[(threadIdx.x & 7) * 8 + (threadIdx.x >> 3)];
        tbl[threadIdx.x] = EXACT ? sc : sc * SCALE - 1;
    }
    __syncthreads();
    const char* tblb = reinterpret_cast<const char*>(tbl);
    if (a.ctr->error) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t lt = sa_lanemask_lt();
    uint4* const s_hits = reinterpret_cast<uint4*>(sa_smem + SA_LANE_TABLES) + wid * TILE;
    unsigned long long* const s_E =
        reinterpret_cast<unsigned long long*>(sa_smem + SA_LANE_TABLES + 128 * (size_t)TILE) + wid * (TILE + 1);
    unsigned char* const em_base = sa_smem + SA_LANE_TABLES + 128 * (size_t)TILE + 64 * (size_t)(TILE + 1);
    uint4* const s_em = reinterpret_cast<uint4*>(em_base) + wid * 64;
    uint2* const s_ex = reinterpret_cast<uint2*>(em_base + 8 * 64 * 16) + wid * 64;

    // H, nnz, ref_len, seed_size and xdrop are read where used (registers
    // are the lane kernel's limit)
    const uint32_t* __restrict__ ref = a.ref;

    uint32_t tile_pos = 0, tile_n = 0;
    bool exhausted = false;
    uint32_t em_head = 0, em_tail = 0;  // ring of kept HSPs (warp-uniform cursors)

    // current hit
    bool has = false, nocap = false, setup = false;
    uint32_t rl = 0, ql = 0, scope = 0, unit_id = 0;
    int dir = 0;
    // scan of the current direction: offset, bases available, word shifts,
    // words w[0..NW] of the coming step, next word addresses
    uint32_t o = 0, avail = 0, sh_r = 0, sh_q = 0;
    uint32_t w_r[NW + 1], w_q[NW + 1];
#pragma unroll
    for (int j = 0; j <= NW; ++j) w_r[j] = w_q[j] = 0;
    const uint32_t* __restrict__ pr = ref;
    const uint32_t* __restrict__ pq = ref;
    // running score, best, offset of the first base reaching best
    int S = 0, best = 0, bpos = 0, Rbest = 0, Rpos = -1;
    uint32_t tiles = 0, tiles_acc = 0, ext_acc = 0;  // per-lane statistics (32-bit per lane)

    // Start of a direction of the current hit (dir 0: right of the hit; 1:
    // left, read rightwards in the reversed copies): offsets, bases
    // available, word shifts and the first NW + 1 words of both sequences.
    auto begin_dir = [&](const uint32_t* __restrict__ qp, uint32_t qlen) {
        const uint32_t ref_len = a.ref_len;
        const uint32_t sr = dir ? ref_len - rl : rl, sq = dir ? qlen - ql : ql;
        avail = min(ref_len - sr, qlen - sq);
        sh_r = (sr & 7u) * 4u;
        sh_q = (sq & 7u) * 4u;
        pr = (dir ? ref + sa_rev_words(ref_len) : ref) + (sr >> 3);
        pq = (dir ? qp + sa_rev_words(qlen) : qp) + (sq >> 3);
#pragma unroll
        for (int j = 0; j <= NW; ++j) {
            w_r[j] = __ldg(pr + j);
            w_q[j] = __ldg(pq + j);
        }
        pr += NW + 1;
        pq += NW + 1;
        o = 0;
        S = 0;
        best = 0;
        bpos = 0;
    };

    while (true) {
        // ---- idle lanes take the next hits of the warp tile, in order ----
        const uint32_t idle = __ballot_sync(SA_FULL, !has);
        bool fresh = false;
        if (idle && !(exhausted && tile_pos >= tile_n)) {
            if (tile_pos >= tile_n) {
                // Take the next tile of hits and expand it: the hits of the
                // tile span at most TILE consecutive hit-bearing seeds from the
                // one holding its first hit, so E over that window locates each
                // hit's seed by binary search.
                unsigned long long t0 = 0;
                if (lane == 0) t0 = atomicAdd(&a.ctr->hit_cursor, (unsigned long long)TILE);
                t0 = __shfl_sync(SA_FULL, t0, 0);
                const uint64_t H = a.ctr->num_hits, nnz = a.ctr->nnz;
                if (t0 >= H) {
                    exhausted = true;
                    tile_n = tile_pos = 0;
                } else {
                    uint32_t n = (uint32_t)min((unsigned long long)TILE, H - t0);
                    const uint64_t c0 = sa_warp_find_seed(a.cs.E, nnz, t0);
                    const uint32_t nw = (uint32_t)min((uint64_t)n, nnz - c0);  // seeds of the window
                    for (uint32_t i = lane; i <= nw; i += 32) s_E[i] = a.cs.E[c0 + i];  // E[nnz] == H
                    __syncwarp();
                    // record of hit t0 + i: its seed by binary search in the E window
                    auto record = [&](uint32_t i) {
                        const unsigned long long h = t0 + i;
                        uint32_t lo = 0, hi = nw;  // last k in [0, nw) with E[c0+k] <= h
                        while (hi - lo > 1) {
                            const uint32_t mid = (lo + hi) >> 1;
                            if (s_E[mid] <= h) lo = mid;
                            else hi = mid;
                        }
                        const uint64_t c = c0 + lo;
                        uint4 r;
                        r.x = __ldg(a.pos_table + a.cs.lo[c] + (uint32_t)(h - s_E[lo])) + a.seed_size;  // find_hits :192
                        r.y = a.cs.qpos[c] + a.seed_size;                                                 // find_hits :176
                        r.z = a.cs.scope[c];
                        r.w = a.cs.unit[c];
                        return r;
                    };
                    if (!a.windowed) {
                        for (uint32_t i = lane; i < n; i += 32) s_hits[i] = record(i);
                    } else {
                        // rm: hits outside [ref_start, ref_end] are never extended
                        // (repeat_masker_src/seed_filter.cu:237-243, 304-333); the
                        // tile keeps only the others, in order, so that no lane is
                        // handed a hit it would skip.  Coordinates past either
                        // sequence end are rejected here too.
                        uint32_t kept = 0;
                        for (uint32_t i0 = 0; i0 < n; i0 += 32) {
                            bool live = false;
                            uint4 r = make_uint4(0, 0, 0, 0);
                            if (i0 + lane < n) {
                                r = record(i0 + lane);
                                const SaUnit U = a.units[r.w];
                                live = !(U.flags & 1u) || (r.x >= U.rm_lo && r.x <= U.rm_hi);
                                if (!live && (r.x > a.ref_len || r.y > U.q_len)) atomicCAS(&a.ctr->error, 0ull, 5ull);
                            }
                            const uint32_t m = __ballot_sync(SA_FULL, live);
                            if (live) s_hits[kept + __popc(m & lt)] = r;
                            kept += __popc(m);
                        }
                        n = kept;
                    }
                    __syncwarp();
                    tile_n = n;
                    tile_pos = 0;
                }
            }
            if (tile_pos < tile_n) {
                const uint32_t m = min((uint32_t)__popc(idle), tile_n - tile_pos);
                const uint32_t rank = __popc(idle & lt);
                if (!has && rank < m) {
                    const uint4 r = s_hits[tile_pos + rank];
                    rl = r.x;
                    ql = r.y;
                    scope = r.z;
                    unit_id = r.w;
                    fresh = true;
                }
                tile_pos += m;
            }
        }

        // ---- start of a direction: a fresh hit (right), or the left side of
        // the current hit after its right end ----
        if (fresh || setup) {
            const SaUnit U = a.units[unit_id];
            if (fresh) {
                // rm: hits outside [ref_start, ref_end] are never extended
                // (repeat_masker_src/seed_filter.cu:237-243, 304-333).
                bool skip = (U.flags & 1u) && !(rl >= U.rm_lo && rl <= U.rm_hi);
                // Coordinates past either sequence end (a caller-supplied table or
                // seed beyond the sequences) are rejected, not read.
                if (rl > a.ref_len || ql > U.q_len) {
                    atomicCAS(&a.ctr->error, 0ull, 5ull);
                    skip = true;
                }
                if (!skip) {
                    has = true;
                    nocap = false;
                    setup = true;
                    dir = 0;
                    tiles = 0;
                    ++ext_acc;
                }
            }
            if (setup) {
                setup = false;
                begin_dir(U.q_packed, U.q_len);
            }
        }
        const bool done = !__any_sync(SA_FULL, has) && exhausted && tile_pos >= tile_n;

        // ---- up to `substeps` STEP-base steps per busy lane: the lanes still
        // scanning go on while any lane of the warp does; a lane stops for
        // this iteration when its direction ends or it goes to the long queue ----
        bool finished = false, to_long = false;
        int Lpos = 0, total = 0;
        bool scanning = has;
#pragma unroll 1
        for (uint32_t sub = 0; sub < a.substeps; ++sub) {
            if (!__any_sync(SA_FULL, scanning)) break;
            if (scanning) {
                uint32_t rwin[NW], qwin[NW];
    #pragma unroll
                for (int j = 0; j < NW; ++j) {
                    rwin[j] = __funnelshift_r(w_r[j], w_r[j + 1], sh_r);
                    qwin[j] = __funnelshift_r(w_q[j], w_q[j + 1], sh_q);
                }
                w_r[0] = w_r[NW];
                w_q[0] = w_q[NW];
    #pragma unroll
                for (int j = 1; j <= NW; ++j) {
                    w_r[j] = __ldg(pr + j - 1);
                    w_q[j] = __ldg(pq + j - 1);
                }
                pr += NW;
                pq += NW;
                const bool edge = o + STEP > avail;
                bool stop = false;
                uint32_t lo, hi;
                if (EXACT) {
                    bool alive = true;
                    int pk = 0;
                    const int best_in = best;
                    if (!edge) {
    #pragma unroll
                        for (int j = 0; j < NW; ++j) {
                            sa_merge8(rwin[j], qwin[j], lo, hi);
                            sa_window_exact<false>(tblb, lo, hi, 8 * j, o + 8 * j, avail, a.xdrop, S, best, pk, alive);
                        }
                    } else {
    #pragma unroll
                        for (int j = 0; j < NW; ++j) {
                            sa_merge8(rwin[j], qwin[j], lo, hi);
                            sa_window_exact<true>(tblb, lo, hi, 8 * j, o + 8 * j, avail, a.xdrop, S, best, pk, alive);
                        }
                    }
                    if (best != best_in) bpos = (int)o + pk;
                    stop = !alive;
                } else {
                    // B - min > SCALE * xdrop + STEP  <=>  (B >> SH) - (min >> SH) > xdrop, because
                    // the low parts of B (0..STEP) and min (0..STEP-1) differ by less than SCALE
                    const uint32_t T = (uint32_t)a.xdrop * SCALE + STEP;
                    int Pk = ((S - best) << SH) + STEP, B = STEP, at = 0;
                    if (!edge) {
    #pragma unroll
                        for (int j = 0; j < NW; ++j) {
                            sa_merge8(rwin[j], qwin[j], lo, hi);
                            sa_window_fast<false>(tblb, lo, hi, o + 8 * j, avail, 0, T, Pk, B, at, stop);
                        }
                    } else {
    #pragma unroll
                        for (int j = 0; j < NW; ++j) {
                            sa_merge8(rwin[j], qwin[j], lo, hi);
                            // a base past the sequence end scores -(xdrop + 1)
                            sa_window_fast<true>(tblb, lo, hi, o + 8 * j, avail, -(a.xdrop + 1) * SCALE - 1, T, Pk,
                                                 B, at, stop);
                        }
                    }
                    const int low = at & (SCALE - 1);
                    if (low != STEP) bpos = (int)o + (STEP - 1 - low);
                    const int best_in = best;
                    best = best_in + (at >> SH);
                    S = best_in + (Pk >> SH);  // exact after a full step without a stop
                }
                if (stop) {
                    // Steps start at multiples of STEP (8, 16 or 32), so the stop offset
                    // lies in 32-base tile o >> 5 whichever base of the step it is.
                    tiles += (o >> 5) + 1;
                    if (dir == 0) {
                        Rbest = best;
                        Rpos = best > 0 ? bpos : -1;  // -1 when no positive score
                        dir = 1;
                        setup = true;
                    } else {
                        finished = true;
                    }
                    scanning = false;
                } else {
                    o += STEP;
                    if (o >= a.lane_cap && !nocap) {
                        to_long = true;
                        scanning = false;
                    }
                }
                if (finished) {
                    Lpos = best > 0 ? bpos + 1 : 0;  // left offsets are 1-based
                    total = Rbest + best;
                    tiles_acc += tiles;
                    has = false;
                }
            }
            // switch_now: a lane whose right side ended in this step starts
            // its left side at once and scans in the iteration's remaining
            // steps instead of idling until the next iteration
            if (a.switch_now && sub + 1 < a.substeps && __any_sync(SA_FULL, setup)) {
                if (setup) {
                    setup = false;
                    const SaUnit U = a.units[unit_id];
                    begin_dir(U.q_packed, U.q_len);
                    scanning = true;
                }
            }
        }

        // ---- long queue pushes (warp-aggregated) ----
        {
            const uint32_t lm = __ballot_sync(SA_FULL, to_long);
            if (lm) {
                const int leader = __ffs(lm) - 1;
                unsigned long long base = 0;
                if (lane == leader) base = atomicAdd(&a.ctr->long_count, (unsigned long long)__popc(lm));
                base = __shfl_sync(SA_FULL, base, leader);
                if (to_long) {
                    const unsigned long long idx = base + __popc(lm & lt);
                    if (idx < a.long_cap) {
                        SaLongHit e;
                        e.ref_loc = rl;
                        e.query_loc = ql;
                        e.unit = unit_id;
                        e.scope = scope;
                        a.long_q[idx] = e;
                        has = false;
                    } else {
                        nocap = true;  // queue full: finish this hit in the lane
                        atomicAdd(&a.ctr->long_overflow, 1ull);
                    }
                }
            }
        }
        // ---- candidate HSPs (total >= hspthresh; the entropy factor is at
        // most 1, so lower totals are never kept) into the warp's ring ----
        {
            const bool emit = finished && (int)(float)total >= a.hspthresh;
            const uint32_t em = __ballot_sync(SA_FULL, emit);
            if (emit) {
                const uint32_t slot = (em_tail + __popc(em & lt)) & 63u;
                // {ref_start, query_start (before the rm flip), len, scope}, {total, unit} (:606-608)
                s_em[slot] = make_uint4(rl - (uint32_t)Lpos, ql - (uint32_t)Lpos, (uint32_t)(Rpos + Lpos), scope);
                s_ex[slot] = make_uint2((uint32_t)total, unit_id);
            }
            em_tail += __popc(em);
            // full batches of 32; at the end, whatever is left
            while (em_tail - em_head >= 32 || (done && em_tail != em_head)) {
                const uint32_t n = min(em_tail - em_head, 32u);
                __syncwarp();
                sa_flush_candidates(a, s_em, s_ex, em_head, n);
                em_head += n;
            }
        }
        if (done) break;
    }
    // flush statistics
    unsigned long long t = tiles_acc, e = ext_acc;
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        t += __shfl_xor_sync(SA_FULL, t, s);
        e += __shfl_xor_sync(SA_FULL, e, s);
    }
    if (lane == 0) {
        atomicAdd(&a.ctr->base_steps, t);
        atomicAdd(&a.ctr->extended, e);
    }
}

// ---------------------------------------------------------------------------
// The scans of listed hits, from where the sweep left off; left sides are read
// rightwards in the reversed copies.  A warp takes a batch of records and one of
// their sides; a lane scans one hit's side, STEP bases per step in the fast form,
// writes the result for sa_k_finish and takes the next of the batch.
//
// Bound by instruction issue.  With one side and no keep test a lane's state fits
// 64 registers (4 CTAs per SM), and a hand-out is the only thing between steps:
// the lane kernel, which took both sides and the keep test, spent half of its
// instructions around the steps.  Scans, chains and keep tests of 2.5 Mbp at
// 1-in-500 differences, us: lane kernel and a kernel for the chains 1674, now
// 1450 (scans 807); of a call of 250,000 positions 203 -> 175.  A launch per side left two tails (248 -> 353 us
// where scans are long).  Batches shrink on short lists so that all warps have some.
// ---------------------------------------------------------------------------
#define SA_SCAN_BATCH 64
#define SA_LONG_NONE 0xffffffffu  // unit of a queue entry for a hit that is in the queue already

// A list this short leaves most lanes without a hit, and a long scan's lane
// steps are the call's critical path: hits past SA_FEW_CAP bases go to the warp
// kernel, whose warps would idle too (lane + warp kernel at caps of 8192 and 128,
// ms: 11 long hits 0.083 and 0.049, 785 0.152 and 0.082, 12 K 0.455 and 0.209).
// A call with more keeps the tuning's cap: a warp per hit of a few hundred bases
// costs more than a lane (120 K long hits: 0.35 and 0.74 ms).
#define SA_FEW_HITS 32768u
#define SA_FEW_CAP 128u

template <int STEP>
__global__ void __launch_bounds__(256, 4)
sa_k_scan(const __grid_constant__ SaExtK a, const __grid_constant__ SaParams P) {
    constexpr int NW = STEP / 8, SCALE = 2 * STEP, SH = STEP == 8 ? 4 : STEP == 16 ? 5 : 6;
    __shared__ int tbl[64];
    __shared__ uint4 s_hit[8][SA_SCAN_BATCH];   // {rl, ql, unit, swept word}
    __shared__ uint2 s_rest[8][SA_SCAN_BATCH];  // {swept rest, list index}
    if (threadIdx.x < 64) tbl[threadIdx.x] = P.sub_mat[(threadIdx.x & 7) * 8 + (threadIdx.x >> 3)] * SCALE - 1;
    __syncthreads();
    const char* tblb = reinterpret_cast<const char*>(tbl);
    sa_wait_prior();
    SaCounters* const ctr = a.ctr;
    const unsigned long long n_list = ctr->list_count;
    if (ctr->error || n_list > a.list_cap) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t lt = sa_lanemask_lt();
    const uint32_t lane_cap = n_list <= SA_FEW_HITS ? min(a.lane_cap, SA_FEW_CAP) : a.lane_cap;
    const unsigned long long warps = gridDim.x * 8ull;
    const uint32_t q = (uint32_t)min((unsigned long long)SA_SCAN_BATCH, max(8ull, (2 * n_list + warps - 1) / warps));
    uint32_t batch_pos = 0, batch_n = 0;
    bool exhausted = false;
    // the lane's scan: place in `scanned`, offset, bases available, word shifts, words of the coming step, next addresses
    bool has = false, nocap = false;
    uint32_t idx = 0, o = 0, avail = 0, sh_r = 0, sh_q = 0, w_r[NW + 1], w_q[NW + 1];
#pragma unroll
    for (int j = 0; j <= NW; ++j) w_r[j] = w_q[j] = 0;
    const uint32_t* __restrict__ pr = a.ref;
    const uint32_t* __restrict__ pq = a.ref;
    int S = 0, best = 0, bpos = -1;
    while (true) {
        const uint32_t idle = __ballot_sync(SA_FULL, !has);
        if (idle) {
            while (batch_pos >= batch_n && !exhausted) {
                // the next q list records' hits that need this side
                unsigned long long t0 = 0;
                if (lane == 0) t0 = atomicAdd(&ctr->scan_cursor, 1ull);
                t0 = __shfl_sync(SA_FULL, t0, 0);
                const uint32_t side = t0 & 1u;
                t0 = (t0 >> 1) * q;
                batch_pos = batch_n = 0;
                if (t0 >= n_list) {
                    exhausted = true;
                    break;
                }
#pragma unroll
                for (int k = 0; k < SA_SCAN_BATCH / 32; ++k) {
                    const unsigned long long i = t0 + 32 * k + lane;
                    uint4 h = make_uint4(0, 0, 0, 0), x = h;
                    bool need = false;
                    if (32 * k + lane < q && i < n_list) {
                        h = a.list[2 * i];
                        x = a.list[2 * i + 1];
                        need = !(x.z & (side ? SA_SWEPT_STOP_L | SA_SWEPT_LONG : SA_SWEPT_STOP_R | SA_SWEPT_LONG));
                    }
                    const uint32_t m = __ballot_sync(SA_FULL, need);
                    if (need) {
                        const uint32_t at = batch_n + __popc(m & lt);
                        s_hit[wid][at] = make_uint4(h.x, h.y, h.w & ~SA_CHAIN_NEXT, side ? x.y : x.x);
                        s_rest[wid][at] = make_uint2(x.z, 2 * (uint32_t)i + side);
                    }
                    batch_n += __popc(m);
                }
                __syncwarp();
            }
            const uint32_t m = min((uint32_t)__popc(idle), batch_n - batch_pos), rank = __popc(idle & lt);
            if (!has && rank < m) {
                const uint4 h = s_hit[wid][batch_pos + rank];
                const uint2 x = s_rest[wid][batch_pos + rank];
                const SaUnit U = a.units[h.z];
                const uint32_t ref_len = a.ref_len;
                const bool seen = x.x & SA_SWEPT_SEEN;
                idx = x.y;
                const uint32_t side = x.y & 1u;
                const uint32_t sr = side ? ref_len - h.x : h.x, sq = side ? U.q_len - h.y : h.y;
                o = seen ? (side ? SA_SWEEP_LEFT : SA_SWEEP_RIGHT) : 0u;
                best = seen ? (int)(h.w & 0xffffu) : 0;
                S = seen ? best - (int)(h.w >> 16) : 0;
                bpos = best ? (int)((x.x >> (side ? 8 : 0)) & 0xffu) : -1;
                avail = min(ref_len - sr, U.q_len - sq);
                sh_r = (sr & 7u) * 4u;
                sh_q = (sq & 7u) * 4u;
                pr = (side ? a.ref + sa_rev_words(ref_len) : a.ref) + (sr >> 3) + (o >> 3);
                pq = (side ? U.q_packed + sa_rev_words(U.q_len) : U.q_packed) + (sq >> 3) + (o >> 3);
#pragma unroll
                for (int j = 0; j <= NW; ++j) {
                    w_r[j] = __ldg(pr + j);
                    w_q[j] = __ldg(pq + j);
                }
                pr += NW + 1;
                pq += NW + 1;
                has = true;
                nocap = false;
            }
            batch_pos += m;
        }
        if (!__any_sync(SA_FULL, has)) break;
        bool to_long = false;
#pragma unroll 1
        for (uint32_t sub = 0; sub < a.substeps; ++sub) {
            if (has && !to_long) {
                uint32_t rwin[NW], qwin[NW];
#pragma unroll
                for (int j = 0; j < NW; ++j) {
                    rwin[j] = __funnelshift_r(w_r[j], w_r[j + 1], sh_r);
                    qwin[j] = __funnelshift_r(w_q[j], w_q[j + 1], sh_q);
                }
                w_r[0] = w_r[NW];
                w_q[0] = w_q[NW];
#pragma unroll
                for (int j = 1; j <= NW; ++j) {
                    w_r[j] = __ldg(pr + j - 1);
                    w_q[j] = __ldg(pq + j - 1);
                }
                pr += NW;
                pq += NW;
                // the lane kernel's fast form
                const uint32_t T = (uint32_t)a.xdrop * SCALE + STEP;
                const int depth = best - S;
                int Pk = STEP - (depth << SH), B = STEP, at = 0;
                bool stop = false;
                uint32_t lo, hi;
                if (o + STEP <= avail) {
#pragma unroll
                    for (int j = 0; j < NW; ++j) {
                        sa_merge8(rwin[j], qwin[j], lo, hi);
                        sa_window_fast<false>(tblb, lo, hi, o + 8 * j, avail, 0, T, Pk, B, at, stop);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < NW; ++j) {
                        sa_merge8(rwin[j], qwin[j], lo, hi);
                        sa_window_fast<true>(tblb, lo, hi, o + 8 * j, avail, -(a.xdrop + 1) * SCALE - 1, T, Pk, B, at,
                                             stop);
                    }
                }
                const int low = at & (SCALE - 1);
                if (low != STEP) bpos = (int)o + (STEP - 1 - low);
                S = best + (Pk >> SH);  // exact after a full step without a stop
                best += at >> SH;
                if (stop) {
                    a.scanned[idx] = make_uint4((uint32_t)best, (uint32_t)bpos, o, (uint32_t)depth);
                    has = false;
                } else {
                    o += STEP;
                    to_long = o >= lane_cap && !nocap;
                }
            }
            if (sub + 1 < a.substeps && !__any_sync(SA_FULL, has && !to_long)) break;
        }
        const uint32_t lm = __ballot_sync(SA_FULL, to_long);
        if (lm) {
            unsigned long long base = 0;
            const int leader = __ffs(lm) - 1;
            if (lane == leader) base = atomicAdd(&ctr->long_count, (unsigned long long)__popc(lm));
            base = __shfl_sync(SA_FULL, base, leader) + __popc(lm & lt);
            bool again = false;
            if (to_long) {
                uint4* const rec = a.list + (idx & ~1u);
                const uint32_t was = atomicOr(&rec[1].z, base < a.long_cap ? SA_SWEPT_LONG : SA_SWEPT_FULL);
                again = was & (SA_SWEPT_LONG | SA_SWEPT_FULL);
                if (base < a.long_cap) {
                    const uint4 h = rec[0];
                    SaLongHit e;
                    e.ref_loc = h.x;
                    e.query_loc = h.y;
                    e.unit = was & SA_SWEPT_LONG ? SA_LONG_NONE : h.w;  // once per hit
                    e.scope = h.z;
                    a.long_q[base] = e;
                    has = false;
                } else {
                    nocap = true;  // queue full: finish this side in the lane
                    atomicAdd(&ctr->long_overflow, 1ull);
                }
            }
            const uint32_t am = __ballot_sync(SA_FULL, again);
            if (lane == 0 && am) atomicAdd(&ctr->long_again, (unsigned long long)__popc(am));
        }
    }
}

// Listed hit i as the sweep and the scans left it.  All loads are issued at once
// (`scanned` is stale for a side that the sweep finished, or never written).
struct SaListed {
    uint4 h, x, r, l;
};

__device__ __forceinline__ SaListed sa_listed(const SaExtK& a, unsigned long long i) {
    return {a.list[2 * i], a.list[2 * i + 1], a.scanned[2 * i], a.scanned[2 * i + 1]};
}

// Its sides in e.r and e.l, also where the sweep stopped (told from offset 0 on), and their tiles.
__device__ __forceinline__ uint32_t sa_listed_sides(SaListed& e) {
    if (e.x.z & SA_SWEPT_STOP_R) e.r = make_uint4(e.x.x & 0xffffu, e.x.x & 0xffffu ? e.x.z & 0xffu : ~0u, 0, 0);
    uint32_t tiles = (e.r.z >> 5) + 2;
    if (e.x.z & SA_SWEPT_STOP_L) {
        e.l = make_uint4(e.x.y & 0xffffu, e.x.y & 0xffffu ? (e.x.z >> 8) & 0xffu : ~0u, 0, 0);
        return tiles + ((e.x.z & SA_SWEPT_TILE_2) ? 1 : 0);
    }
    return tiles + (e.l.z >> 5);
}

// Listed hits to HSPs: tiles; for a hit that others may follow the dropped ones
// after it (sa_chain_members), which survive if its HSP is kept; and the keep
// test.  A warp sorts its records into those that start chains and candidates,
// and takes either 32 at a time: with a record per lane throughout the kernel
// took 1.27 ms where this takes 0.51 (60.2 M hits).  Candidates that the set holds already (most)
// end with that look-up; the others gather again, because a few lanes of nearly every batch
// counting matches cost 0.07 ms.  The chains are 0.2 ms.
#define SA_FINISH_RING 128
__global__ void __launch_bounds__(256, 4)
sa_k_finish(const __grid_constant__ SaExtK a, const __grid_constant__ SaParams P) {
    constexpr int SH = 4;  // log2 of the score scale of sa_stop_offset's table
    __shared__ int tbl[64];
    __shared__ uint32_t s_lead[8][SA_FINISH_RING];
    __shared__ uint2 s_cand[8][SA_FINISH_RING];  // {list index, survivors it stands for}
    __shared__ uint4 s_seg[8][64], s_new[8][64];  // candidates that the set does not hold: segment, {total, unit, survivors}
    if (threadIdx.x < 64) tbl[threadIdx.x] = (P.sub_mat[(threadIdx.x & 7) * 8 + (threadIdx.x >> 3)] << SH) - 1;
    __syncthreads();
    const char* tblb = reinterpret_cast<const char*>(tbl);
    sa_wait_prior();
    SaCounters* const ctr = a.ctr;
    const unsigned long long n = ctr->list_count;
    if (ctr->error || n > a.list_cap) return;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = sa_lanemask_lt();
    uint32_t* const lead = s_lead[threadIdx.x >> 5];
    uint2* const cand = s_cand[threadIdx.x >> 5];
    uint4* const fresh_seg = s_seg[threadIdx.x >> 5];
    uint4* const fresh = s_new[threadIdx.x >> 5];
    uint32_t l0 = 0, l1 = 0, c0 = 0, c1 = 0, f0 = 0, f1 = 0;  // ring cursors
    unsigned long long tiles = 0, known = 0;
    for (unsigned long long i0 = (blockIdx.x * 8ull + (threadIdx.x >> 5)) * 32;; i0 += gridDim.x * 256ull) {
        const bool done = i0 >= n;
        const unsigned long long i = i0 + lane;
        bool leads = false, high = false;
        if (i < n) {
            SaListed e = sa_listed(a, i);
            if (!(e.x.z & SA_SWEPT_LONG)) {
                tiles += sa_listed_sides(e);
                leads = e.h.w & SA_CHAIN_NEXT;
                high = !leads && (int)(float)((int)e.r.x + (int)e.l.x) >= a.hspthresh;
            }
        }
        const uint32_t lm = __ballot_sync(SA_FULL, leads), cm = __ballot_sync(SA_FULL, high);
        if (leads) lead[(l1 + __popc(lm & lt)) % SA_FINISH_RING] = (uint32_t)i;
        if (high) cand[(c1 + __popc(cm & lt)) % SA_FINISH_RING] = make_uint2((uint32_t)i, 1);
        l1 += __popc(lm);
        c1 += __popc(cm);
        __syncwarp();
        while (l1 - l0 >= 32 || (done && l1 != l0)) {
            const bool on = lane < (int)(l1 - l0);
            uint32_t k = 0, hits = 1;
            high = false;
            if (on) {
                k = lead[(l0 + lane) % SA_FINISH_RING];
                SaListed e = sa_listed(a, k);
                sa_listed_sides(e);
                const uint32_t rl = e.h.x, ql = e.h.y, unit = e.h.w & ~SA_CHAIN_NEXT;
                const SaUnit U = a.units[unit];
                const uint32_t stop_r = sa_stop_offset<SH>(tblb, a.ref, U.q_packed, rl, ql,
                                                           min(a.ref_len - rl, U.q_len - ql), a.xdrop, e.r.z, e.r.w);
                const uint32_t stop_l = sa_stop_offset<SH>(
                    tblb, a.ref + sa_rev_words(a.ref_len), U.q_packed + sa_rev_words(U.q_len), a.ref_len - rl,
                    U.q_len - ql, min(rl, ql), a.xdrop, e.l.z, e.l.w);
                high = (int)(float)((int)e.r.x + (int)e.l.x) >= a.hspthresh;
                const SaChain c = sa_chain_members(a, P, unit, rl, ql, stop_r, stop_l, high);
                hits += c.n;
                tiles += c.tiles;
            }
            l0 += min(l1 - l0, 32u);
            const uint32_t m = __ballot_sync(SA_FULL, high);
            if (high) cand[(c1 + __popc(m & lt)) % SA_FINISH_RING] = make_uint2(k, hits);
            c1 += __popc(m);
            __syncwarp();
        }
        while (c1 - c0 >= 32 || (done && c1 != c0)) {
            const bool on = lane < (int)(c1 - c0);
            uint4 seg = make_uint4(0, 0, 0, 0), x = seg;
            bool is_new = false;
            if (on) {
                const uint2 c = cand[(c0 + lane) % SA_FINISH_RING];
                SaListed e = sa_listed(a, c.x);
                sa_listed_sides(e);
                const uint32_t left = e.l.y + 1;  // left offsets are 1-based, 0 when best is 0
                seg = make_uint4(e.h.x - left, e.h.y - left, e.r.y + left, e.h.z);
                x = make_uint4(e.r.x + e.l.x, e.h.w & ~SA_CHAIN_NEXT, c.y, 0);
                // a key in the set was kept: see sa_keep_candidates
                is_new = !sa_hash_contains(a.hset, ctr->hash_mask, seg.w, seg.x,
                                           sa_set_query(a, a.units[x.y].flags, seg), seg.z);
                if (!is_new) known += c.y;
            }
            c0 += min(c1 - c0, 32u);
            const uint32_t m = __ballot_sync(SA_FULL, is_new);
            if (is_new) {
                fresh_seg[(f1 + __popc(m & lt)) % 64] = seg;
                fresh[(f1 + __popc(m & lt)) % 64] = x;
            }
            f1 += __popc(m);
            __syncwarp();
            if (f1 - f0 >= 32) {
                seg = fresh_seg[(f0 + lane) % 64];
                x = fresh[(f0 + lane) % 64];
                f0 += 32;
                __syncwarp();
                sa_keep_candidates<false>(a, true, seg, (int)x.x, x.y, x.z);
            }
        }
        if (done && f1 != f0) {
            const bool on = lane < (int)(f1 - f0);
            const uint4 seg = fresh_seg[(f0 + lane) % 64], x = fresh[(f0 + lane) % 64];
            f0 = f1;
            sa_keep_candidates<false>(a, on, seg, (int)x.x, x.y, x.z);
        }
        if (done) break;
    }
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        tiles += __shfl_xor_sync(SA_FULL, tiles, s);
        known += __shfl_xor_sync(SA_FULL, known, s);
    }
    if (lane == 0 && tiles) atomicAdd(&ctr->base_steps, tiles);
    if (lane == 0 && known) atomicAdd(&ctr->surv_count, known);
}

// Between the segments of a call: the list starts again (the queue of long hits goes
// on, for the warp kernel after the last one).  An overflow stays to be seen, and
// the sweeps after it find their cursor past every run.  (To end the sweep that
// overflows, by a test where it writes or takes runs, cost every sweep 0.6%.)
__global__ void sa_k_next_segment(SaCounters* ctr, uint64_t list_cap) {
    if (ctr->list_count > list_cap) ctr->sweep_cursor = 1ull << 48;
    else ctr->list_count = ctr->sweep_cursor = ctr->scan_cursor = 0;
}

// ---------------------------------------------------------------------------
// Phase B: two warps per long hit, one per side, 256 bases per step, 8 per lane;
// then the right side's warp runs the keep test and the other follows the chain.
//
// Bound by the latency of a step: its loads are issued a step ahead, and the
// warp's part of it is one scan of sums and one of maxima (10 shuffles).  One warp
// for both sides, and a chain followed by one lane, made it 22 us for a call
// of 881 positions (15 now), 29 (22) for 250,000 against 1 Mbp, 95 (84) for a repeat-masker call.
// ---------------------------------------------------------------------------
struct SaDirResult {
    int best;
    int pos;        // offset of the first base reaching best (-1: best is 0)
    uint32_t stop;  // offset at which the scan stops
};

__device__ __forceinline__ int sa_warp_incl_max(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(SA_FULL, v, o);
        if (lane >= o) v = max(v, t);
    }
    return v;
}

// Rightward scan from base sr of R and sq of Q; `avail` bases until either
// ends.  The end stops the scan by itself, whatever the scores and xdrop (which
// has no upper limit): a base past it scores 0, and the lane that holds the
// first of them stops there.
// tblb: plain scores.
__device__ SaDirResult sa_warp_xdrop(const char* tblb, const uint32_t* __restrict__ R, const uint32_t* __restrict__ Q,
                                     uint32_t sr, uint32_t sq, uint32_t avail, int xdrop) {
    const int lane = threadIdx.x & 31;
    const uint32_t* __restrict__ pr = R + (sr >> 3) + lane;
    const uint32_t* __restrict__ pq = Q + (sq >> 3) + lane;
    const uint32_t shr = (sr & 7u) * 4u, shq = (sq & 7u) * 4u;
    int S_prev = 0, best = 0, bpos = -1;
    uint32_t o = 0, r0 = 0, r1 = 0, q0 = 0, q1 = 0;
    auto fetch = [&](uint32_t at) {  // the lane's words of the step at offset `at`
        if (at + 8u * lane < avail) {
            r0 = __ldg(pr);
            r1 = __ldg(pr + 1);
            q0 = __ldg(pq);
            q1 = __ldg(pq + 1);
        }
        pr += 32;
        pq += 32;
    };
    fetch(0);
    while (true) {
        const uint32_t loff = o + 8u * lane;
        const uint32_t in = avail > loff ? min(avail - loff, 8u) : 0u;
        uint32_t lo, hi;
        sa_merge8(__funnelshift_r(r0, r1, shr), __funnelshift_r(q0, q1, shq), lo, hi);
        fetch(o + 256);
        // prefix sums; the largest and its first base
        int ps[8], p = 0, lmax = INT_MIN, lmax_k = 0, lmin = INT_MAX;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            p += (uint32_t)k < in ? sa_tbl(tblb, lo, hi, k) : 0;
            ps[k] = p;
            if (p > lmax) {
                lmax = p;
                lmax_k = k;
            }
            lmin = min(lmin, p);
        }
        const int incl = sa_warp_incl_sum(p);
        const int base = S_prev + incl - p;
        const int amax = base + lmax;
        const int im = sa_warp_incl_max(amax);
        int before = __shfl_up_sync(SA_FULL, im, 1);
        before = lane ? max(best, before) : best;
        const bool possible = in < 8 || max(before, amax) - (base + lmin) > xdrop;
        if (__any_sync(SA_FULL, possible)) {
            // exact test of the lanes where a stop is possible
            int stop_k = -1, bmax = INT_MIN, bmax_k = 0;
            if (possible) {
                int M = before;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (stop_k < 0) {
                        const int Sv = base + ps[k];
                        M = max(M, Sv);
                        if ((uint32_t)k >= in || M - Sv > xdrop) {
                            stop_k = k;
                        } else if (Sv > bmax) {
                            bmax = Sv;
                            bmax_k = k;
                        }
                    }
            }
            const uint32_t sm = __ballot_sync(SA_FULL, stop_k >= 0);
            if (sm) {
                const int f = __ffs(sm) - 1;
                // best of the lanes before the stop, and of the stopping one up to it
                const int cv = lane < f ? amax : lane == f ? bmax : INT_MIN;
                const int top = __reduce_max_sync(SA_FULL, cv);
                if (top > best) {
                    const int src = __ffs(__ballot_sync(SA_FULL, cv == top)) - 1;
                    bpos = (int)__shfl_sync(SA_FULL, loff + (uint32_t)(lane == f ? bmax_k : lmax_k), src);
                    best = top;
                }
                return {best, bpos, __shfl_sync(SA_FULL, loff + (uint32_t)stop_k, f)};
            }
        }
        const int top = __shfl_sync(SA_FULL, im, 31);
        if (top > best) {
            const int src = __ffs(__ballot_sync(SA_FULL, amax == top)) - 1;
            bpos = (int)__shfl_sync(SA_FULL, loff + (uint32_t)lmax_k, src);
            best = top;
        }
        S_prev += __shfl_sync(SA_FULL, incl, 31);
        o += 256;
    }
}

__global__ void __launch_bounds__(256)
sa_k_extend_warp(const __grid_constant__ SaExtK a, const __grid_constant__ SaParams P) {
    __shared__ int tbl[64];
    __shared__ unsigned long long s_idx[4];
    __shared__ SaDirResult s_dir[4][2];
    __shared__ uint32_t s_follow[4];
    if (threadIdx.x < 64) tbl[threadIdx.x] = P.sub_mat[(threadIdx.x & 7) * 8 + (threadIdx.x >> 3)];
    __syncthreads();
    const char* tblb = reinterpret_cast<const char*>(tbl);
    sa_wait_prior();
    if (a.ctr->error) return;
    const int lane = threadIdx.x & 31, pair = threadIdx.x >> 6;
    const bool left = threadIdx.x & 32u;
    const unsigned long long nlong = min(a.ctr->long_count, (unsigned long long)a.long_cap);
    unsigned long long tiles_acc = 0, next = 0;
    bool kept = false;  // the right warp's last hit
    auto meet = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory"); };
    if (!left && lane == 0) next = atomicAdd(&a.ctr->long_cursor, 1ull);
    while (true) {
        if (!left && lane == 0) s_idx[pair] = next;
        meet();
        const unsigned long long idx = s_idx[pair];
        if (kept && lane == 0) atomicAdd(&a.ctr->surv_count, 1ull + s_follow[pair]);
        kept = false;
        if (idx >= nlong) break;
        if (!left && lane == 0) next = atomicAdd(&a.ctr->long_cursor, 1ull);  // read while this hit is scanned
        const SaLongHit L = a.long_q[idx];
        const bool on = L.unit != SA_LONG_NONE;
        const uint32_t unit = L.unit & ~SA_CHAIN_NEXT;
        const SaUnit U = a.units[on ? unit : 0];
        const uint32_t rl = L.ref_loc, ql = L.query_loc;
        if (on) {
            const SaDirResult d = left ? sa_warp_xdrop(tblb, a.ref + sa_rev_words(a.ref_len),
                                                       U.q_packed + sa_rev_words(U.q_len), a.ref_len - rl,
                                                       U.q_len - ql, min(rl, ql), a.xdrop)
                                       : sa_warp_xdrop(tblb, a.ref, U.q_packed, rl, ql,
                                                       min(a.ref_len - rl, U.q_len - ql), a.xdrop);
            if (lane == 0) s_dir[pair][left] = d;
        }
        meet();
        if (!on) continue;
        const SaDirResult R = s_dir[pair][0];
        SaDirResult Lr = s_dir[pair][1];
        ++Lr.pos;  // left offsets are 1-based, 0 when best is 0
        const int total = R.best + Lr.best;
        const int ext = R.pos + Lr.pos;
        if (left) {  // the dropped hits that follow, while the right warp runs the keep test
            SaChain ch = {0, 0};
            if (L.unit & SA_CHAIN_NEXT)
                ch = sa_warp_chain_members(a, P, unit, rl, ql, R.stop, Lr.stop, (int)(float)total >= a.hspthresh);
            if (lane == 0) s_follow[pair] = ch.n;
            tiles_acc += (R.stop >> 5) + (Lr.stop >> 5) + 2 + ch.tiles;
            continue;
        }
        int cnt[4] = {0, 0, 0, 0};
        const bool eb = sa_entropy_branch(a, total);
        if (eb) {
            const int64_t r0 = (int64_t)rl - Lr.pos, q0 = (int64_t)ql - Lr.pos, nb = (int64_t)ext + 1;
            for (int64_t i = 8 * lane; i < nb; i += 256) {
                uint32_t nm = (nb - i >= 8) ? 0xffu : ((1u << (uint32_t)(nb - i)) - 1u);
                sa_count_matches8(sa_load8(a.ref, r0 + i), sa_load8(U.q_packed, q0 + i), nm, cnt);
            }
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int s = 16; s >= 1; s >>= 1) cnt[b] += __shfl_xor_sync(SA_FULL, cnt[b], s);
        }
        if (lane == 0) {
            int keep, score;
            sa_keep_score(total, ext, cnt, eb, a.hspthresh, &keep, &score);
            kept = keep;
            if (keep) {
                const uint32_t rs = rl - (uint32_t)Lr.pos;
                uint32_t qs = ql - (uint32_t)Lr.pos;
                const uint32_t len = (uint32_t)ext;
                if (U.flags & 2u) qs = a.ref_len - 1 - (qs + len);
                const unsigned long long cl =
                    sa_hash_insert(a.hset, a.ctr->hash_mask, L.scope, rs, qs, len, score, &a.ctr->hash_overflow);
                if (cl != ~0ull) {
                    const unsigned long long i = atomicAdd(&a.ctr->hash_used, 1ull);
                    if (i < a.hset.used_cap) a.hset.used[i] = cl;
                }
            }
        }
    }
    if (left && lane == 0 && tiles_acc) atomicAdd(&a.ctr->base_steps, tiles_acc);
}

// The fast scoring form holds when 7 * max(0, max_sub) <= xdrop (see the
// phase A notes) and its packed scores stay inside 31 bits: a step starts at
// >= -xdrop * SCALE and adds STEP scores of >= min_sub * SCALE - 1 (or
// -(xdrop + 1) * SCALE - 1 past a sequence end).
static bool sa_lane_fast_form(const SaParams& p, int step) {
    long long mx = 0, mn = 0;
    for (int i = 0; i < 64; ++i) {
        mx = std::max<long long>(mx, p.sub_mat[i]);
        mn = std::min<long long>(mn, p.sub_mat[i]);
    }
    const long long scale = 2ll * step, x = p.xdrop;
    const long long low = std::min(mn, -(x + 1)) * scale - 1;
    return x >= 0 && 7 * mx <= x && x * scale - low * step < (1ll << 31) && mx * scale * step < (1ll << 31);
}

// The sweep and the scans after it use the fast form, and what passes
// between them fits its 16-bit fields.
bool sa_sweep_params(const SaParams& p, const SaTuning& t) {
    int mx = 0;
    for (int i = 0; i < 64; ++i) mx = std::max(mx, p.sub_mat[i]);
    return sa_lane_fast_form(p, t.step_bases) && sa_lane_fast_form(p, SA_SWEEP_LEFT) && p.xdrop <= 0xffff &&
           mx <= 0xffff / (int)SA_SWEEP_LEFT;
}

// Scores for which sa_chain_joined's bounds hold: matches of A, C, G and T
// score above 0, and the sweep is in use.
bool sa_chain_params(const SaParams& p, const SaTuning& t) {
    if (!sa_sweep_params(p, t) || p.seed_size > 31) return false;
    for (int b = 0; b < 4; ++b)
        if (p.sub_mat[9 * b] <= 0) return false;
    return true;
}

static SaExtK sa_ext_args(SaWork& w, const SaExtendArgs& x, const SaParams& p, const SaTuning& t) {
    SaExtK a;
    int match = p.sub_mat[0], low = p.sub_mat[1];
    for (int i = 0; i < 4; ++i)
        for (int k = 0; k < 4; ++k) (i == k ? match : low) = std::min(i == k ? match : low, p.sub_mat[8 * i + k]);
    a.chain = x.chain && sa_chain_params(p, t) ? 1u : 0u;
    a.match = match;
    a.swing = match - std::min(low, -1);
    a.mismatches = (uint32_t)std::min(32, p.xdrop / -std::min(low, -1));
    for (int i = 0; i < 16; ++i) a.shift[i] = (uint32_t)p.shape_pos[i < p.kmer_size ? i : 0];
    // buffers of the dedup that are free until then
    a.list = reinterpret_cast<uint4*>(w.out);
    a.list_cap = x.sweep && sa_sweep_params(p, t) ? w.list_cap : 0;
    a.scanned = reinterpret_cast<uint4*>(w.rec[0]);
    // the 48-base window of sa_chain_test holds the seeds of hits up to `gap` either way
    a.gap = (uint32_t)std::max(0, std::min({(int)SA_CHAIN_GAP, p.seed_size - 1, 32 - p.seed_size}));
    a.ref = x.ref;
    a.ref_len = x.ref_len;
    a.pos_table = x.pos_table;
    a.cs = w.cs;
    a.units = w.units;
    a.ctr = w.ctr;
    a.long_q = w.long_q;
    a.long_cap = w.long_cap;
    a.hset = w.hset;
    a.seed_size = x.seed_size;
    a.xdrop = x.xdrop;
    a.hspthresh = x.hspthresh;
    a.noentropy = x.noentropy;
    a.lane_cap = (uint32_t)t.lane_cap;
    a.tile_hits = (uint32_t)t.tile_hits;
    a.substeps = (uint32_t)t.substeps;
    a.switch_now = t.switch_now ? 1u : 0u;
    a.windowed = x.windowed ? 1u : 0u;
    return a;
}

template <int C, int STEP, bool EXACT>
static void sa_lane_launch(const SaExtK& a, const SaParams& p, int grid, size_t smem, cudaStream_t st) {
    if (grid > 0) sa_k_extend_lane<C, STEP, EXACT><<<grid, 256, smem, st>>>(a, p);
    else cudaFuncSetAttribute(sa_k_extend_lane<C, STEP, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <int C>
static void sa_lane_dispatch(const SaExtK& a, const SaParams& p, int step, bool exact, int grid, size_t smem,
                             cudaStream_t st) {
    if (step == 32) {
        if (exact) sa_lane_launch<C, 32, true>(a, p, grid, smem, st);
        else sa_lane_launch<C, 32, false>(a, p, grid, smem, st);
    } else if (step == 16) {
        if (exact) sa_lane_launch<C, 16, true>(a, p, grid, smem, st);
        else sa_lane_launch<C, 16, false>(a, p, grid, smem, st);
    } else {
        if (exact) sa_lane_launch<C, 8, true>(a, p, grid, smem, st);
        else sa_lane_launch<C, 8, false>(a, p, grid, smem, st);
    }
}

// Allows every lane-kernel instance the largest tile's shared memory, once
// per device (kernel attributes cannot be set while a stream is captured).
void sa_prepare_extend_lane(const SaParams& p, const SaTuning& t) {
    (void)t;
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    if (dev < 0 || dev >= 64 || done[dev]) return;
    const size_t smem = sa_lane_smem(1024);
    SaExtK none{};
    for (int step : {8, 16, 32})
        for (bool exact : {false, true}) {
            sa_lane_dispatch<2>(none, p, step, exact, 0, smem, 0);
            sa_lane_dispatch<3>(none, p, step, exact, 0, smem, 0);
            sa_lane_dispatch<4>(none, p, step, exact, 0, smem, 0);
        }
    done[dev] = true;
}

template <int STEP>
static void sa_scan_launch(const SaExtK& a, const SaParams& p, int grid, cudaStream_t st) {
    sa_launch_next(sa_k_scan<STEP>, grid, 256, st, a, p);
    sa_note_launch();
}

void sa_launch_extend_lane(SaWork& w, const SaExtendArgs& x, const SaParams& p, const SaTuning& t, int num_sms,
                           cudaStream_t st, int grid_ctas) {
    sa_prepare_extend_lane(p, t);
    const SaExtK a = sa_ext_args(w, x, p, t);
    if (!a.list_cap) {
        // Register budget follows the CTAs per SM: 4 -> <= 64 registers, 3 -> <= 85, 2 -> <= 128.
        const int grid = grid_ctas > 0 ? grid_ctas : num_sms * t.ext_ctas_per_sm;
        const size_t smem = sa_lane_smem(a.tile_hits);
        const bool exact = !sa_lane_fast_form(p, t.step_bases);
        if (t.ext_ctas_per_sm >= 4) sa_lane_dispatch<4>(a, p, t.step_bases, exact, grid, smem, st);
        else if (t.ext_ctas_per_sm == 3) sa_lane_dispatch<3>(a, p, t.step_bases, exact, grid, smem, st);
        else sa_lane_dispatch<2>(a, p, t.step_bases, exact, grid, smem, st);
        sa_note_launch();
        return;
    }
    // One segment unless the caller knows of more hits (x.hits).  A list that
    // overflows is seen by the host (list_count), which runs the call again: in segments
    // where one sweep had more hits than that, else without the sweep.
    const uint64_t seg = sa_sweep_segment(a.list_cap);
    // A batch fills the chip; a call leaves a place per SM to the kernels beside it
    // and the next of its own (2, 3 and 4 CTAs per SM, ms: 250,000 positions against 100 Mbp 0.323, 0.292, 0.294;
    // against 1 Mbp 0.028, 0.030, 0.033; the 40 calls of a 5 Mbp seeder run on 12 slots
    // 15.4, 15.8, 16.5).
    const int grid = x.ctas > 0 ? x.ctas : num_sms * (grid_ctas > 0 ? 3 : 4);
    uint64_t h0 = 0;
    do {
        const uint64_t h1 = x.hits > h0 + seg ? h0 + seg : ~0ull;
        if (h0) sa_k_next_segment<<<1, 1, 0, st>>>(w.ctr, a.list_cap);
        sa_launch_next(p.transition ? sa_k_sweep<true> : sa_k_sweep<false>, grid, 256, st, a, p, h0, h1);
        sa_note_launch();
        if (t.step_bases == 32) sa_scan_launch<32>(a, p, grid, st);
        else if (t.step_bases == 16) sa_scan_launch<16>(a, p, grid, st);
        else sa_scan_launch<8>(a, p, grid, st);
        sa_launch_next(sa_k_finish, grid, 256, st, a, p);
        sa_note_launch();
        h0 = h1;
    } while (h0 != ~0ull);
}

void sa_launch_extend_warp(SaWork& w, const SaExtendArgs& x, const SaParams& p, const SaTuning& t, int num_sms,
                           cudaStream_t st) {
    sa_launch_next(sa_k_extend_warp, num_sms * 4, t.long_block, st, sa_ext_args(w, x, p, t), p);
    sa_note_launch();
}
