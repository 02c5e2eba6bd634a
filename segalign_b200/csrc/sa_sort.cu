// sa_sort.cu — the set of distinct HSPs of a call and their output order.
//
// Reference (per SeedAndFilter call and MAX_HITS iteration):
//   plain: thrust::stable_sort(hspComp) + unique_copy(hspEqual)
//          src/seed_filter.cu:47-80, 728-732
//   rm:    then stable_sort(hspDiagComp) + unique_copy(hspDiagEqual) +
//          stable_sort(hspFinalComp)   repeat_masker_src/seed_filter.cu:45-107, 797-811
// unique_copy on the CUDA backend keeps element i iff i == 0 or
// !pred(x[i-1], x[i]) with x[i-1] the input predecessor (CUB FlagHeads), which
// matters for the non-transitive hspDiagEqual.
//
// Keys.  Records of one scope come from one (query, target) pair, so the HSP
// score is a function of (ref_start, query_start, len): total is the sum of
// substitution scores over the segment and the entropy factor depends only on
// the segment's base counts.  The HSP set holds distinct (scope, ref_start,
// query_start, len), so hspComp orders a scope totally by (query_start asc,
// len desc, ref_start asc) and unique_copy(hspEqual) keeps every record.
// The rm sorts are stable on their input.  hspDiagComp orders by (diag,
// ref_start, score desc); records equal in these have the same query_start and
// come by len desc from the first sort, so (diag, ref_start, score desc, len
// desc) gives its output without the first sort.  hspFinalComp orders by
// (query_start, score desc, ref_start desc); records equal in these lie on one
// diagonal and come by len desc, so len desc is its last key too.  The scope is
// the most significant key throughout.
//
// A record becomes five words whose lexicographic order is the wanted one (and
// which give the record back), and the sort is a merge sort of them: tiles of
// SA_SORT_TILE records sorted in shared memory, straight out of the set, then
// passes that merge pairs of runs.  The host has read the record count by then,
// so a call launches what its size needs: one kernel up to one tile.  An LSD
// radix sort of every key byte, planned on the device, took 46 launches for any
// size and a one-CTA histogram scan per pass.  Measured (one B200, records ->
// order, ms): 37 records 0.21 -> 0.025, 26 K 0.28 -> 0.10, 458 K 1.18 -> 0.25, 4.7 M
// 2.90 -> 2.03; a repeat-masker call's 3.7 K, three sorts before and two now, 0.67 ->
// 0.14.
#include <algorithm>

#include "sa_launch.h"
#include "sa_radix.cuh"

#define SA_SORT_TILE 2048

enum SaOrder { kOrderPlain, kOrderDiag, kOrderFinal };

struct SaKey {
    uint64_t a, b;
    uint32_t c;
};

__device__ __forceinline__ bool sa_key_less(const SaKey& x, const SaKey& y) {
    if (x.a != y.a) return x.a < y.a;
    if (x.b != y.b) return x.b < y.b;
    return x.c < y.c;
}

__device__ __forceinline__ uint64_t sa_u64(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }

// Scores ascend as (score ^ 0x80000000) unsigned; descending fields are inverted.
template <int ORDER>
__device__ __forceinline__ SaKey sa_key_of(const SaRec& r, uint32_t scope) {
    const uint32_t score_desc = ~((uint32_t)r.score ^ 0x80000000u);
    if (ORDER == kOrderPlain) return {sa_u64(scope, r.query_start), sa_u64(~r.len, r.ref_start), (uint32_t)r.score};
    if (ORDER == kOrderDiag) return {sa_u64(scope, r.ref_start - r.query_start), sa_u64(r.ref_start, score_desc), ~r.len};
    return {sa_u64(scope, r.query_start), sa_u64(score_desc, ~r.ref_start), ~r.len};
}

template <int ORDER>
__device__ __forceinline__ SaRec sa_rec_of(const SaKey& k) {
    SaRec r;
    if (ORDER == kOrderPlain) {
        r.ref_start = (uint32_t)k.b;
        r.query_start = (uint32_t)k.a;
        r.len = ~(uint32_t)(k.b >> 32);
        r.score = (int32_t)k.c;
    } else if (ORDER == kOrderDiag) {
        r.ref_start = (uint32_t)(k.b >> 32);
        r.query_start = r.ref_start - (uint32_t)k.a;
        r.len = ~k.c;
        r.score = (int32_t)(~(uint32_t)k.b ^ 0x80000000u);
    } else {
        r.ref_start = ~(uint32_t)k.b;
        r.query_start = (uint32_t)k.a;
        r.len = ~k.c;
        r.score = (int32_t)(~(uint32_t)(k.b >> 32) ^ 0x80000000u);
    }
    return r;
}

// Keys in a record buffer between the passes.
__device__ __forceinline__ SaKey sa_load_key(const SaRec* rec, const uint32_t* scope, uint64_t i) {
    const ulonglong2 v = reinterpret_cast<const ulonglong2*>(rec)[i];
    return {v.x, v.y, scope[i]};
}

template <int ORDER>
__device__ __forceinline__ void sa_store_key(SaRec* rec, uint32_t* scope, uint64_t i, const SaKey& k, bool last) {
    if (last) {
        rec[i] = sa_rec_of<ORDER>(k);
        scope[i] = (uint32_t)(k.a >> 32);
    } else {
        reinterpret_cast<ulonglong2*>(rec)[i] = make_ulonglong2(k.a, k.b);
        scope[i] = k.c;
    }
}

struct SaTileSmem {
    ulonglong2 ab[SA_SORT_TILE];
    uint32_t c[SA_SORT_TILE];
    unsigned long long ws[33];
};

// Bitonic sort of the tile's first n2 (a power of two, <= SA_SORT_TILE) keys by
// SA_SORT_TILE / 2 threads, one pair per thread and stage.  A warp's pairs at
// distance <= 32 lie in its own 64 keys, so those stages need no block barrier.
__device__ __forceinline__ void sa_tile_sort(SaTileSmem& s, uint32_t n2) {
    const uint32_t t = threadIdx.x;
    __syncthreads();
    for (uint32_t k = 2; k <= n2; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) __syncthreads();
            else __syncwarp();
            if (t < n2 / 2) {
                const uint32_t i = ((t & ~(j - 1)) << 1) | (t & (j - 1)), p = i + j;
                const ulonglong2 x = s.ab[i], y = s.ab[p];
                const uint32_t xc = s.c[i], yc = s.c[p];
                const bool less = sa_key_less({y.x, y.y, yc}, {x.x, x.y, xc});
                if (less == ((i & k) == 0)) {
                    s.ab[i] = y;
                    s.ab[p] = x;
                    s.c[i] = yc;
                    s.c[p] = xc;
                }
            }
        }
    __syncthreads();
}

__device__ __forceinline__ uint32_t sa_pow2_at_least(uint32_t n) { return n <= 64 ? 64u : 1u << (32 - __clz(n - 1)); }

__device__ __forceinline__ void sa_tile_put(SaTileSmem& s, uint32_t i, const SaKey& k) {
    s.ab[i] = make_ulonglong2(k.a, k.b);
    s.c[i] = k.c;
}

__device__ __forceinline__ SaKey sa_tile_get(const SaTileSmem& s, uint32_t i) { return {s.ab[i].x, s.ab[i].y, s.c[i]}; }

// Distinct HSP i of the set, in claim order; its slot is emptied, so that the set
// is left empty for the next call.
__device__ __forceinline__ SaRec sa_take_from_set(const SaHashSet& hs, uint64_t i, uint32_t& scope) {
    const unsigned long long h = hs.used[i];
    const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(hs.keys + 2 * h);
    SaRec r;
    r.ref_start = (uint32_t)k.x;
    r.query_start = (uint32_t)(k.y >> 32);
    r.len = (uint32_t)k.y;
    r.score = hs.score[h];
    scope = (uint32_t)(k.x >> 32);
    *reinterpret_cast<ulonglong2*>(hs.keys + 2 * h) = make_ulonglong2(~0ull, ~0ull);
    return r;
}

// hspDiagEqual (repeat_masker_src/seed_filter.cu:45-50).
__device__ __forceinline__ bool sa_rec_diag_equal(const SaRec& x, const SaRec& y) {
    if ((uint32_t)(x.ref_start - x.query_start) != (uint32_t)(y.ref_start - y.query_start)) return false;
    const bool xin = x.ref_start >= y.ref_start && (uint32_t)(x.ref_start + x.len) <= (uint32_t)(y.ref_start + y.len);
    const bool yin = y.ref_start >= x.ref_start && (uint32_t)(y.ref_start + y.len) <= (uint32_t)(x.ref_start + x.len);
    return xin || yin;
}

// Whether unique_copy(hspDiagEqual) keeps r after its predecessor in the
// diagonal order; exclude: main-diagonal records of the plus strand go as well.
__device__ __forceinline__ bool sa_diag_keep(const SaRec& r, uint32_t scope, bool first, const SaRec& before,
                                             uint32_t before_scope, bool exclude) {
    if (exclude && r.ref_start == r.query_start) return false;
    return first || before_scope != scope || !sa_rec_diag_equal(before, r);
}

// Sorts one tile of the n records: out of the set (SET) or out of src/src_scope
// (records), into dst.  last: dst gets records, else keys.  Bound by the
// latency of the scattered set reads and of the 66 stages; 2048 records of 20
// bytes leave 4 CTAs per SM their shared memory.
template <int ORDER, bool SET>
__global__ void __launch_bounds__(SA_SORT_TILE / 2)
sa_k_tile_sort(SaHashSet hs, const SaRec* src, const uint32_t* src_scope, SaRec* dst, uint32_t* dst_scope, uint64_t n,
               const unsigned long long* d_n, bool last) {
    __shared__ SaTileSmem s;
    if (d_n) n = *d_n;
    const uint64_t base = (uint64_t)blockIdx.x * SA_SORT_TILE;
    if (base >= n) return;
    const uint32_t cnt = (uint32_t)min((uint64_t)SA_SORT_TILE, n - base), n2 = sa_pow2_at_least(cnt);
    for (uint32_t i = threadIdx.x; i < n2; i += SA_SORT_TILE / 2) {
        SaKey k{~0ull, ~0ull, ~0u};
        if (i < cnt) {
            uint32_t scope;
            SaRec r;
            if (SET) {
                r = sa_take_from_set(hs, base + i, scope);
            } else {
                r = src[base + i];
                scope = src_scope[base + i];
            }
            k = sa_key_of<ORDER>(r, scope);
        }
        sa_tile_put(s, i, k);
    }
    sa_tile_sort(s, n2);
    for (uint32_t i = threadIdx.x; i < cnt; i += SA_SORT_TILE / 2)
        sa_store_key<ORDER>(dst, dst_scope, base + i, sa_tile_get(s, i), last);
}

// A repeat-masker call of at most one tile: diagonal order, unique, final order.
__global__ void __launch_bounds__(SA_SORT_TILE / 2)
sa_k_tile_rm(SaHashSet hs, SaRec* dst, uint32_t n, bool exclude, unsigned long long* n_out) {
    __shared__ SaTileSmem s;
    constexpr int T = SA_SORT_TILE / 2;
    const uint32_t t = threadIdx.x, n2 = sa_pow2_at_least(n);
    for (uint32_t i = t; i < n2; i += T) {
        SaKey k{~0ull, ~0ull, ~0u};
        if (i < n) {
            uint32_t scope;
            const SaRec r = sa_take_from_set(hs, i, scope);
            k = sa_key_of<kOrderDiag>(r, scope);
        }
        sa_tile_put(s, i, k);
    }
    sa_tile_sort(s, n2);
    // records 2t and 2t + 1 of this thread, and the one before
    SaRec r[3];
    uint32_t sc[3];
    bool keep[2];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const uint32_t i = 2 * t + j;  // record i - 1
        if (i >= 1 && i <= n) {
            const SaKey k = sa_tile_get(s, i - 1);
            r[j] = sa_rec_of<kOrderDiag>(k);
            sc[j] = (uint32_t)(k.a >> 32);
        }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
        keep[j] = 2 * t + j < n && sa_diag_keep(r[j + 1], sc[j + 1], 2 * t + j == 0, r[j], sc[j], exclude);
    unsigned long long m;
    const uint32_t at = (uint32_t)sa_block_excl_sum<unsigned long long, T>((unsigned long long)keep[0] + keep[1], s.ws, &m);
    const uint32_t m2 = sa_pow2_at_least((uint32_t)m);
    if (keep[0]) sa_tile_put(s, at, sa_key_of<kOrderFinal>(r[1], sc[1]));
    if (keep[1]) sa_tile_put(s, at + keep[0], sa_key_of<kOrderFinal>(r[2], sc[2]));
    for (uint32_t i = (uint32_t)m + t; i < m2; i += T) sa_tile_put(s, i, {~0ull, ~0ull, ~0u});
    __syncthreads();
    sa_tile_sort(s, m2);
    for (uint32_t i = t; i < (uint32_t)m; i += T) dst[i] = sa_rec_of<kOrderFinal>(sa_tile_get(s, i));
    if (t == 0) *n_out = m;
}

// One merge pass: runs of `run` sorted keys, pair by pair.  A CTA writes
// SA_SORT_TILE consecutive outputs: two warps find where its first and last
// output cut the two runs (merge path, a 32-way search: each probe is a
// scattered read), the inputs between go to shared memory, and each thread
// merges 8 outputs.  Bound by memory traffic (40 bytes per record and pass) for
// large n, by latency for small.
template <int ORDER>
__global__ void __launch_bounds__(256)
sa_k_merge(const SaRec* __restrict__ src, const uint32_t* __restrict__ src_scope, SaRec* __restrict__ dst,
           uint32_t* __restrict__ dst_scope, uint64_t n, const unsigned long long* d_n, uint64_t run, bool last) {
    __shared__ SaTileSmem s;
    __shared__ uint64_t cut[2];
    if (d_n) n = *d_n;
    const uint64_t o0 = (uint64_t)blockIdx.x * SA_SORT_TILE;
    if (o0 >= n) return;
    const uint64_t pair = o0 / (2 * run) * (2 * run);  // runs are multiples of the tile
    const uint64_t la = min(run, n - pair), b0 = pair + la, lb = min(run, n - b0);
    const uint64_t d0 = o0 - pair, d1 = min(d0 + SA_SORT_TILE, la + lb);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 2) {
        const uint64_t d = warp ? d1 : d0;
        uint64_t lo = d > lb ? d - lb : 0, hi = min(d, la);  // outputs before d that come from the first run
        while (lo < hi) {
            const uint64_t step = (hi - lo + 31) / 32, i = lo + (uint64_t)lane * step;
            const bool first = i < hi && sa_key_less(sa_load_key(src, src_scope, pair + i),
                                                     sa_load_key(src, src_scope, b0 + (d - 1 - i)));
            const uint32_t c = __popc(__ballot_sync(0xffffffffu, first));
            if (c == 0) break;
            const uint64_t nlo = lo + (uint64_t)(c - 1) * step + 1;
            hi = min(hi, lo + (uint64_t)c * step);
            lo = nlo;
        }
        if (lane == 0) cut[warp] = lo;
    }
    __syncthreads();
    const uint32_t na = (uint32_t)(cut[1] - cut[0]), m = (uint32_t)(d1 - d0), nb = m - na;
    const uint64_t a0 = pair + cut[0], bb = b0 + (d0 - cut[0]);
    for (uint32_t i = threadIdx.x; i < m; i += 256)
        sa_tile_put(s, i, sa_load_key(src, src_scope, i < na ? a0 + i : bb + (i - na)));
    __syncthreads();
    constexpr uint32_t PER = SA_SORT_TILE / 256;
    const uint32_t d = min(threadIdx.x * PER, m);
    uint32_t lo = d > nb ? d - nb : 0, hi = min(d, na);
    while (lo < hi) {
        const uint32_t i = (lo + hi) >> 1;
        if (sa_key_less(sa_tile_get(s, i), sa_tile_get(s, na + d - 1 - i))) lo = i + 1;
        else hi = i;
    }
    uint32_t ia = lo, ib = na + d - lo;
    SaKey out[PER];
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
        if (d + k < m) {
            const bool take_a = ib >= m || (ia < na && sa_key_less(sa_tile_get(s, ia), sa_tile_get(s, ib)));
            out[k] = sa_tile_get(s, take_a ? ia : ib);
            ia += take_a;
            ib += !take_a;
        }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k)
        if (d + k < m) sa_tile_put(s, d + k, out[k]);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < m; i += 256) sa_store_key<ORDER>(dst, dst_scope, o0 + i, sa_tile_get(s, i), last);
}

// unique_copy(hspDiagEqual) over records in diagonal order (keys of
// kOrderDiag): per-CTA counts, then the ordered compaction into records.
__device__ __forceinline__ bool sa_diag_keep_at(const SaRec* rec, const uint32_t* scope, uint64_t i, bool exclude) {
    const SaKey k = sa_load_key(rec, scope, i);
    SaRec before{};
    uint32_t before_scope = 0;
    if (i) {
        const SaKey b = sa_load_key(rec, scope, i - 1);
        before = sa_rec_of<kOrderDiag>(b);
        before_scope = (uint32_t)(b.a >> 32);
    }
    return sa_diag_keep(sa_rec_of<kOrderDiag>(k), (uint32_t)(k.a >> 32), i == 0, before, before_scope, exclude);
}

__global__ void __launch_bounds__(256)
sa_k_diag_count(const SaRec* rec, const uint32_t* scope, uint64_t n, bool exclude, unsigned long long* cta_a) {
    uint64_t a, b;
    sa_cta_range(n, a, b);
    unsigned long long c = 0;
    for (uint64_t i = a + threadIdx.x; i < b; i += 256) c += sa_diag_keep_at(rec, scope, i, exclude);
    __shared__ unsigned long long ws[9];
    unsigned long long tot;
    sa_block_excl_sum<unsigned long long, 256>(c, ws, &tot);
    if (threadIdx.x == 0) cta_a[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(256)
sa_k_diag_emit(const SaRec* rec, const uint32_t* scope, uint64_t n, bool exclude, const unsigned long long* cta_a,
               SaRec* out, uint32_t* out_scope) {
    uint64_t a, b;
    sa_cta_range(n, a, b);
    unsigned long long base = cta_a[blockIdx.x];
    __shared__ unsigned long long ws[9];
    for (uint64_t r0 = a; r0 < b; r0 += 256) {
        const uint64_t i = r0 + threadIdx.x;
        const bool k = i < b && sa_diag_keep_at(rec, scope, i, exclude);
        unsigned long long tot;
        const unsigned long long e = sa_block_excl_sum<unsigned long long, 256>((unsigned long long)k, ws, &tot);
        if (k) {
            const SaKey x = sa_load_key(rec, scope, i);
            out[base + e] = sa_rec_of<kOrderDiag>(x);
            out_scope[base + e] = (uint32_t)(x.a >> 32);
        }
        base += tot;
    }
}

// Records per batch unit: the sorted scopes (unit << 4 | iteration) of unit u
// start at the first one >= u << 4.
__global__ void sa_k_unit_counts(const uint32_t* __restrict__ scope, uint64_t n, uint32_t units, uint32_t* count) {
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < units; u += gridDim.x * blockDim.x) {
        uint64_t at[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            uint64_t lo = 0, hi = n;
            while (lo < hi) {
                const uint64_t mid = (lo + hi) >> 1;
                if ((scope[mid] >> 4) < u + e) lo = mid + 1;
                else hi = mid;
            }
            at[e] = lo;
        }
        count[u] = (uint32_t)(at[1] - at[0]);
    }
}

// Sizes the call's HSP set: the smallest power of two >= 2 * hits (at least
// 1024), at most `max_slots` (a power of two, the whole table).  The table is
// known to be empty (the previous call's output emptied the slots it used).
__global__ void sa_k_hash_init(SaCounters* ctr, unsigned long long max_slots) {
    unsigned long long want = 2 * ctr->num_hits;
    if (want < 1024) want = 1024;
    unsigned long long slots = 1;
    while (slots < want && slots < max_slots) slots <<= 1;
    ctr->hash_mask = slots - 1;
}

static unsigned long long sa_hash_max_slots(const SaWork& w) {
    unsigned long long max_slots = 1;
    while (max_slots * 2 <= 2 * w.surv_cap) max_slots <<= 1;
    return max_slots;
}

void sa_launch_hash_init(SaWork& w, cudaStream_t st) {
    sa_k_hash_init<<<1, 1, 0, st>>>(w.ctr, sa_hash_max_slots(w));
    sa_note_launch();
}

__global__ void sa_k_hash_clear(unsigned long long* keys, unsigned long long n) {
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x)
        keys[i] = ~0ull;
}

void sa_launch_hash_clear(SaWork& w, cudaStream_t st) {
    sa_k_hash_clear<<<148 * 8, 256, 0, st>>>(w.hset.keys, 2 * sa_hash_max_slots(w));
    sa_note_launch();
}

int sa_check_set(const SaWork& w, const SaCounters& c) {
    if (c.error) return (int)c.error;
    return c.hash_overflow || c.hash_used > w.surv_cap || c.hash_used > w.hset.used_cap ? SA_DERR_SURV_OVERFLOW : 0;
}

// Merge passes over n keys in buffer b; the last one writes records.  Returns
// the buffer they end in.
template <int ORDER>
static int sa_merge_passes(SaWork& w, int b, uint64_t n, const unsigned long long* d_n, cudaStream_t st) {
    const unsigned tiles = (unsigned)((n + SA_SORT_TILE - 1) / SA_SORT_TILE);
    for (uint64_t run = SA_SORT_TILE; run < n; run *= 2, b ^= 1) {
        sa_k_merge<ORDER><<<tiles, 256, 0, st>>>(w.rec[b], w.scope[b], w.rec[b ^ 1], w.scope[b ^ 1], n, d_n, run,
                                                 2 * run >= n && ORDER != kOrderDiag);
        sa_note_launch();
    }
    return b;
}

int sa_launch_sort(SaWork& w, uint64_t n, cudaStream_t st) {
    if (n == 0) return 0;
    const unsigned tiles = (unsigned)((n + SA_SORT_TILE - 1) / SA_SORT_TILE);
    sa_k_tile_sort<kOrderPlain, true><<<tiles, SA_SORT_TILE / 2, 0, st>>>(w.hset, nullptr, nullptr, w.rec[0], w.scope[0], n,
                                                                    nullptr, tiles == 1);
    sa_note_launch();
    return sa_merge_passes<kOrderPlain>(w, 0, n, nullptr, st);
}

void sa_launch_unit_counts(SaWork& w, int buf, uint64_t n, uint32_t units, cudaStream_t st) {
    sa_k_unit_counts<<<(units + 127) / 128, 128, 0, st>>>(w.scope[buf], n, units, w.scope_count);
    sa_note_launch();
}

int sa_launch_sort_rm(SaWork& w, uint64_t n, bool exclude, cudaStream_t st) {
    if (n == 0) return 0;
    if (n <= SA_SORT_TILE) {
        sa_k_tile_rm<<<1, SA_SORT_TILE / 2, 0, st>>>(w.hset, w.rec[0], (uint32_t)n, exclude, &w.ctr->uniq_count);
        sa_note_launch();
        return 0;
    }
    const unsigned tiles = (unsigned)((n + SA_SORT_TILE - 1) / SA_SORT_TILE);
    const int G = (int)std::min<uint64_t>(tiles, SA_MAX_CTAS);
    sa_k_tile_sort<kOrderDiag, true><<<tiles, SA_SORT_TILE / 2, 0, st>>>(w.hset, nullptr, nullptr, w.rec[0], w.scope[0], n,
                                                                   nullptr, false);
    sa_note_launch();
    const int b = sa_merge_passes<kOrderDiag>(w, 0, n, nullptr, st);
    sa_k_diag_count<<<G, 256, 0, st>>>(w.rec[b], w.scope[b], n, exclude, w.cta_a);
    sa_note_launch();
    sa_k_scan_partials<<<1, 1024, 0, st>>>(w.cta_a, w.cta_b, G, &w.ctr->uniq_count, nullptr);
    sa_note_launch();
    sa_k_diag_emit<<<G, 256, 0, st>>>(w.rec[b], w.scope[b], n, exclude, w.cta_a, w.rec[b ^ 1], w.scope[b ^ 1]);
    sa_note_launch();
    // the count after unique stays on the device: n bounds it, and passes past it copy
    sa_k_tile_sort<kOrderFinal, false><<<tiles, SA_SORT_TILE / 2, 0, st>>>(w.hset, w.rec[b ^ 1], w.scope[b ^ 1], w.rec[b],
                                                                     w.scope[b], n, &w.ctr->uniq_count, false);
    sa_note_launch();
    return sa_merge_passes<kOrderFinal>(w, b, n, &w.ctr->uniq_count, st);
}
