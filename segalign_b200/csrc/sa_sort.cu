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
// which give the record back).  The sort: tiles of SA_SORT_TILE records, straight
// out of the set; then, up to SA_RANK_MAX records, passes in which 8 lanes find a
// record's rank in 8 runs at once; for more, passes that merge pairs of runs.  The host has read the record count by then, so a call launches
// what its size needs: one kernel up to one tile.  An LSD radix sort of every
// key byte, planned on the device, took 46 launches for any size and a one-CTA
// histogram scan per pass.  Measured (one B200, dedup phase, ms, radix sort and
// this): 36 records 0.21 and 0.023, 26 K 0.28 and 0.052, 458 K 1.18 and 0.22, 4.7 M 2.90
// and 2.23; a repeat-masker call's 3.7 K, three sorts and two, 0.67 and 0.083.
#include <algorithm>

#include "sa_launch.h"
#include "sa_radix.cuh"

#define SA_SORT_TILE 1024
// Records up to which rank passes are used.  They and merge passes, us: 26 K records 21 and 62, 57 K
// 26 and 84, 106 K 75 and 100; at 458 K 424 and 143 (each probe is a scattered read).
#define SA_RANK_MAX 131072u
#define SA_MERGE_OUT 2048

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

// Key i of a merge CTA lies at i + i / 8: a thread's 8 keys start 9 places after
// its neighbour's, so that the threads' reads spread over the banks.
#define SA_MERGE_PER 8
#define SA_MERGE_THREADS (SA_MERGE_OUT / SA_MERGE_PER)
struct SaMergeSmem {
    ulonglong2 ab[SA_MERGE_OUT + SA_MERGE_THREADS];
    uint32_t c[SA_MERGE_OUT + SA_MERGE_THREADS];
};

__device__ __forceinline__ void sa_merge_put(SaMergeSmem& s, uint32_t i, const SaKey& k) {
    i += i / SA_MERGE_PER;
    s.ab[i] = make_ulonglong2(k.a, k.b);
    s.c[i] = k.c;
}

__device__ __forceinline__ SaKey sa_merge_get(const SaMergeSmem& s, uint32_t i) {
    i += i / SA_MERGE_PER;
    const ulonglong2 v = s.ab[i];
    return {v.x, v.y, s.c[i]};
}

// One tile: SA_SORT_TILE threads, a key each.
struct SaTileSmem {
    ulonglong2 ab[2][SA_SORT_TILE];
    uint32_t c[2][SA_SORT_TILE];
};

__device__ __forceinline__ uint32_t sa_pow2_at_least(uint32_t n) { return n <= 32 ? 32u : 1u << (32 - __clz(n - 1)); }

// Bitonic sort of the keys of threads 0 .. n2 - 1 (a power of two, at least 32;
// keys that are no records hold all ones).  Partners up to 16 lanes away are
// read by shuffles, the others through shared memory, two buffers in turn:
// 15 of 55 stages have a barrier.  (With the keys in shared memory throughout,
// or merged there, a tile took 35-40 us.)
__device__ __forceinline__ SaKey sa_tile_sort(SaTileSmem& s, SaKey mine, uint32_t n2) {
    const uint32_t t = threadIdx.x;
    uint32_t buf = 0;
    for (uint32_t k = 2; k <= n2; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            SaKey other;
            if (j >= 32) {
                s.ab[buf][t] = make_ulonglong2(mine.a, mine.b);
                s.c[buf][t] = mine.c;
                __syncthreads();
                const ulonglong2 v = s.ab[buf][t ^ j];
                other = {v.x, v.y, s.c[buf][t ^ j]};
                buf ^= 1;
            } else {
                other.a = __shfl_xor_sync(0xffffffffu, mine.a, j);
                other.b = __shfl_xor_sync(0xffffffffu, mine.b, j);
                other.c = __shfl_xor_sync(0xffffffffu, mine.c, j);
            }
            const bool want_less = ((t & j) == 0) == ((t & k) == 0);
            if (sa_key_less(other, mine) == want_less) mine = other;
        }
    return mine;
}

// Distinct HSP i of the set, in claim order; its slot is emptied, so that the set
// is left empty for the next call.
__device__ __forceinline__ SaRec sa_take_from_set(const SaHashSet& hs, uint64_t i, uint32_t& scope) {
    const unsigned long long h = hs.used[i];
    const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(hs.keys + 2 * h);
    SaRec r;
    r.score = hs.score[h];
    r.ref_start = (uint32_t)k.x;
    r.query_start = (uint32_t)(k.y >> 32);
    r.len = (uint32_t)k.y;
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
// (records), into dst.  last: dst gets records, else keys.
template <int ORDER, bool SET>
__global__ void __launch_bounds__(SA_SORT_TILE)
sa_k_tile_sort(SaHashSet hs, const SaRec* src, const uint32_t* src_scope, SaRec* dst, uint32_t* dst_scope, uint64_t n,
               const unsigned long long* d_n, bool last) {
    __shared__ SaTileSmem s;
    if (d_n) n = *d_n;
    const uint64_t base = (uint64_t)blockIdx.x * SA_SORT_TILE, i = base + threadIdx.x;
    if (base >= n) return;
    SaKey k{~0ull, ~0ull, ~0u};
    if (i < n) {
        uint32_t scope;
        SaRec r;
        if (SET) {
            r = sa_take_from_set(hs, i, scope);
        } else {
            r = src[i];
            scope = src_scope[i];
        }
        k = sa_key_of<ORDER>(r, scope);
    }
    k = sa_tile_sort(s, k, sa_pow2_at_least((uint32_t)min((uint64_t)SA_SORT_TILE, n - base)));
    if (i < n) sa_store_key<ORDER>(dst, dst_scope, i, k, last);
}

// A repeat-masker call of at most one tile: diagonal order, unique, final order.
__global__ void __launch_bounds__(SA_SORT_TILE)
sa_k_tile_rm(SaHashSet hs, SaRec* dst, uint32_t n, bool exclude, unsigned long long* n_out) {
    __shared__ SaTileSmem s;
    __shared__ uint32_t ws[SA_SORT_TILE / 32 + 1];
    const uint32_t t = threadIdx.x;
    SaKey k{~0ull, ~0ull, ~0u};
    if (t < n) {
        uint32_t scope;
        const SaRec r = sa_take_from_set(hs, t, scope);
        k = sa_key_of<kOrderDiag>(r, scope);
    }
    k = sa_tile_sort(s, k, sa_pow2_at_least(n));
    __syncthreads();
    s.ab[0][t] = make_ulonglong2(k.a, k.b);
    s.c[0][t] = k.c;
    __syncthreads();
    bool keep = false;
    if (t < n) {
        const uint32_t scope = (uint32_t)(k.a >> 32);
        SaKey b = k;
        if (t) b = {s.ab[0][t - 1].x, s.ab[0][t - 1].y, s.c[0][t - 1]};
        const SaRec r = sa_rec_of<kOrderDiag>(k);
        keep = sa_diag_keep(r, scope, t == 0, sa_rec_of<kOrderDiag>(b), (uint32_t)(b.a >> 32), exclude);
        k = sa_key_of<kOrderFinal>(r, scope);
    }
    uint32_t m;
    const uint32_t at = sa_block_excl_sum<uint32_t, SA_SORT_TILE>(keep, ws, &m);
    if (keep) {
        s.ab[1][at] = make_ulonglong2(k.a, k.b);
        s.c[1][at] = k.c;
    }
    __syncthreads();
    k = {~0ull, ~0ull, ~0u};
    if (t < m) k = {s.ab[1][t].x, s.ab[1][t].y, s.c[1][t]};
    __syncthreads();
    k = sa_tile_sort(s, k, sa_pow2_at_least(m));
    if (t < m) dst[t] = sa_rec_of<kOrderFinal>(k);
    if (t == 0) *n_out = m;
}

// One pass over groups of 8 runs of `run` sorted keys: 8 lanes per record, lane l
// counts the keys of its group's run l below the record's, and the sum is its
// place in the group.  Distinct keys.  Each count is a chain of dependent reads, but
// one pass replaces three merge passes of 14 us, which are latency too.  (A lane per
// tile and a warp per record, all of up to 32 tiles in one pass, took 28 us for 26 K; two
// passes of 8 take 21, and go on past 32 tiles.)
template <int ORDER>
__global__ void __launch_bounds__(256)
sa_k_rank8(const SaRec* src, const uint32_t* src_scope, SaRec* dst, uint32_t* dst_scope, uint64_t n_max,
           const unsigned long long* d_n, uint32_t run, bool last) {
    sa_wait_prior();
    const uint32_t n = (uint32_t)(d_n ? *d_n : n_max);
    const uint32_t lane = threadIdx.x & 7;
    // a warp's four records stay together: i0 is the first
    for (uint32_t i0 = blockIdx.x * 32 + (threadIdx.x >> 5) * 4; i0 < n; i0 += gridDim.x * 32) {
        const uint32_t i = i0 + (threadIdx.x >> 3) % 4;
        SaKey k = {0, 0, 0};
        uint32_t lo = 0, hi = 0, group = 0;
        if (i < n) {
            k = sa_load_key(src, src_scope, i);
            group = i / (8 * run) * (8 * run);
            const uint32_t base = group + lane * run;
            hi = base < n ? min(run, n - base) : 0u;
            if (lane == i % (8 * run) / run) lo = hi = i % run;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (sa_key_less(sa_load_key(src, src_scope, base + mid), k)) lo = mid + 1;
                else hi = mid;
            }
        }
        __syncwarp();
#pragma unroll
        for (int x = 4; x >= 1; x >>= 1) lo += __shfl_xor_sync(0xffffffffu, lo, x);
        if (lane == 0 && i < n) sa_store_key<ORDER>(dst, dst_scope, group + lo, k, last);
    }
}

// One merge pass: runs of `run` sorted keys, pair by pair.  A CTA writes
// SA_MERGE_OUT consecutive outputs: two warps find where its first and last
// output cut the two runs (merge path, a 32-way search: each probe is a
// scattered read), the inputs between go to shared memory, and each thread
// merges 8 outputs.  Moves 40 bytes per record and pass.
template <int ORDER>
__global__ void __launch_bounds__(SA_MERGE_THREADS)
sa_k_merge(const SaRec* __restrict__ src, const uint32_t* __restrict__ src_scope, SaRec* __restrict__ dst,
           uint32_t* __restrict__ dst_scope, uint64_t n, const unsigned long long* d_n, uint64_t run, bool last) {
    __shared__ SaMergeSmem s;
    __shared__ uint64_t cut[2];
    if (d_n) n = *d_n;
    const uint64_t o0 = (uint64_t)blockIdx.x * SA_MERGE_OUT;
    if (o0 >= n) return;
    const uint64_t pair = o0 / (2 * run) * (2 * run);  // pairs of runs are multiples of SA_MERGE_OUT
    const uint64_t la = min(run, n - pair), b0 = pair + la, lb = min(run, n - b0);
    const uint64_t d0 = o0 - pair, d1 = min(d0 + SA_MERGE_OUT, la + lb);
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
#pragma unroll
    for (int j = 0; j < SA_MERGE_PER; ++j) {
        const uint32_t i = j * SA_MERGE_THREADS + threadIdx.x;
        if (i < m) sa_merge_put(s, i, sa_load_key(src, src_scope, i < na ? a0 + i : bb + (i - na)));
    }
    __syncthreads();
    const uint32_t d = threadIdx.x * SA_MERGE_PER;
    SaKey out[SA_MERGE_PER];
    if (d < m) {
        uint32_t lo = d > nb ? d - nb : 0, hi = min(d, na);
        while (lo < hi) {
            const uint32_t i = (lo + hi) >> 1;
            if (sa_key_less(sa_merge_get(s, i), sa_merge_get(s, na + d - 1 - i))) lo = i + 1;
            else hi = i;
        }
        uint32_t ia = lo, ib = d - lo;
        SaKey ka{~0ull, ~0ull, ~0u}, kb = ka;
        if (ia < na) ka = sa_merge_get(s, ia);
        if (ib < nb) kb = sa_merge_get(s, na + ib);
#pragma unroll
        for (int k = 0; k < SA_MERGE_PER; ++k) {
            const bool take_a = ib >= nb || (ia < na && sa_key_less(ka, kb));
            out[k] = take_a ? ka : kb;
            if (take_a) {
                if (++ia < na) ka = sa_merge_get(s, ia);
            } else {
                if (++ib < nb) kb = sa_merge_get(s, na + ib);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SA_MERGE_PER; ++k)
        if (d + k < m) sa_merge_put(s, d + k, out[k]);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < m; i += SA_MERGE_THREADS)
        sa_store_key<ORDER>(dst, dst_scope, o0 + i, sa_merge_get(s, i), last);
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

// Sizes a batch's HSP set (sa_hash_slots).
__global__ void sa_k_hash_init(SaCounters* ctr, unsigned long long max_slots) {
    ctr->hash_mask = sa_hash_slots(ctr->num_hits, max_slots) - 1;
}

unsigned long long sa_hash_max_slots(const SaWork& w) {
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

// From sorted tiles of n keys in buffer b to one order, of records (of keys for
// kOrderDiag).  Returns the buffer they end in.
template <int ORDER>
static int sa_merge_tiles(SaWork& w, int b, uint64_t n, const unsigned long long* d_n, cudaStream_t st) {
    const bool records = ORDER != kOrderDiag;
    if (n <= SA_SORT_TILE) return b;
    if (n <= SA_RANK_MAX) {
        const int g = (int)std::min<uint64_t>((n + 31) / 32, 148 * 8);
        for (uint32_t run = SA_SORT_TILE; run < n; run *= 8, b ^= 1) {
            sa_launch_next(sa_k_rank8<ORDER>, g, 256, st, w.rec[b], w.scope[b], w.rec[b ^ 1], w.scope[b ^ 1], n, d_n, run,
                           8ull * run >= n && records);
            sa_note_launch();
        }
        return b;
    }
    const unsigned g = (unsigned)((n + SA_MERGE_OUT - 1) / SA_MERGE_OUT);
    for (uint64_t run = SA_SORT_TILE; run < n; run *= 2, b ^= 1) {
        sa_k_merge<ORDER><<<g, SA_MERGE_THREADS, 0, st>>>(w.rec[b], w.scope[b], w.rec[b ^ 1], w.scope[b ^ 1], n, d_n, run,
                                                          2 * run >= n && records);
        sa_note_launch();
    }
    return b;
}

int sa_launch_sort(SaWork& w, uint64_t n, cudaStream_t st) {
    if (n == 0) return 0;
    const unsigned tiles = (unsigned)((n + SA_SORT_TILE - 1) / SA_SORT_TILE);
    sa_k_tile_sort<kOrderPlain, true><<<tiles, SA_SORT_TILE, 0, st>>>(w.hset, nullptr, nullptr, w.rec[0], w.scope[0], n,
                                                                    nullptr, tiles == 1);
    sa_note_launch();
    return sa_merge_tiles<kOrderPlain>(w, 0, n, nullptr, st);
}

void sa_launch_unit_counts(SaWork& w, int buf, uint64_t n, uint32_t units, cudaStream_t st) {
    sa_k_unit_counts<<<(units + 127) / 128, 128, 0, st>>>(w.scope[buf], n, units, w.scope_count);
    sa_note_launch();
}

int sa_launch_sort_rm(SaWork& w, uint64_t n, bool exclude, cudaStream_t st) {
    if (n == 0) return 0;
    if (n <= SA_SORT_TILE) {
        sa_k_tile_rm<<<1, SA_SORT_TILE, 0, st>>>(w.hset, w.rec[0], (uint32_t)n, exclude, &w.ctr->uniq_count);
        sa_note_launch();
        return 0;
    }
    const unsigned tiles = (unsigned)((n + SA_SORT_TILE - 1) / SA_SORT_TILE);
    const int G = (int)std::min<uint64_t>(tiles, SA_MAX_CTAS);
    sa_k_tile_sort<kOrderDiag, true><<<tiles, SA_SORT_TILE, 0, st>>>(w.hset, nullptr, nullptr, w.rec[0], w.scope[0], n,
                                                                   nullptr, false);
    sa_note_launch();
    const int b = sa_merge_tiles<kOrderDiag>(w, 0, n, nullptr, st);
    sa_k_diag_count<<<G, 256, 0, st>>>(w.rec[b], w.scope[b], n, exclude, w.cta_a);
    sa_note_launch();
    sa_k_scan_partials<<<1, 1024, 0, st>>>(w.cta_a, w.cta_b, G, &w.ctr->uniq_count, nullptr);
    sa_note_launch();
    sa_k_diag_emit<<<G, 256, 0, st>>>(w.rec[b], w.scope[b], n, exclude, w.cta_a, w.rec[b ^ 1], w.scope[b ^ 1]);
    sa_note_launch();
    // the count after unique stays on the device: n bounds it, and passes past it copy
    sa_k_tile_sort<kOrderFinal, false><<<tiles, SA_SORT_TILE, 0, st>>>(w.hset, w.rec[b ^ 1], w.scope[b ^ 1], w.rec[b],
                                                                     w.scope[b], n, &w.ctr->uniq_count, false);
    sa_note_launch();
    return sa_merge_tiles<kOrderFinal>(w, b, n, &w.ctr->uniq_count, st);
}
