// sa_lookup.cu — seed lookup: bucket bounds per seed, hit prefix, compaction
// of seeds that have hits, and the MAX_HITS iteration split.
//
// Reference behaviour restated here:
//   find_num_hits + inclusive_scan + num_hits D2H   src/seed_filter.cu:129-154, 680-684
//   MAX_HITS split (lower_bound loop)              src/seed_filter.cu:686-697
//   find_hits hit records {pos+seed_size, j+seed_size}   src/seed_filter.cu:156-202
// The reference materialises one 16-byte record per hit; here only seeds with
// hits are compacted (E = exclusive hit prefix, lo = bucket start, j), and the
// extension kernel expands hits on the fly from that list.
#include "sa_launch.h"
#include "sa_radix.cuh"

// Error codes raised on the device (SaCounters::error).
#define SA_DERR_BAD_KEY 1        // seed key outside the 4^K table
#define SA_DERR_MAX_HITS 2       // one seed holds >= MAX_HITS hits (reference UB)
#define SA_DERR_ITERS 3          // more MAX_HITS iterations than supported

// A call's words are split over the CTAs at multiples of 4 (16-byte loads).
__device__ __forceinline__ void sa_seed_range(uint64_t n, uint64_t& a, uint64_t& b) {
    sa_cta_range((n + 3) / 4, a, b);
    a *= 4;
    b = min(n, 4 * b);
}

// Bucket bounds of every word, and per CTA its hits and its words with hits; the
// CTA that finishes last turns these into prefixes and sets what depends on the
// totals: the number of MAX_HITS iterations (src/seed_filter.cu:686) and the
// size of the HSP set.  (A launch each for the prefixes, the iterations, the
// scopes and the set took 13 us of a call's 76.)
//
// Bound by latency: word, bucket bounds and, with `chain`, the query window are
// loads that wait for one another, so a thread takes SA_WORDS words at a time and
// a CTA has 512 threads (1.3 M words with transitions: 58 us with one word at a time and 256
// threads, 56 with four, 38 with both; the next kernel 64, 30 and 22 us).
//
// With `chain`, also checks that the call's words are every seed word of the
// query window [j_lo, j_hi), in seeder order (src/seeder.cpp:57-74): word i is
// the one that its position and its place i % S in the position's group of S
// words call for, positions increase, and there are as many of them as valid
// windows (counted into ctr->windows).  Only then may the extension tell a call's
// hits from the sequences alone.  A word out of place sets ctr->chain_bad; nothing
// else depends on the check.  Hits of different iterations are deduplicated
// apart, so chains need one iteration too.
#define SA_WORDS 4
#define SA_CALL_BLOCK 512
__global__ void __launch_bounds__(SA_CALL_BLOCK)
sa_k_lookup_count(const uint64_t* __restrict__ seeds, const SaCallDesc* __restrict__ desc,
                  const uint32_t* __restrict__ index, uint32_t nbuckets, uint32_t* __restrict__ s_lo,
                  uint32_t* __restrict__ s_cnt, unsigned long long* cta_a, unsigned long long* cta_b,
                  SaCounters* ctr, const SaUnit* __restrict__ units, SaParams P, int chain,
                  unsigned long long max_slots) {
    constexpr int J = SA_WORDS;
    sa_allow_next();
    const uint64_t n = desc->num_seeds;
    uint64_t a, b;
    sa_seed_range(n, a, b);
    unsigned long long hits = 0, nz = 0;
    const uint32_t S = P.transition ? 1u + (uint32_t)P.kmer_size : 1u;
    SaUnit U{};
    bool bad = false;
    if (chain) {
        U = units[0];
        const uint64_t span = U.j_hi > U.j_lo ? U.j_hi - U.j_lo : 0;
        // few words over a wide window are no seeder's chunk, and counting its windows would cost more than the call
        if (n % S || U.j_hi > U.q_len || span > (1u << 20) + 2 * n) {
            bad = true;
            chain = 0;
        } else {
            uint64_t ga, gb;  // words of 8 positions
            sa_cta_range(span ? ((U.j_hi - 1) >> 3) - (U.j_lo >> 3) + 1 : 0, ga, gb);
            unsigned long long windows = 0;
            for (uint64_t g = (U.j_lo >> 3) + ga + threadIdx.x; g < (U.j_lo >> 3) + gb; g += SA_CALL_BLOCK) {
                uint32_t ok = sa_valid_windows8(U.q_packed + g, (uint32_t)P.seed_size);
                if (8 * g < U.j_lo) ok &= 0xffu << (U.j_lo - 8 * g);
                if (8 * g + 8 > U.j_hi) ok &= 0xffu >> (8 * g + 8 - U.j_hi);
                windows += __popc(ok & 0xffu);
            }
#pragma unroll
            for (int s = 16; s >= 1; s >>= 1) windows += __shfl_xor_sync(0xffffffffu, windows, s);
            if ((threadIdx.x & 31) == 0 && windows) atomicAdd(&ctr->windows, windows);
        }
    }
    for (uint64_t i0 = a + threadIdx.x; i0 < b; i0 += SA_CALL_BLOCK * J) {
        uint64_t word[J];
        uint32_t lo[J], hi[J];
#pragma unroll
        for (int k = 0; k < J; ++k) word[k] = i0 + SA_CALL_BLOCK * k < b ? seeds[i0 + SA_CALL_BLOCK * k] : 0;
#pragma unroll
        for (int k = 0; k < J; ++k) {
            const uint32_t key = (uint32_t)(word[k] >> 32);
            lo[k] = hi[k] = 0;
            if (i0 + SA_CALL_BLOCK * k < b) {
                if (key < nbuckets) {
                    hi[k] = __ldg(index + key);
                    lo[k] = key ? __ldg(index + key - 1) : 0u;
                } else {
                    atomicCAS(&ctr->error, 0ull, (unsigned long long)SA_DERR_BAD_KEY);
                }
            }
        }
        if (chain) {
#pragma unroll
            for (int k = 0; k < J; ++k) {
                const uint64_t i = i0 + SA_CALL_BLOCK * k;
                if (i >= b) break;
                const uint32_t key = (uint32_t)(word[k] >> 32), j = (uint32_t)word[k], v = (uint32_t)i % S;
                const uint32_t before = i ? (uint32_t)seeds[i - 1] : 0u;
                bool ok = j >= U.j_lo && j < U.j_hi && (v ? before == j : (i == 0 || before < j));
                if (ok) {
                    // the position's first word is checked against its window, the others against that word
                    const uint32_t k0 = v ? (uint32_t)(seeds[i - v] >> 32) : sa_window_key(U.q_packed, j, P);
                    ok = k0 != SA_INVALID_KEY && key == (v ? k0 ^ (2u << (2 * (v - 1))) : k0);
                }
                bad |= !ok;
            }
        }
#pragma unroll
        for (int k = 0; k < J; ++k) {
            const uint64_t i = i0 + SA_CALL_BLOCK * k;
            if (i < b) {
                s_lo[i] = lo[k];
                s_cnt[i] = hi[k] - lo[k];
                hits += hi[k] - lo[k];
                nz += hi[k] != lo[k];
            }
        }
    }
    if (bad) ctr->chain_bad = 1;
    __shared__ unsigned long long ws[SA_CALL_BLOCK / 32 + 1];
    __shared__ bool last;
    unsigned long long th, tz;
    sa_block_excl_sum<unsigned long long, SA_CALL_BLOCK>(hits, ws, &th);
    sa_block_excl_sum<unsigned long long, SA_CALL_BLOCK>(nz, ws, &tz);
    if (threadIdx.x == 0) {
        cta_a[blockIdx.x] = th;
        cta_b[blockIdx.x] = tz;
    }
    __threadfence();  // this CTA's sums and counters before its ticket
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&ctr->lookup_done, 1ull) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    constexpr int PER = SA_MAX_CTAS / SA_CALL_BLOCK;  // sums per thread
    unsigned long long va[PER], vb[PER], sa = 0, sb = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const uint32_t c = PER * threadIdx.x + k;
        va[k] = c < gridDim.x ? __ldcg(cta_a + c) : 0;
        vb[k] = c < gridDim.x ? __ldcg(cta_b + c) : 0;
        sa += va[k];
        sb += vb[k];
    }
    unsigned long long ea = sa_block_excl_sum<unsigned long long, SA_CALL_BLOCK>(sa, ws, &th);
    unsigned long long eb = sa_block_excl_sum<unsigned long long, SA_CALL_BLOCK>(sb, ws, &tz);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const uint32_t c = PER * threadIdx.x + k;
        if (c < gridDim.x) {
            cta_a[c] = ea;
            cta_b[c] = eb;
        }
        ea += va[k];
        eb += vb[k];
    }
    if (threadIdx.x == 0) {
        ctr->num_hits = th;
        ctr->nnz = tz;
        ctr->hash_mask = sa_hash_slots(th, max_slots) - 1;
        const uint64_t MH = desc->max_hits;
        uint64_t num_iter = MH ? th / MH + 1 : 1;
        if (num_iter > 1 || __ldcg(&ctr->windows) * S != n) ctr->chain_bad = 1;
        if (num_iter > SA_MAX_ITERS) {
            atomicCAS(&ctr->error, 0ull, (unsigned long long)SA_DERR_ITERS);
            num_iter = 1;
        }
        ctr->num_iter = num_iter;
    }
}

// The words with hits, compacted.  A thread takes four consecutive words, and
// both prefixes come from one scan: a round's hits above the low 12 bits, its
// words with hits in them.  With more than one iteration the scope is the
// word's index until sa_k_iterations, which also needs the hit prefix of every word.
__global__ void __launch_bounds__(SA_CALL_BLOCK)
sa_k_lookup_emit(const uint64_t* __restrict__ seeds, const SaCallDesc* __restrict__ desc,
                 const uint32_t* s_lo, const uint32_t* s_cnt, uint64_t* s_P, SaSeedList cs, const unsigned long long* cta_a,
                 const unsigned long long* cta_b, SaCounters* ctr) {
    sa_wait_prior();
    sa_allow_next();
    const uint64_t n = desc->num_seeds;
    uint64_t a, b;
    sa_seed_range(n, a, b);
    const bool split = ctr->num_iter > 1;
    unsigned long long hbase = cta_a[blockIdx.x], cbase = cta_b[blockIdx.x];
    __shared__ unsigned long long ws[SA_CALL_BLOCK / 32 + 1];
    for (uint64_t r = a; r < b; r += 4 * SA_CALL_BLOCK) {
        const uint64_t i0 = r + 4 * threadIdx.x;
        uint32_t cnt[4] = {0, 0, 0, 0};
        if (i0 + 4 <= b) {
            const uint4 v = *reinterpret_cast<const uint4*>(s_cnt + i0);
            cnt[0] = v.x, cnt[1] = v.y, cnt[2] = v.z, cnt[3] = v.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (i0 + k < b) cnt[k] = s_cnt[i0 + k];
        }
        unsigned long long sum = 0, total;
#pragma unroll
        for (int k = 0; k < 4; ++k) sum += ((unsigned long long)cnt[k] << 12) + (cnt[k] != 0);
        const unsigned long long e = sa_block_excl_sum<unsigned long long, SA_CALL_BLOCK>(sum, ws, &total);
        uint64_t h = hbase + (e >> 12), c = cbase + (e & 4095);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (cnt[k]) {
                cs.E[c] = h;
                cs.lo[c] = s_lo[i0 + k];
                cs.qpos[c] = (uint32_t)seeds[i0 + k];
                cs.scope[c] = split ? (uint32_t)(i0 + k) : 0u;
                cs.unit[c] = 0;
                ++c;
                h += cnt[k];
            }
            if (split && i0 + k < b) s_P[i0 + k] = h;  // inclusive prefix (thrust::inclusive_scan, :682)
        }
        hbase += total >> 12;
        cbase += total & 4095;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) cs.E[ctr->nnz] = ctr->num_hits;
}

// MAX_HITS iterations (src/seed_filter.cu:686-697), for calls with more than one:
// limit[i] = lower_bound(P, lim) - 1, lim = P[limit[i]] + MAX_HITS, last limit =
// n - 1; a word's scope is the first iteration whose limit is at least its index.
// Every CTA finds the limits for itself.
__global__ void __launch_bounds__(256)
sa_k_iterations(const uint64_t* P, const SaCallDesc* desc, SaSeedList cs, SaCounters* ctr) {
    sa_wait_prior();
    sa_allow_next();
    const uint64_t num_iter = ctr->num_iter;
    if (num_iter <= 1) return;
    __shared__ uint64_t limits[SA_MAX_ITERS];
    if (threadIdx.x == 0) {
        const uint64_t n = desc->num_seeds, MH = desc->max_hits;
        uint64_t lim = MH;
        int64_t prev = -1;
        for (uint64_t it = 0; it + 1 < num_iter; ++it) {
            uint64_t lo = 0, hi = n;  // first index with P >= lim
            while (lo < hi) {
                uint64_t mid = (lo + hi) >> 1;
                if (P[mid] < lim) lo = mid + 1;
                else hi = mid;
            }
            int64_t pos = (int64_t)lo - 1;
            if (pos <= prev) {
                atomicCAS(&ctr->error, 0ull, (unsigned long long)SA_DERR_MAX_HITS);
                pos = prev + 1;
            }
            limits[it] = (uint64_t)pos;
            lim = P[pos] + MH;
            prev = pos;
        }
        limits[num_iter - 1] = n ? n - 1 : 0;
    }
    __syncthreads();
    const uint64_t nnz = ctr->nnz;
    for (uint64_t c = blockIdx.x * 256ull + threadIdx.x; c < nnz; c += gridDim.x * 256ull) {
        const uint32_t s = cs.scope[c];
        uint32_t g = 0;
        while (g + 1 < num_iter && (uint64_t)s > limits[g]) ++g;
        cs.scope[c] = g;
    }
}

void sa_launch_lookup_seeds(SaWork& w, const uint32_t* index, uint32_t nbuckets, const SaParams& p, int G,
                            cudaStream_t st, bool chain) {
    sa_k_lookup_count<<<G, SA_CALL_BLOCK, 0, st>>>(w.seeds, w.desc, index, nbuckets, w.s_lo, w.s_cnt, w.cta_a, w.cta_b, w.ctr,
                                         w.units, p, chain ? 1 : 0, sa_hash_max_slots(w));
    sa_note_launch();
    sa_launch_next(sa_k_lookup_emit, G, SA_CALL_BLOCK, st, w.seeds, w.desc, w.s_lo, w.s_cnt, w.s_P, w.cs, w.cta_a,
                   w.cta_b, w.ctr);
    sa_note_launch();
    sa_launch_next(sa_k_iterations, 148, 256, st, w.s_P, w.desc, w.cs, w.ctr);
    sa_note_launch();
}

// ---------------------------------------------------------------------------
// Batched lookup over "seed slots".  Unit u covers query positions
// [q_start, q_end) of one strand; each position owns S = 1 (+K with
// transitions) consecutive slots in the order the host seeder emits seed
// words (key, then key ^ (2 << 2t), t = 0..K-1).  Positions whose window is
// not all uppercase ACGT produce no seed in the reference; here their slots
// simply have no hits, which leaves every hit and its MAX_HITS iteration
// unchanged (iterations are defined by the hit prefix only).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t sa_find_unit(const SaBatchUnit* __restrict__ bu, uint32_t n, uint64_t slot) {
    uint32_t lo = 0, hi = n;  // last unit with slot_begin <= slot
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (bu[mid].slot_begin <= slot) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The unit holding slot s, kept per thread: a thread's slots only increase,
// so the binary search runs only when s passes the current unit's end.
struct SaUnitCursor {
    uint32_t u = 0;
    uint64_t end = 0;  // one past the unit's last slot (0: not located yet)
    SaBatchUnit B{};
    __device__ __forceinline__ void seek(const SaBatchUnit* __restrict__ bu, uint32_t nu, uint64_t n, uint64_t s) {
        if (s < end) return;
        u = sa_find_unit(bu, nu, s);
        B = bu[u];
        end = (u + 1 < nu) ? bu[u + 1].slot_begin : n;
    }
};

// Per CTA: hits and hit-bearing slots of its range.  A thread takes
// SA_COUNT_ITEMS slots 256 apart per round and issues all their key loads,
// then all their bucket-bound loads, then the stores (the loads of one round
// are in flight together).
#define SA_COUNT_ITEMS 4
__global__ void __launch_bounds__(256)
sa_k_blookup_count(const SaBatchUnit* __restrict__ bu, const SaCallDesc* __restrict__ desc,
                   const uint32_t* __restrict__ index, uint32_t nbuckets, int S,
                   uint32_t* __restrict__ s_lo, uint32_t* __restrict__ s_cnt, unsigned long long* cta_a,
                   unsigned long long* cta_b, SaCounters* ctr) {
    constexpr int J = SA_COUNT_ITEMS;
    const uint64_t n = desc->num_seeds;
    uint64_t a, b;
    sa_cta_range(n, a, b);
    const uint32_t nu = desc->num_units;
    unsigned long long hits = 0, nz = 0;
    bool bad_key = false;
    SaUnitCursor cur;
    for (uint64_t s0 = a + threadIdx.x; s0 < b; s0 += 256 * J) {
        uint32_t key[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const uint64_t s = s0 + 256ull * j;
            key[j] = SA_INVALID_KEY;
            if (s < b) {
                cur.seek(bu, nu, n, s);
                const SaBatchUnit& B = cur.B;
                const uint64_t off = s - B.slot_begin;
                // find_num_hits (src/seed_filter.cu:129-154) on a call's own words; a key
                // outside the table is reported (a plain call's SA_ERR_BAD_SEED), never read
                if (B.seeds) {
                    const uint32_t k = (uint32_t)(__ldg(reinterpret_cast<const unsigned long long*>(B.seeds) +
                                                        B.q_start + off) >> 32);
                    if (k >= nbuckets) bad_key = true;
                    else key[j] = k;
                } else {
                    const uint32_t v = (uint32_t)(off % S);
                    const uint32_t k = __ldg(B.keys + B.q_start + (uint32_t)(off / S));
                    key[j] = (k == SA_INVALID_KEY || !v) ? k : k ^ (2u << (2 * (v - 1)));
                }
            }
        }
        uint32_t lo[J], hi[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            lo[j] = hi[j] = 0;
            if (key[j] < nbuckets) {
                hi[j] = __ldg(index + key[j]);
                lo[j] = key[j] ? __ldg(index + key[j] - 1) : 0u;
            }
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const uint64_t s = s0 + 256ull * j;
            if (s < b) {
                const uint32_t c = hi[j] - lo[j];
                s_lo[s] = lo[j];
                s_cnt[s] = c;
                hits += c;
                nz += c != 0;
            }
        }
    }
    if (bad_key) atomicCAS(&ctr->error, 0ull, (unsigned long long)SA_DERR_BAD_KEY);
    __shared__ unsigned long long ws[9];
    unsigned long long tot;
    sa_block_excl_sum<unsigned long long, 256>(hits, ws, &tot);
    if (threadIdx.x == 0) cta_a[blockIdx.x] = tot;
    sa_block_excl_sum<unsigned long long, 256>(nz, ws, &tot);
    if (threadIdx.x == 0) cta_b[blockIdx.x] = tot;
}

// Compaction of hit-bearing slots; also records each unit's hit range
// [unit_hit_base, unit_hit_end) in the global hit prefix.  A round covers
// 256 x SA_EMIT_ITEMS consecutive slots, SA_EMIT_ITEMS per thread, with one
// block scan of the packed (hits << 16 | hit-bearing slots) per round (a
// round has at most 2^12 hit-bearing slots, so the low field never carries).
#define SA_EMIT_ITEMS 4
__global__ void __launch_bounds__(256)
sa_k_blookup_emit(const SaBatchUnit* __restrict__ bu, const SaCallDesc* __restrict__ desc, int S,
                  const uint32_t* __restrict__ s_lo, const uint32_t* __restrict__ s_cnt, SaSeedList cs,
                  const unsigned long long* cta_a, const unsigned long long* cta_b, unsigned long long* unit_hit_base,
                  unsigned long long* unit_hit_end, SaCounters* ctr) {
    static_assert(256 * SA_EMIT_ITEMS < (1 << 16), "packed scan field");
    const uint64_t n = desc->num_seeds;
    const uint32_t nu = desc->num_units;
    uint64_t a, b;
    sa_cta_range(n, a, b);
    unsigned long long hbase = cta_a[blockIdx.x], cbase = cta_b[blockIdx.x];
    __shared__ unsigned long long ws[9];
    SaUnitCursor cur;
    // each round's counts and bucket starts are loaded during the round before
    uint32_t cnt[SA_EMIT_ITEMS], lo[SA_EMIT_ITEMS];
    auto fetch = [&](uint64_t r, uint32_t* c, uint32_t* l) {
        const uint64_t s0 = r + (uint64_t)threadIdx.x * SA_EMIT_ITEMS;
#pragma unroll
        for (int k = 0; k < SA_EMIT_ITEMS; ++k) {
            const bool in = s0 + k < b;
            c[k] = in ? s_cnt[s0 + k] : 0u;
            l[k] = in ? s_lo[s0 + k] : 0u;
        }
    };
    fetch(a, cnt, lo);
    for (uint64_t r = a; r < b; r += 256 * SA_EMIT_ITEMS) {
        const uint64_t s0 = r + (uint64_t)threadIdx.x * SA_EMIT_ITEMS;
        uint32_t ncnt[SA_EMIT_ITEMS], nlo[SA_EMIT_ITEMS];
        fetch(r + 256 * SA_EMIT_ITEMS, ncnt, nlo);
        unsigned long long mine = 0;
#pragma unroll
        for (int k = 0; k < SA_EMIT_ITEMS; ++k) mine += ((unsigned long long)cnt[k] << 16) | (cnt[k] != 0);
        unsigned long long tot;
        const unsigned long long e = sa_block_excl_sum<unsigned long long, 256>(mine, ws, &tot);
        unsigned long long eh = hbase + (e >> 16), ec = cbase + (e & 0xffffu);
#pragma unroll
        for (int k = 0; k < SA_EMIT_ITEMS; ++k) {
            const uint64_t s = s0 + k;
            if (s < b) {
                cur.seek(bu, nu, n, s);
                const SaBatchUnit& B = cur.B;
                if (s == B.slot_begin) unit_hit_base[cur.u] = eh;
                if (s + 1 == cur.end) unit_hit_end[cur.u] = eh + cnt[k];
                if (cnt[k]) {
                    cs.E[ec] = eh;
                    cs.lo[ec] = lo[k];
                    cs.qpos[ec] = B.seeds ? (uint32_t)__ldg(reinterpret_cast<const unsigned long long*>(B.seeds) +
                                                            B.q_start + (s - B.slot_begin))
                                          : B.q_start + (uint32_t)((s - B.slot_begin) / S);
                    cs.unit[ec] = B.unit;
                    cs.scope[ec] = cur.u << 4;  // (batch unit, iteration 0); sa_k_bscope sets later iterations
                    ++ec;
                }
                eh += cnt[k];
            }
        }
        hbase += tot >> 16;
        cbase += tot & 0xffffu;
#pragma unroll
        for (int k = 0; k < SA_EMIT_ITEMS; ++k) {
            cnt[k] = ncnt[k];
            lo[k] = nlo[k];
        }
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) cs.E[ctr->nnz] = ctr->num_hits;
}

// Per unit: MAX_HITS iteration boundaries in hit space (relative to the unit's
// first hit).  The reference's limit_pos[i] = lower_bound(P, lim) - 1 selects
// the last seed whose inclusive prefix is < lim; its prefix is the boundary.
__global__ void sa_k_bgroups(const SaCallDesc* __restrict__ desc, SaSeedList cs,
                             const unsigned long long* __restrict__ unit_hit_base,
                             const unsigned long long* __restrict__ unit_hit_end, unsigned long long* bounds,
                             uint32_t* unit_iters, SaCounters* ctr) {
    const uint32_t nu = desc->num_units;
    const uint64_t MH = desc->max_hits, nnz = ctr->nnz;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < nu; u += gridDim.x * blockDim.x) {
        const uint64_t base = unit_hit_base[u], H = unit_hit_end[u] - base;
        uint64_t it = MH ? H / MH + 1 : 1;
        if (it > SA_BATCH_ITERS) {
            atomicCAS(&ctr->error, 0ull, 3ull);
            it = 1;
        }
        unit_iters[u] = (uint32_t)it;
        if (it > 1) ctr->chain_bad = 1;  // its hits are deduplicated per iteration
        unsigned long long* B = bounds + (uint64_t)u * SA_BATCH_ITERS;
        if (it > 1) {
            // compacted seeds of the unit: c with base <= E[c] < base + H
            uint64_t lo = 0, hi = nnz;
            while (lo < hi) {
                uint64_t m = (lo + hi) >> 1;
                if (cs.E[m] < base) lo = m + 1;
                else hi = m;
            }
            const uint64_t c0 = lo;
            hi = nnz;
            while (lo < hi) {
                uint64_t m = (lo + hi) >> 1;
                if (cs.E[m] < base + H) lo = m + 1;
                else hi = m;
            }
            const uint64_t c1 = lo;
            uint64_t lim = MH, prev_bound = 0;
            for (uint64_t i = 0; i + 1 < it; ++i) {
                // last c in [c0, c1) with inclusive prefix E[c+1] - base < lim
                uint64_t l = c0, h = c1;
                while (l < h) {
                    uint64_t m = (l + h) >> 1;
                    if (cs.E[m + 1] - base < lim) l = m + 1;
                    else h = m;
                }
                uint64_t bnd = (l > c0) ? cs.E[l] - base : 0;  // prefix of the last qualifying seed
                if (l == c0 || bnd <= prev_bound) {
                    if (i > 0 || l == c0) atomicCAS(&ctr->error, 0ull, 2ull);
                }
                B[i] = bnd;
                prev_bound = bnd;
                lim = bnd + MH;
            }
        }
        B[it - 1] = ~0ull;
    }
}

// Compacted seed -> scope = (batch unit << 4) | iteration, for the units with
// more than one MAX_HITS iteration (the emit wrote iteration 0).  One CTA per
// such unit: its compacted seeds are those with E in [base, base + H).
__global__ void __launch_bounds__(256)
sa_k_bscope(const SaCallDesc* __restrict__ desc, SaSeedList cs, const unsigned long long* __restrict__ unit_hit_base,
            const unsigned long long* __restrict__ unit_hit_end, const unsigned long long* __restrict__ bounds,
            const uint32_t* __restrict__ unit_iters, SaCounters* ctr) {
    const uint32_t nu = desc->num_units;
    const uint64_t nnz = ctr->nnz;
    for (uint32_t u = blockIdx.x; u < nu; u += gridDim.x) {
        const uint32_t it = unit_iters[u];
        if (it <= 1) continue;
        const uint64_t base = unit_hit_base[u], H = unit_hit_end[u] - base;
        uint64_t lo = 0, hi = nnz;
        while (lo < hi) {
            const uint64_t m = (lo + hi) >> 1;
            if (cs.E[m] < base) lo = m + 1;
            else hi = m;
        }
        const uint64_t c0 = lo;
        hi = nnz;
        while (lo < hi) {
            const uint64_t m = (lo + hi) >> 1;
            if (cs.E[m] < base + H) lo = m + 1;
            else hi = m;
        }
        const unsigned long long* B = bounds + (uint64_t)u * SA_BATCH_ITERS;
        for (uint64_t c = c0 + threadIdx.x; c < lo; c += blockDim.x) {
            const uint64_t p = cs.E[c + 1] - base;
            uint32_t g = 0;
            while (g + 1 < it && p > B[g]) ++g;
            cs.scope[c] = (u << 4) | g;
        }
    }
}

void sa_launch_lookup_batch(SaWork& w, const uint32_t* index, uint32_t nbuckets, uint32_t n_bunits, const SaParams& p,
                            int G, cudaStream_t st) {
    const int S = p.transition ? 1 + p.kmer_size : 1;
    // a unit without slots (an empty window) gets the empty hit range [0, 0)
    cudaMemsetAsync(w.unit_hit_base, 0, 8ull * n_bunits, st);
    cudaMemsetAsync(w.unit_hit_end, 0, 8ull * n_bunits, st);
    sa_k_blookup_count<<<G, 256, 0, st>>>(w.bunits, w.desc, index, nbuckets, S, w.s_lo, w.s_cnt, w.cta_a, w.cta_b,
                                          w.ctr);
    sa_note_launch();
    sa_k_scan_partials<<<1, 1024, 0, st>>>(w.cta_a, w.cta_b, G, &w.ctr->num_hits, &w.ctr->nnz);
    sa_note_launch();
    sa_k_blookup_emit<<<G, 256, 0, st>>>(w.bunits, w.desc, S, w.s_lo, w.s_cnt, w.cs, w.cta_a, w.cta_b,
                                         w.unit_hit_base, w.unit_hit_end, w.ctr);
    sa_note_launch();
    const int ub = (int)std::min<uint32_t>((n_bunits + 255) / 256, 1024u);
    sa_k_bgroups<<<ub > 0 ? ub : 1, 256, 0, st>>>(w.desc, w.cs, w.unit_hit_base, w.unit_hit_end, w.bounds,
                                                  w.unit_iters, w.ctr);
    sa_note_launch();
    sa_k_bscope<<<(int)std::min<uint32_t>(std::max<uint32_t>(n_bunits, 1u), 1024u), 256, 0, st>>>(w.desc, w.cs, w.unit_hit_base, w.unit_hit_end,
                                                                      w.bounds, w.unit_iters, w.ctr);
    sa_note_launch();
}
