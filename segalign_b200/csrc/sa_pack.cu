// sa_pack.cu — sequence packing, reverse complement, target seed-position
// table build on the device, and the shared scan kernels.
//
// Reference behaviour restated here:
//   compress_string            common/seed_filter_interface.cu:18-47
//   compress_string_rev_comp   src/seed_filter.cu:82-127
//   rev_comp_string (rm)       repeat_masker_src/seed_filter.cu:137-167
//   GenerateSeedPosTable       common/seed_pos_table.cu:49-109 (CPU in the reference)
#include <cstdio>

#include "sa_launch.h"
#include "sa_radix.cuh"

// ---------------------------------------------------------------------------
// Scans shared by the range-partitioned kernels
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024)
sa_k_scan_partials(unsigned long long* a, unsigned long long* b, int G, unsigned long long* ta,
                   unsigned long long* tb) {
    __shared__ unsigned long long ws[33];
    const int t = threadIdx.x;
    unsigned long long va = t < G ? a[t] : 0ull, vb = t < G ? b[t] : 0ull, tot;
    unsigned long long ea = sa_block_excl_sum<unsigned long long, 1024>(va, ws, &tot);
    if (t == 0 && ta) *ta = tot;
    unsigned long long eb = sa_block_excl_sum<unsigned long long, 1024>(vb, ws, &tot);
    if (t == 0 && tb) *tb = tot;
    if (t < G) {
        a[t] = ea;
        b[t] = eb;
    }
}

// One CTA per digit: its row of the bin-major histogram [256][A] becomes
// exclusive prefixes within the digit; the row's sum goes to hist[256 * A + digit].
// (One CTA for the whole histogram took 78 us at 592 active CTAs.)
__global__ void __launch_bounds__(256)
sa_k_radix_scan(unsigned int* hist, int G, const unsigned long long* d_n) {
    __shared__ unsigned int ws[9];
    const uint32_t A = sa_radix_active(*d_n, (uint32_t)G);
    unsigned int* const row = hist + (uint64_t)blockIdx.x * A;
    unsigned int carry = 0;
    for (uint32_t i0 = 0; i0 < A; i0 += 256) {
        const uint32_t i = i0 + threadIdx.x;
        const unsigned int v = i < A ? row[i] : 0u;
        unsigned int tot;
        const unsigned int e = sa_block_excl_sum<unsigned int, 256>(v, ws, &tot);
        if (i < A) row[i] = carry + e;
        carry += tot;
    }
    if (threadIdx.x == 0) hist[256ull * A + blockIdx.x] = carry;
}

// ---------------------------------------------------------------------------
// Packing
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t sa_char_code(uint8_t ch) {
    // common/seed_filter_interface.cu:28-46
    switch (ch) {
        case 'A': return 0;
        case 'C': return 1;
        case 'G': return 2;
        case 'T': return 3;
        case 'a': case 'c': case 'g': case 't': return 4;
        case 'n': case 'N': return 5;
        case '&': return 7;
        default: return 6;
    }
}

// One thread per output word: 8 text bytes -> 8 nibbles; bases past `len` are E.
__global__ void sa_k_pack_text(const uint8_t* __restrict__ text, uint64_t len, uint32_t* __restrict__ out,
                               uint64_t nwords) {
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwords;
         w += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t b = w * 8;
        uint32_t word = 0;
        if (b + 8 <= len) {
            uint2 v = *reinterpret_cast<const uint2*>(text + b);
#pragma unroll
            for (int k = 0; k < 4; ++k) word |= sa_char_code((v.x >> (8 * k)) & 0xff) << (4 * k);
#pragma unroll
            for (int k = 0; k < 4; ++k) word |= sa_char_code((v.y >> (8 * k)) & 0xff) << (4 * (k + 4));
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) word |= (b + k < len ? sa_char_code(text[b + k]) : 7u) << (4 * k);
        }
        out[w] = word;
    }
}

// Reversed copy of a packed sequence: out[i] = in[len-1-i]; with COMP the
// codes 0..3 are complemented as well (reverse complement, A<->T, C<->G;
// L/N/X/E unchanged; src/seed_filter.cu:96-125).  Bases past len are E.
template <bool COMP>
__global__ void sa_k_reverse_packed(const uint32_t* __restrict__ in, uint64_t len, uint32_t* __restrict__ out,
                                    uint64_t nwords) {
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwords;
         w += (uint64_t)gridDim.x * blockDim.x) {
        // output bases 8w..8w+7 come from in[len-1-8w-k]; load in[len-8w-8 .. len-8w)
        int64_t p = (int64_t)len - (int64_t)(8 * w) - 8;
        uint32_t x = sa_load8(in, p);
        // reverse nibble order
        x = __byte_perm(x, 0, 0x0123);
        x = ((x >> 4) & 0x0f0f0f0fu) | ((x & 0x0f0f0f0fu) << 4);
        if (COMP) {
            // complement codes 0..3 (bit 2 clear) by xor 3
            uint32_t m = (~(x >> 2)) & 0x11111111u;
            x ^= m * 3u;
        }
        uint64_t b = w * 8;
        if (b + 8 > len) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (b + k >= len) x = (x & ~(0xfu << (4 * k))) | (7u << (4 * k));
        }
        out[w] = x;
    }
}

__global__ void sa_k_fill_u32(uint32_t* p, uint64_t n, uint32_t v) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        p[i] = v;
}

void sa_launch_pack_text(const char* d_text, uint64_t len, uint32_t* packed, cudaStream_t st) {
    uint64_t nwords = (len + 7) / 8;
    if (!nwords) return;
    int blocks = (int)std::min<uint64_t>((nwords + 255) / 256, 148ull * 16);
    sa_k_pack_text<<<blocks, 256, 0, st>>>((const uint8_t*)d_text, len, packed, nwords);
    sa_note_launch();
}

void sa_launch_reverse_packed(const uint32_t* in, uint64_t len, uint32_t* out, bool complement, cudaStream_t st) {
    uint64_t nwords = (len + 7) / 8;
    if (!nwords) return;
    int blocks = (int)std::min<uint64_t>((nwords + 255) / 256, 148ull * 16);
    if (complement) sa_k_reverse_packed<true><<<blocks, 256, 0, st>>>(in, len, out, nwords);
    else sa_k_reverse_packed<false><<<blocks, 256, 0, st>>>(in, len, out, nwords);
    sa_note_launch();
}

void sa_launch_pad_fill(uint32_t* base, uint64_t n, cudaStream_t st) {
    if (!n) return;
    int blocks = (int)std::min<uint64_t>((n + 255) / 256, 148ull * 16);
    sa_k_fill_u32<<<blocks, 256, 0, st>>>(base, n, 0x77777777u);
    sa_note_launch();
}

// ---------------------------------------------------------------------------
// Table keys of target positions p = start + i * step (sa_window_key), in order
// ---------------------------------------------------------------------------
// Any step, pass 1: per-CTA count of the valid positions.
__global__ void __launch_bounds__(256)
sa_k_table_count(const uint32_t* __restrict__ ref, uint32_t start, uint64_t n, uint32_t step, SaParams P,
                 unsigned long long* cta_a) {
    uint64_t a, b;
    sa_cta_range(n, a, b);
    unsigned long long c = 0;
    for (uint64_t i = a + threadIdx.x; i < b; i += 256)
        c += sa_window_key(ref, (uint32_t)(start + i * step), P) != SA_INVALID_KEY;
    __shared__ unsigned long long ws[9];
    unsigned long long tot;
    sa_block_excl_sum<unsigned long long, 256>(c, ws, &tot);
    if (threadIdx.x == 0) cta_a[blockIdx.x] = tot;
}

// Any step, pass 2: ordered compaction of (key, position) pairs.
__global__ void __launch_bounds__(256)
sa_k_table_emit(const uint32_t* __restrict__ ref, uint32_t start, uint64_t n, uint32_t step, SaParams P,
                const unsigned long long* cta_a, uint32_t* keys, uint32_t* vals) {
    uint64_t a, b;
    sa_cta_range(n, a, b);
    unsigned long long base = cta_a[blockIdx.x];
    __shared__ unsigned long long ws[9];
    for (uint64_t r = a; r < b; r += 256) {
        uint64_t i = r + threadIdx.x;
        uint32_t key = SA_INVALID_KEY;
        uint32_t pos = start + (uint32_t)(i * step);
        if (i < b) key = sa_window_key(ref, (uint32_t)(start + i * step), P);
        unsigned long long v = key != SA_INVALID_KEY, tot;
        unsigned long long e = sa_block_excl_sum<unsigned long long, 256>(v, ws, &tot);
        if (v) {
            keys[base + e] = key;
            vals[base + e] = pos;
        }
        base += tot;
    }
}

// Keys of the windows that start at the 8 bases of word pw[0] (not checked for
// ACGT), from the five words that hold every base they reach (seed_size <= 32).
// For each shape position s in order (common/ntcoding.cpp:21-37) the word of
// bases s .. s + 7 gives the next 2-bit code of all 8 keys at once.
__device__ __forceinline__ void sa_keys8(const uint32_t* __restrict__ pw, const SaParams& P, uint32_t* key) {
    const uint32_t W0 = __ldg(pw), W1 = __ldg(pw + 1), W2 = __ldg(pw + 2), W3 = __ldg(pw + 3), W4 = __ldg(pw + 4);
#pragma unroll
    for (int k = 0; k < 8; ++k) key[k] = 0;
    for (int i = 0; i < P.kmer_size; ++i) {
        const uint32_t sp = (uint32_t)P.shape_pos[i], q = sp >> 3;
        const uint32_t a = q == 0 ? W0 : q == 1 ? W1 : q == 2 ? W2 : W3;
        const uint32_t b = q == 0 ? W1 : q == 1 ? W2 : q == 2 ? W3 : W4;
        const uint32_t win = __funnelshift_r(a, b, 4u * (sp & 7u));
#pragma unroll
        for (int k = 0; k < 8; ++k) key[k] = (key[k] << 2) | ((win >> (4 * k)) & 3u);
    }
}

// Step 1: a thread takes the 8 positions of one packed word.  Pass 1 counts the
// valid ones (no keys), pass 2 computes the 8 keys together (sa_keys8) and
// writes those.  20 Mbp: 164 + 248 us with a key per position and pass, each
// through local memory, 20 + 93 us now.
__device__ __forceinline__ uint32_t sa_table_valid8(const uint32_t* __restrict__ ref, uint64_t g, uint64_t p0, uint64_t p1,
                                                    uint32_t seed_size) {
    uint32_t ok = sa_valid_windows8(ref + g, seed_size);
    if (8 * g < p0) ok &= 0xffu << (p0 - 8 * g);
    if (8 * g + 8 > p1) ok &= 0xffu >> (8 * g + 8 - p1);
    return ok & 0xffu;
}

__global__ void __launch_bounds__(256)
sa_k_table_count8(const uint32_t* __restrict__ ref, uint64_t p0, uint64_t p1, uint32_t seed_size,
                  unsigned long long* cta_a) {
    uint64_t a, b;
    sa_cta_range(p1 > p0 ? ((p1 - 1) >> 3) - (p0 >> 3) + 1 : 0, a, b);
    unsigned long long c = 0;
    for (uint64_t g = (p0 >> 3) + a + threadIdx.x; g < (p0 >> 3) + b; g += 256)
        c += __popc(sa_table_valid8(ref, g, p0, p1, seed_size));
    __shared__ unsigned long long ws[9];
    unsigned long long tot;
    sa_block_excl_sum<unsigned long long, 256>(c, ws, &tot);
    if (threadIdx.x == 0) cta_a[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(256)
sa_k_table_emit8(const uint32_t* __restrict__ ref, uint64_t p0, uint64_t p1, SaParams P,
                 const unsigned long long* cta_a, uint32_t* keys, uint32_t* vals) {
    uint64_t a, b;
    sa_cta_range(p1 > p0 ? ((p1 - 1) >> 3) - (p0 >> 3) + 1 : 0, a, b);
    unsigned long long base = cta_a[blockIdx.x];
    __shared__ uint32_t ws[9];
    __shared__ uint32_t s_key[2048], s_pos[2048];  // a round's valid positions, to be written in whole lines
    for (uint64_t g0 = (p0 >> 3) + a; g0 < (p0 >> 3) + b; g0 += 256) {
        const uint64_t g = g0 + threadIdx.x;
        const uint32_t ok = g < (p0 >> 3) + b ? sa_table_valid8(ref, g, p0, p1, (uint32_t)P.seed_size) : 0u;
        uint32_t tot;
        uint32_t at = sa_block_excl_sum<uint32_t, 256>(__popc(ok), ws, &tot);
        if (ok) {
            uint32_t key[8];
            sa_keys8(ref + g, P, key);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (ok >> k & 1u) {
                    s_key[at] = key[k];
                    s_pos[at++] = (uint32_t)(8 * g + k);
                }
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < tot; i += 256) {
            keys[base + i] = s_key[i];
            vals[base + i] = s_pos[i];
        }
        base += tot;
        __syncthreads();
    }
}

void sa_launch_table_keys(const uint32_t* ref, uint32_t start, uint64_t num_steps, uint32_t step,
                          const SaParams& p, uint32_t* keys, uint32_t* vals, unsigned long long* cta_a,
                          unsigned long long* cta_b, unsigned long long* d_total, int G, cudaStream_t st) {
    if (step == 1) sa_k_table_count8<<<G, 256, 0, st>>>(ref, start, start + num_steps, (uint32_t)p.seed_size, cta_a);
    else sa_k_table_count<<<G, 256, 0, st>>>(ref, start, num_steps, step, p, cta_a);
    sa_note_launch();
    sa_k_scan_partials<<<1, 1024, 0, st>>>(cta_a, cta_b, G, d_total, nullptr);
    sa_note_launch();
    if (step == 1) sa_k_table_emit8<<<G, 256, 0, st>>>(ref, start, start + num_steps, p, cta_a, keys, vals);
    else sa_k_table_emit<<<G, 256, 0, st>>>(ref, start, num_steps, step, p, cta_a, keys, vals);
    sa_note_launch();
}

// index[k] = number of valid positions with key <= k (the shifted inclusive
// table the reference ships, common/seed_pos_table.cu:83,103): each sorted item
// i fills buckets [key_i, key_{i+1}) with i+1.  `index` must be zeroed first.
__global__ void sa_k_table_index(const uint32_t* __restrict__ keys, const unsigned long long* d_n,
                                 uint32_t* __restrict__ index, uint64_t nbuckets) {
    const uint64_t n = *d_n;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t k = keys[i];
        uint64_t nx = (i + 1 < n) ? keys[i + 1] : nbuckets;
        for (uint64_t bkt = k; bkt < nx; ++bkt) index[bkt] = (uint32_t)(i + 1);
    }
}

void sa_launch_table_index(const uint32_t* sorted_keys, const unsigned long long* d_n, uint32_t* index,
                           uint64_t nbuckets, cudaStream_t st) {
    cudaMemsetAsync(index, 0, nbuckets * sizeof(uint32_t), st);
    sa_k_table_index<<<148 * 8, 256, 0, st>>>(sorted_keys, d_n, index, nbuckets);
    sa_note_launch();
}

// ---------------------------------------------------------------------------
// (key, value) radix sort
// ---------------------------------------------------------------------------
struct SaKvOps {
    struct Ctx {
        uint32_t* k[2];
        uint32_t* v[2];
    };
    struct Pass {
        const uint32_t *k, *v;
        uint32_t *k_out, *v_out;
        uint32_t shift;
    };
    static __device__ __forceinline__ Pass pass_of(const Ctx& c, int pass) {
        if (pass & 1) return {c.k[1], c.v[1], c.k[0], c.v[0], 8u * (uint32_t)pass};
        return {c.k[0], c.v[0], c.k[1], c.v[1], 8u * (uint32_t)pass};
    }
    struct Item {
        uint32_t k, v;
    };
    static __device__ __forceinline__ Item load(const Pass& p, uint64_t i) { return {p.k[i], p.v[i]}; }
    static __device__ __forceinline__ uint32_t digit_of(const Pass& p, const Item& x) { return (x.k >> p.shift) & 0xffu; }
    static __device__ __forceinline__ void store(const Pass& p, const Item& x, uint32_t dst) {
        p.k_out[dst] = x.k;
        p.v_out[dst] = x.v;
    }
};

void sa_launch_sort_kv(uint32_t* keys, uint32_t* vals, uint32_t* keys_tmp, uint32_t* vals_tmp,
                       const unsigned long long* d_n, int bits, unsigned int* cta_hist, int G,
                       cudaStream_t st, int* result_in_tmp) {
    int passes = (bits + 7) / 8;
    SaKvOps::Ctx c;
    c.k[0] = keys;
    c.k[1] = keys_tmp;
    c.v[0] = vals;
    c.v[1] = vals_tmp;
    for (int p = 0; p < passes; ++p) {
        sa_k_radix_up<SaKvOps><<<G, SA_RADIX_BLOCK, 0, st>>>(c, p, d_n, cta_hist);
        sa_note_launch();
        sa_k_radix_scan<<<256, 256, 0, st>>>(cta_hist, G, d_n);
        sa_note_launch();
        sa_k_radix_down<SaKvOps><<<G, SA_RADIX_BLOCK, 0, st>>>(c, p, d_n, cta_hist);
        sa_note_launch();
    }
    *result_in_tmp = passes & 1;
}

// ---------------------------------------------------------------------------
// Spaced-seed key of every query position (device-side seeding, the work of
// src/seeder.cpp:57-74 without the host loop): keys[j] = key of the window at
// j, SA_INVALID_KEY unless all seed_size bases are uppercase ACGT.
// ---------------------------------------------------------------------------
//
// One thread takes the 8 positions of one packed word.
__global__ void __launch_bounds__(256)
sa_k_query_keys(const uint32_t* __restrict__ packed, uint64_t len, SaParams P, uint32_t* __restrict__ keys) {
    const uint64_t ngroups = (len + 7) / 8;
    for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < ngroups;
         g += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t* pw = packed + g;
        const uint32_t ok = sa_valid_windows8(pw, (uint32_t)P.seed_size);
        uint32_t key[8];
        sa_keys8(pw, P, key);
        const uint64_t p0 = 8 * g;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (p0 + k < len) keys[p0 + k] = (ok >> k & 1u) ? key[k] : SA_INVALID_KEY;
    }
}

void sa_launch_query_keys(const uint32_t* packed, uint64_t len, const SaParams& p, uint32_t* keys, cudaStream_t st) {
    if (!len) return;
    const uint64_t groups = (len + 7) / 8;
    int blocks = (int)std::min<uint64_t>((groups + 255) / 256, 148ull * 16);
    sa_k_query_keys<<<blocks, 256, 0, st>>>(packed, len, p, keys);
    sa_note_launch();
}
