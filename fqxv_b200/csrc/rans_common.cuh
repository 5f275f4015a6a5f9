// Warp-level helpers shared by the encode and decode kernels.
#pragma once

#include <stdint.h>

namespace fqxv {

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Inclusive warp scan of u32.
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

__device__ __forceinline__ uint64_t warp_incl_scan_u64(uint64_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint64_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

__device__ __forceinline__ uint32_t ld_u32_le(const uint8_t *p) {
    return (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
}

__device__ __forceinline__ uint64_t ld_u64_le(const uint8_t *p) {
    uint64_t v = 0;
#pragma unroll
    for (int i = 7; i >= 0; i--) v = (v << 8) | p[i];
    return v;
}

// ---- encode table entries ---------------------------------------------------
// The map of a state v below x_max = f << 20 (model.rs:125-133),
//   x' = (v / f) 4096 + v % f + cum = v + cum + q (4096 - f),  q = v / f,
// without a correction step: q is exact from one multiplication,
//   q = hi32(v m + b m) >> s, b = 0 or 1.
// For f not a power of two and 2^s < f: with m = ceil(2^(32+s) / f), b = 0
// the product overshoots v / f by v (m f - 2^(32+s)) / (f 2^(32+s)), less
// than the 1 / f it has to stay below, as v < 2^20 f, whenever f (m f -
// 2^(32+s)) <= 2^(12+s) -- always for f < 2048; where it does not hold, the
// floor with b = 1 does (its own remainder is then the smaller). A power of
// two 2^k, k > 0, is m = 2^31, s = k - 1, and f = 1 takes q = v - 1 (m = 2^32
// - 1, v > 0) with 4095 added to cum.
// In the table arena an entry is 8 bytes:
//   .m   m
//   .y   (f - 1) << 20 | (cum, plus 4095 for f = 1) << 7 | b << 5 | s;
//        0 for an absent symbol (no present one has 0).
struct EncEntry {
    uint32_t m, y;
};
__host__ __device__ inline EncEntry enc_entry_of(uint32_t f, uint32_t cum) {
    if (f == 0) return {0u, 0u};
    if (f == 1) return {0xffffffffu, (cum + 4095u) << 7};
#ifdef __CUDA_ARCH__
    const uint32_t s = 31u - (uint32_t)__clz((int)f);  // 2^s <= f < 2^(s+1)
#else
    uint32_t s = 0;
    while ((2u << s) <= f) s++;
#endif
    if (f == 1u << s) return {0x80000000u, (f - 1u) << 20 | cum << 7 | (s - 1u)};
    // 2^(32+s) = m f + r by 32-bit divisions: 2^32 = q f + r0 first
    const uint32_t q = 0xffffffffu / f, r0 = 0xffffffffu - q * f + 1u;
    const uint32_t t = (r0 << s) / f, r = (r0 << s) - t * f;
    const uint32_t m = (q << s) + t, over = f - r;
    const uint32_t b = f * over <= 4096u << s ? 0u : 1u;
    return {m + 1u - b, (f - 1u) << 20 | cum << 7 | b << 5 | s};
}
// Frequency of an entry (0: absent).
__host__ __device__ inline uint32_t enc_freq(uint32_t y) { return y ? (y >> 20) + 1u : 0u; }

// The entry as the state's step takes it: a chain warp spends its time
// issuing instructions, and this form leaves three to unpack it.
struct EncStep {
    uint32_t m;
    uint32_t keep;  // largest state that keeps its low 16 bits, (f << 20) - 1
    uint32_t pack;  // (cum, plus 4095 for f = 1) << 17 | (4096 - f) << 5 | s
    uint32_t bias;  // b m
};
__host__ __device__ inline EncStep enc_unpack(uint32_t m, uint32_t y) {
    return {m, y | 0xfffffu, ((y >> 7) & 0x1fffu) << 17 | (4095u - (y >> 20)) << 5 | (y & 31u), (y >> 5) & 1u ? m : 0u};
}
__host__ __device__ inline uint32_t enc_map(uint32_t v, const EncStep &e) {
    const uint32_t hi = (uint32_t)(((uint64_t)v * e.m + e.bias) >> 32);
#ifdef __CUDA_ARCH__
    const uint32_t q = __funnelshift_r(hi, 0u, e.pack);  // by e.pack modulo 32: s
#else
    const uint32_t q = hi >> (e.pack & 31u);
#endif
    return v + (e.pack >> 17) + q * ((e.pack >> 5) & 0xfffu);
}

// ---- the encoder's symbol chunks ---------------------------------------------
// A block of n elements of `size` bytes at address `first` has n / 32 whole
// rounds. The encoder walks them from the last to the first in chunks of
// kEncChunk rounds, which it copies in aligned granules of 16 bytes; the rounds
// below the chunks it reads element by element. No granule reaches outside the
// block: where the lowest whole chunk has no round below it to hold its first
// granule's lower part, it is left to the rounds below (tail 16), and of the
// last granule only the part in the block is copied.
constexpr int kEncChunk = 16;
struct SymbolPlan {
    uint64_t top;     // address of the first granule of chunk 0, the highest
    uint32_t mis;     // bytes of it that lie below the chunk, the same for every chunk
    uint32_t behind;  // bytes to copy of the granule that holds chunk 0's last `mis` bytes
    int64_t chunks;   // chunks, each kEncChunk * 32 * size bytes below the one before
    int64_t tail;     // rounds below them, 0 to kEncChunk
};
__host__ __device__ inline SymbolPlan symbol_plan(uint64_t first, uint64_t n, uint32_t size) {
    const int64_t full = (int64_t)(n / 32);
    SymbolPlan p;
    p.top = first + (uint64_t)((full - kEncChunk) * 32) * size;
    p.mis = (uint32_t)(p.top & 15u);
    p.top -= p.mis;
    const uint32_t in_block = p.mis + (uint32_t)(n % 32) * size;
    p.behind = in_block < 16u ? in_block : 16u;
    p.chunks = full / kEncChunk;
    if (p.mis && full && p.chunks * kEncChunk == full) p.chunks--;
    p.tail = full - p.chunks * kEncChunk;
    return p;
}

// ---- runs of fast decode rounds ---------------------------------------------
// Groups of G rounds, from round r on, that need no check of the words left:
// all their symbols are there (below round full), and their words (32 a round
// at most), with the 64 that a decoder's window may look ahead, end before
// navail. A run follows its word position in 32 bits, so it takes 2^31 words
// at most.
constexpr int64_t kRunRounds = (int64_t)1 << 26;
template <int G>
__host__ __device__ __forceinline__ int64_t fast_groups(uint64_t navail, uint64_t wp, uint64_t full, uint64_t r) {
    const int64_t spare = (int64_t)navail - (int64_t)wp - 64;
    int64_t groups = spare > 0 ? spare / (32 * G) : 0;
    const int64_t left = r < full ? (int64_t)(full - r) / G : 0;
    if (groups > left) groups = left;
    if (groups > kRunRounds / G) groups = kRunRounds / G;
    return groups;
}

// Normalise m (<= 256) counts, held in ascending symbol order, into
// frequencies summing to 4096 with the reference's rounding and tie rules
// (crates/fqxv-rans/src/model.rs:213-264):
//   f = max(1, c * 4096 / total) for every occurring symbol;
//   max_s = first symbol with the strictly largest f;
//   a positive residual goes to max_s; a negative one drains max_s down to 1,
//   then re-picks the first symbol with the strictly largest f > 1, repeating.
// One warp; lane l owns entries [8l, 8l + 8). Also returns the exclusive
// cumulative frequency of each entry. `present` is false for an all-zero row.
__device__ __forceinline__ void warp_normalize(const uint32_t *counts, int m, uint32_t f[8],
                                               uint32_t cum[8], bool &present) {
    const int lane = threadIdx.x & 31;
    uint32_t c[8];
    uint64_t tot = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int idx = lane * 8 + k;
        c[k] = idx < m ? counts[idx] : 0u;
        tot += c[k];
    }
    tot = warp_sum_u64(tot);
    present = tot != 0;
    if (!present) {
#pragma unroll
        for (int k = 0; k < 8; k++) f[k] = cum[k] = 0;
        return;
    }
    uint32_t sum = 0, key = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint32_t idx = lane * 8 + k;
        uint32_t v = 0;
        if (c[k]) {
            v = (uint32_t)(((uint64_t)c[k] * 4096u) / tot);
            if (v == 0) v = 1;
        }
        f[k] = v;
        sum += v;
        const uint32_t kk = v ? (v << 9) | (511u - idx) : 0u;
        key = kk > key ? kk : key;
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    key = __reduce_max_sync(0xffffffffu, key);
    int max_s = 511 - (int)(key & 511u);
    int diff = 4096 - (int)sum;
    if (diff > 0) {
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (lane * 8 + k == max_s) f[k] += (uint32_t)diff;
    } else {
        // At most one pass per occurring symbol; the guard only bounds the loop.
        for (int iter = 0; diff < 0 && iter < 512; iter++) {
            uint32_t take = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                if (lane * 8 + k == max_s) {
                    take = f[k] - 1u;
                    if (take > (uint32_t)(-diff)) take = (uint32_t)(-diff);
                    f[k] -= take;
                }
            }
            take = __reduce_add_sync(0xffffffffu, take);
            diff += (int)take;
            if (diff != 0) {
                key = 0;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const uint32_t idx = lane * 8 + k;
                    const uint32_t kk = f[k] > 1u ? (f[k] << 9) | (511u - idx) : 0u;
                    key = kk > key ? kk : key;
                }
                key = __reduce_max_sync(0xffffffffu, key);
                if (key == 0) break;
                max_s = 511 - (int)(key & 511u);
            }
        }
    }
    uint32_t local = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        cum[k] = local;
        local += f[k];
    }
    const uint32_t excl = warp_incl_scan(local) - local;
#pragma unroll
    for (int k = 0; k < 8; k++) cum[k] += excl;
}

}  // namespace fqxv
