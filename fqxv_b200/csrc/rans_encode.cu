// Encode path of the B200 rANS Nx16 coder.
//
// Stages (each one launch over the whole batch):
//   1. enc_model_kernel   a cluster of CTAs per block: order-0 histogram (warp-
//      private shared-memory atomics with run-length folding), exact
//      normalisation, encode tables; for order-1 the occurring bytes, then a
//      dense |U| x |U| pair histogram (whose column sums are the order-0
//      counts) and one normalised model per present context.
//   2. enc_run_kernel     two warps per (block, order) job taken from a device
//      work queue (jobs sorted largest first): lane l owns state l and walks
//      the rounds from the last to the first, emitting renorm words with a
//      ballot/popc compaction written back to front into a word scratch.
//   3. enc_select_scan    encoded sizes, order selection, exclusive scan.
//   4. enc_pack_kernel    eight CTAs per block: header, frequency tables, states
//      and words written to their compacted place in the output arena.
// Byte format and arithmetic follow crates/fqxv-rans/src/scalar.rs:29-140 and
// model.rs:52-264.
#include <cooperative_groups.h>
#include <mutex>

#include "../../include/fqxv_rans_gpu_testing.h"
#include "rans_common.cuh"
#include "rans_internal.cuh"

namespace fqxv {

namespace {

__device__ __forceinline__ void unpack16(const uint4 v, uint32_t b[16]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 16; k++) b[k] = (w[k >> 2] >> (8 * (k & 3))) & 0xffu;
}

// Visit positions [lo, hi) of the block p in 16-byte aligned vector chunks
// (one per thread per step) and in single bytes for the unaligned head and
// the tail. For every byte the visitor gets (previous byte or 0 at position
// 0, byte); runs of equal keys are folded into one shared-memory atomic.
template <class KeyFn, class AddFn, class EmitFn, class Emit16Fn>
__device__ __forceinline__ void histogram_pass(const uint8_t *__restrict__ p, uint64_t lo, uint64_t hi, KeyFn key,
                                               AddFn add, EmitFn emit, Emit16Fn emit16) {
    if (hi <= lo) return;
    const uint64_t n = hi - lo;
    const uint64_t mis = (uint64_t)(uintptr_t)(p + lo) & 15u;
    uint64_t head = mis ? 16 - mis : 0;
    if (head > n) head = n;
    const uint64_t body = (n - head) / 16;
    const uint64_t tail0 = lo + head + body * 16;
    for (uint64_t i = lo + threadIdx.x; i < lo + head; i += blockDim.x) {
        const uint32_t k = key(i ? p[i - 1] : 0u, p[i]);
        emit(i, k);
        add(k, 1u);
    }
    for (uint64_t i = tail0 + threadIdx.x; i < hi; i += blockDim.x) {
        const uint32_t k = key(i ? p[i - 1] : 0u, p[i]);
        emit(i, k);
        add(k, 1u);
    }
    for (uint64_t c = threadIdx.x; c < body; c += blockDim.x) {
        const uint64_t pos = lo + head + 16 * c;
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p + pos));
        uint32_t b[16];
        unpack16(v, b);
        uint32_t prev = pos ? (uint32_t)p[pos - 1] : 0u;
        uint32_t ks[16];
        uint32_t k0 = key(prev, b[0]);
        ks[0] = k0;
        uint32_t run = 1;
#pragma unroll
        for (int k = 1; k < 16; k++) {
            const uint32_t kk = key(b[k - 1], b[k]);
            ks[k] = kk;
            if (kk != k0) {
                add(k0, run);
                k0 = kk;
                run = 1;
            } else {
                run++;
            }
        }
        add(k0, run);
        emit16(pos, ks);
    }
}

// Marks the bytes that occur in positions [lo, hi) of p: plain byte stores,
// which lanes with the same or neighbouring symbols share, where a count
// takes an atomic per byte and serialises on equal ones (1 shared-memory
// wavefront per 32 bytes against 4).
__device__ __forceinline__ void seen_pass(const uint8_t *__restrict__ p, uint64_t lo, uint64_t hi,
                                          volatile uint8_t *seen) {
    if (hi <= lo) return;
    const uint64_t n = hi - lo;
    const uint64_t mis = (uint64_t)(uintptr_t)(p + lo) & 15u;
    uint64_t head = mis ? 16 - mis : 0;
    if (head > n) head = n;
    const uint64_t body = (n - head) / 16;
    for (uint64_t i = lo + threadIdx.x; i < lo + head; i += blockDim.x) seen[p[i]] = 1;
    for (uint64_t i = lo + head + body * 16 + threadIdx.x; i < hi; i += blockDim.x) seen[p[i]] = 1;
    const uint4 *q = reinterpret_cast<const uint4 *>(p + lo + head);
    for (uint64_t c = threadIdx.x; c < body; c += blockDim.x) {
        uint32_t b[16];
        unpack16(__ldg(q + c), b);
#pragma unroll
        for (int k = 0; k < 16; k++)
            if (k == 0 || b[k] != b[k - 1]) seen[b[k]] = 1;
    }
}

__device__ __forceinline__ uint2 enc_entry(uint32_t f, uint32_t cum) {
    const EncEntry e = enc_entry_of(f, cum);
    return make_uint2(e.m, e.y);
}

}  // namespace

// Model of one block per thread-block cluster of kModelCluster CTAs: every
// CTA histograms its slice of the block into its own shared memory and the
// slices are summed through distributed shared memory. Counts: scalar.rs:30-33
// (order-0) and :62-80 (order-1); normalisation: model.rs:213-264.
__global__ void __launch_bounds__(kModelThreads)
    enc_model_kernel(const uint8_t *__restrict__ src, EncBlock *__restrict__ blocks,
                     const uint32_t *__restrict__ order, int nblocks, uint8_t *__restrict__ tbl,
                     uint32_t *__restrict__ hist_scratch, uint16_t *__restrict__ keys) {
    namespace cg = cooperative_groups;
    constexpr int W = kModelThreads / 32;
    constexpr int kSmemU = 64;
    __shared__ uint32_t h0[W][256];
    __shared__ uint32_t h1[kSmemU * kSmemU];
    __shared__ uint32_t part[256];      // this CTA's order-0 counts
    __shared__ uint32_t cnt[256];       // the block's order-0 counts
    __shared__ uint32_t occurs[256];    // order-1: bytes of this CTA's slice
    __shared__ uint8_t seen[256];
    __shared__ uint32_t rowbuf[W][kSmemU];
    __shared__ uint8_t umap[256];
    __shared__ int s_nu, s_nctx;
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cid = blockIdx.x / C, ncl = gridDim.x / C;
    uint32_t *gh = hist_scratch + (size_t)cid * 65536;

    for (int bi = cid; bi < nblocks; bi += ncl) {
        const int b = order[bi];
        const uint8_t *p = src + blocks[b].src_off;
        const uint64_t n = blocks[b].n;
        const int mode = blocks[b].mode;
        uint8_t *T = tbl + blocks[b].tbl_off;
        const uint64_t lo = n * (uint64_t)rank / C, hi = n * (uint64_t)(rank + 1) / C;

        if (tid == 0) s_nctx = 0;
        // order-0 counts of this CTA's slice in `part`, then of the block in
        // `cnt`, and the order-0 table from them
        auto count_slice = [&] {
            for (int i = tid; i < W * 256; i += blockDim.x) (&h0[0][0])[i] = 0;
            __syncthreads();
            uint32_t *hw = h0[warp];
            histogram_pass(
                p, lo, hi, [](uint32_t, uint32_t c) { return c; },
                [&](uint32_t k, uint32_t r) { atomicAdd(&hw[k], r); }, [](uint64_t, uint32_t) {},
                [](uint64_t, const uint32_t *) {});
            __syncthreads();
            if (tid < 256) {
                uint32_t t = 0;
#pragma unroll
                for (int w = 0; w < W; w++) t += h0[w][tid];
                part[tid] = t;
            }
        };
        auto sum_slices = [&] {
            if (tid < 256) {
                uint32_t t = 0;
                for (int r = 0; r < C; r++) t += cl.map_shared_rank(part, r)[tid];
                cnt[tid] = t;
            }
            __syncthreads();
        };
        auto order0_table = [&] {
            if (rank != 0 || warp != 0) return;
            uint32_t f[8], cum[8];
            bool present;
            warp_normalize(cnt, 256, f, cum, present);
            uint2 *T0 = reinterpret_cast<uint2 *>(T + kTblO0);
#pragma unroll
            for (int k = 0; k < 8; k++) T0[lane * 8 + k] = enc_entry(f[k], cum[k]);
        };
        if (mode == FQXV_RANS_ORDER0) {
            count_slice();
            cl.sync();  // every slice's counts are in place
            sum_slices();
            order0_table();
            cl.sync();  // no CTA rewrites `part` while another still reads it
            continue;
        }

        // Order-1 (scalar.rs:62-80). U = occurring bytes plus context 0, in
        // ascending byte order; contexts and symbols share that dense index.
        // Every CTA derives the same map from the same marks.
        if (tid < 256) seen[tid] = 0;
        __syncthreads();
        seen_pass(p, lo, hi, seen);
        __syncthreads();
        if (tid < 256) occurs[tid] = seen[tid];
        cl.sync();
        if (tid < 256) {
            uint32_t t = 0;
            for (int r = 0; r < C; r++) t |= cl.map_shared_rank(occurs, r)[tid];
            seen[tid] = (uint8_t)t;
        }
        __syncthreads();
        if (warp == 0) {
            uint32_t flags = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int s = lane * 8 + k;
                if (seen[s] != 0 || s == 0) flags |= 1u << k;
            }
            const uint32_t c = __popc(flags);
            uint32_t base = warp_incl_scan(c) - c;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int s = lane * 8 + k;
                umap[s] = (flags >> k) & 1u ? (uint8_t)(base++) : (uint8_t)0xff;
            }
            if (lane == 31) s_nu = (int)(base);
        }
        __syncthreads();
        const int nu = s_nu;
        auto pair = [&](uint32_t prev, uint32_t c) { return (uint32_t)umap[prev] * nu + umap[c]; };
        // the order-1 table index of every position, for the encode (when
        // the caller gave scratch for it); indexed from src rounded down to
        // 16 bytes, so a 16-byte input chunk's indices are one aligned 32 B
        uint16_t *kb = keys ? keys + ((uintptr_t)src & 15u) + blocks[b].src_off : nullptr;
        auto emit = [&](uint64_t i, uint32_t k) {
            if (kb) kb[i] = (uint16_t)k;
        };
        auto emit16 = [&](uint64_t pos, const uint32_t *k) {
            if (!kb) return;
            uint4 *d = reinterpret_cast<uint4 *>(kb + pos);
            d[0] = make_uint4(k[0] | k[1] << 16, k[2] | k[3] << 16, k[4] | k[5] << 16, k[6] | k[7] << 16);
            d[1] = make_uint4(k[8] | k[9] << 16, k[10] | k[11] << 16, k[12] | k[13] << 16, k[14] | k[15] << 16);
        };
        uint2 *T1 = reinterpret_cast<uint2 *>(T + kTblO1);
        if (rank == 0 && tid < 256) T[kTblUmap + tid] = umap[tid];
        if (nu <= kSmemU) {
            // pair counts of this slice in shared memory, rows summed over
            // the cluster; context rows are spread over all warps of it
            for (int i = tid; i < nu * nu; i += blockDim.x) h1[i] = 0;
            __syncthreads();
            histogram_pass(p, lo, hi, pair, [&](uint32_t k, uint32_t r) { atomicAdd(&h1[k], r); }, emit, emit16);
            // every position is counted in one pair, so a symbol's order-0
            // count is its column's sum
            if (mode != FQXV_RANS_ORDER1) {
                __syncthreads();
                if (tid < 256) {
                    const uint32_t u = umap[tid];
                    uint32_t t = 0;
                    if (u != 0xffu)
                        for (int r = 0; r < nu; r++) t += h1[r * nu + u];
                    part[tid] = t;
                }
            }
            cl.sync();
            if (mode != FQXV_RANS_ORDER1) {
                sum_slices();
                order0_table();
            }
            for (int t = warp + W * rank; t < nu; t += W * C) {
                for (int u = lane; u < nu; u += 32) {
                    uint32_t v = 0;
                    for (int r = 0; r < C; r++) v += cl.map_shared_rank(h1, r)[t * nu + u];
                    rowbuf[warp][u] = v;
                }
                __syncwarp();
                uint32_t f[8], cum[8];
                bool present;
                warp_normalize(rowbuf[warp], nu, f, cum, present);
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const int u = lane * 8 + k;
                    if (u < nu) T1[(size_t)t * nu + u] = enc_entry(f[k], cum[k]);
                }
                if (lane == 0 && present) atomicAdd(&s_nctx, 1);
                __syncwarp();
            }
        } else {
            if (mode != FQXV_RANS_ORDER1) {
                count_slice();
                cl.sync();
                sum_slices();
                order0_table();
            }
            // large alphabets: the cluster's first CTA counts the whole block
            // in global scratch
            if (rank == 0) {
                for (int i = tid; i < nu * nu; i += blockDim.x) gh[i] = 0;
                __syncthreads();
                histogram_pass(p, 0, n, pair, [&](uint32_t k, uint32_t r) { atomicAdd(&gh[k], r); }, emit, emit16);
                __syncthreads();
                for (int t = warp; t < nu; t += W) {
                    uint32_t f[8], cum[8];
                    bool present;
                    warp_normalize(gh + (size_t)t * nu, nu, f, cum, present);
    #pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int u = lane * 8 + k;
                        if (u < nu) T1[(size_t)t * nu + u] = enc_entry(f[k], cum[k]);
                    }
                    if (lane == 0 && present) atomicAdd(&s_nctx, 1);
                }
            }
        }
        cl.sync();  // all rows done; s_nctx final in every CTA
        if (rank == 0 && tid == 0) {
            int k = 0;
            for (int r = 0; r < C; r++) k += *cl.map_shared_rank(&s_nctx, r);
            blocks[b].nu = nu;
            blocks[b].nctx = k;
        }
        cl.sync();  // no CTA rewrites shared state while another still reads it
    }
}

// One encode step of a lane (scalar.rs:120-127 with the map of
// model.rs:125-133): a state at or above x_max = f << 20 gives up its low 16
// bits (at most one word). Returns whether the lane emits a word (its pre-step
// low 16 bits).
__device__ __forceinline__ bool enc_step(uint32_t &x, const EncStep &e) {
    const bool need = x > e.keep;
    x = enc_map(need ? x >> 16 : x, e);
    return need;
}

// Reverse-order encode of one block (scalar.rs:39-43 / :84-90) by two warps.
// The states' chain is all that is serial; where each word goes is not. So a
// chain warp (lane l owns state l, round r covers positions [32r, 32r + 32))
// walks the rounds from the last to the first in chunks of kEncChunk, and
// leaves each round's pre-step states and every lane's emit flags in shared
// memory; an emit warp on another scheduler compacts the words of one chunk
// (a vote and two population counts per round) while the chain runs the next.
// Two message buffers per pair, a named barrier for each buffer and direction.
//
// Measured on B200, cycles per round of one stream (1 MiB): one warp doing
// both, with a corrected reciprocal, 81 (order-0) and 86 (order-1); two warps
// 57. Bulk (2048 x 128 KiB), GB/s of input: binned order-0 497 -> 708,
// full-range order-1 476 -> 535, the latter at 88% of the shared-memory
// wavefronts (12 a round, most of them 16-byte table entries).
struct EncMsg {
    uint16_t word[kEncChunk][32];  // pre-step states' low halves, by round
    uint32_t bits[32];             // lane's emit flags, bit k = round k of the chunk
    int32_t job;                   // -1: no more jobs
    int32_t flags;                 // 1: first chunk of the job, 2: last
};

// Message fields by 32-bit shared addresses (through a pointer kept in a
// struct the compiler would take generic loads and stores).
constexpr uint32_t kMsgBits = kEncChunk * 64, kMsgJob = kMsgBits + 128, kMsgBytes = kMsgJob + 8;
static_assert(sizeof(EncMsg) == kMsgBytes, "message layout");
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
// Table entries (the table was written before a __syncwarp): unpacked ones
// of 16 bytes, and the arena's of 8.
__device__ __forceinline__ EncStep lds_step(uint32_t a) {
    EncStep e;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(e.m), "=r"(e.keep), "=r"(e.pack), "=r"(e.bias)
                 : "r"(a));
    return e;
}
__device__ __forceinline__ EncStep lds_entry(uint32_t a) {
    uint32_t m, y;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(m), "=r"(y) : "r"(a));
    return enc_unpack(m, y);
}
__device__ __forceinline__ void sts_u16(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((unsigned short)v));
}
__device__ __forceinline__ void sts_u32(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v));
}

// Barriers of pair p: 1 + 4 p + b when buffer b is full, + 2 when it is empty.
struct WordPipe {
    uint32_t msg;  // shared address of buffer 0
    int id;
    uint32_t sent;
    __device__ WordPipe(EncMsg *m, int pair)
        : msg((uint32_t)__cvta_generic_to_shared(m)), id(1 + 4 * pair), sent(0) {}
    // The buffer of the next message, once the emit warp has read it.
    __device__ __forceinline__ uint32_t open() {
        if (sent >= 2) asm volatile("bar.sync %0, 64;" ::"r"(id + 2 + (int)(sent & 1)) : "memory");
        return msg + (sent & 1) * kMsgBytes;
    }
    __device__ __forceinline__ void close(uint32_t m, uint32_t bits, int job, int flags) {
        const uint32_t lane = threadIdx.x & 31;
        sts_u32(m + kMsgBits + 4 * lane, bits);
        if (lane == 0) {
            sts_u32(m + kMsgJob, (uint32_t)job);
            sts_u32(m + kMsgJob + 4, (uint32_t)flags);
        }
        __syncwarp();
        asm volatile("bar.arrive %0, 64;" ::"r"(id + (int)(sent & 1)) : "memory");
        sent++;
    }
    // The last message: no buffer is left in flight (one arrival of the emit
    // warp, for the message before, is still to be taken).
    __device__ void finish() {
        close(open(), 0u, -1, 0);
        if (sent >= 2) asm volatile("bar.sync %0, 64;" ::"r"(id + 2 + (int)(sent & 1)) : "memory");
    }
};

// Emit warp: the words of every chunk of its pair's jobs, stored back to
// front below the end of the job's region -- the reference emits them high
// lane first (scalar.rs:39-43), so they land in ascending lane order and the
// finished region is already in decode order (scalar.rs:134-139).
__device__ __forceinline__ void emit_words(EncMsg *buffers, int pair, EncBlock *__restrict__ blocks,
                                           const EncJob *__restrict__ jobs, uint16_t *__restrict__ words) {
    const int lane = threadIdx.x & 31, id = 1 + 4 * pair;
    const uint32_t ge = 0xffffffffu << lane;
    const uint32_t msg = (uint32_t)__cvta_generic_to_shared(buffers);
    uint16_t *end = nullptr, *wend = nullptr;
    for (uint32_t b = 0;; b ^= 1u) {
        asm volatile("bar.sync %0, 64;" ::"r"(id + (int)b) : "memory");
        const uint32_t m = msg + b * kMsgBytes;
        const int j = (int)lds_u32(m + kMsgJob);
        if (j < 0) return;
        const int flags = (int)lds_u32(m + kMsgJob + 4);
        const uint32_t bits = lds_u32(m + kMsgBits + 4 * lane);
        uint32_t w[kEncChunk];
#pragma unroll
        for (int k = 0; k < kEncChunk; k++) w[k] = lds_u16(m + 64 * k + 2 * lane);
        if (flags & 1) {
            const EncJob job = jobs[j];
            end = wend = words + blocks[job.block].word_off[job.order] + blocks[job.block].n;
        }
        // at: the write position, in words from wend (below 0). One block of
        // PTX per round, so that the vote and the store share a predicate.
        int32_t at = 0;
#pragma unroll
        for (int k = 0; k < kEncChunk; k++)
            asm volatile(
                "{\n"
                " .reg .pred q;\n"
                " .reg .b32 t, v, c;\n"
                " .reg .b64 a;\n"
                " and.b32 t, %1, %5;\n"
                " setp.ne.u32 q, t, 0;\n"
                " vote.sync.ballot.b32 v, q, 0xffffffff;\n"
                " and.b32 t, v, %2;\n"
                " popc.b32 c, t;\n"
                " sub.s32 c, %0, c;\n"
                " mad.wide.s32 a, c, 2, %3;\n"
                " @q st.global.u16 [a], %4;\n"
                " popc.b32 c, v;\n"
                " sub.s32 %0, %0, c;\n"
                "}"
                : "+r"(at)
                : "r"(bits), "r"(ge), "l"(wend), "h"((unsigned short)w[k]), "r"(1u << k)
                : "memory");
        wend += at;
        __syncwarp();
        asm volatile("bar.arrive %0, 64;" ::"r"(id + 2 + (int)b) : "memory");
        if ((flags & 2) && lane == 0) {
            const EncJob job = jobs[j];
            blocks[job.block].nwords[job.order] = (uint64_t)(end - wend);
        }
    }
}

// Symbols (or order-1 table indices) of the chunks ahead: a ring of kStages
// chunks in shared memory filled by 16-byte asynchronous copies.
constexpr int kStages = 4;
template <class E>
struct SymbolRing {
    static constexpr uint32_t kBytes = kEncChunk * 32 * sizeof(E), kStage = kBytes + 16;
    const uint8_t *top;  // the plan's
    uint32_t ring;       // shared address
    uint32_t mis, behind;
    int64_t chunks;

    // Chunk c holds the rounds [full - 16 (c + 1), full - 16 c) of a block of
    // `full` whole rounds.
    __device__ SymbolRing(const SymbolPlan &p, uint32_t smem)
        : top(reinterpret_cast<const uint8_t *>(p.top)), ring(smem), mis(p.mis), behind(p.behind), chunks(p.chunks) {}
    __device__ __forceinline__ uint32_t stage(int64_t c) const { return ring + (uint32_t)(c & (kStages - 1)) * kStage; }
    __device__ __forceinline__ void fetch(int64_t c) const {
        const uint32_t lane = threadIdx.x & 31;
        if (c < chunks) {
            const uint8_t *g = top - c * (int64_t)kBytes;
            const uint32_t d = stage(c);
#pragma unroll
            for (uint32_t o = 0; o < kBytes; o += 512)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + o + 16 * lane), "l"(g + o + 16 * lane));
            if (lane == 0 && mis)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d + kBytes), "l"(g + kBytes),
                             "r"(c == 0 ? behind : 16u));
        }
        asm volatile("cp.async.commit_group;");
    }
    // Waits until at most LEFT of the fetched chunks are still on their way.
    template <int LEFT>
    static __device__ __forceinline__ void wait() {
        asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
        __syncwarp();
    }
    // Element of the chunk's k-th round from the top.
    __device__ __forceinline__ uint32_t at(uint32_t s, int k) const {
        const uint32_t a = s + mis + (uint32_t)sizeof(E) * (32 * (kEncChunk - 1 - k) + (threadIdx.x & 31));
        if constexpr (sizeof(E) == 1) {
            uint32_t v;
            asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
            return v;
        } else {
            return lds_u16(a);
        }
    }
};

// Chain warp of one job. `first`: element 0 of the block (E: symbols, or
// order-1 table indices); `entry(s, up)`: the table entry of element s. CTX
// (order-1 on symbols): up is the context, byte i - 1 of position i, which
// for lanes 1-31 is the symbol the lane below holds in the same round, and for
// lane 0 the symbol lane 31 holds one round lower -- one shuffle per round
// instead of a second load.
template <bool CTX, class E, class Entry>
__device__ __forceinline__ uint32_t encode_chain(uint64_t n, const E *__restrict__ first, Entry &&entry,
                                                 WordPipe &pipe, int job, uint32_t ring) {
    const int lane = threadIdx.x & 31;
    uint32_t x = kRansL;
    const int64_t full = (int64_t)(n / 32);
    const uint32_t rem = (uint32_t)(n % 32);
    auto sym = [&](uint64_t i) -> uint32_t { return (uint32_t)first[i]; };
    const SymbolPlan plan = symbol_plan((uint64_t)(uintptr_t)first, n, sizeof(E));
    const SymbolRing<E> R(plan, ring);
    __syncwarp();  // the last job's reads of the ring are done
#pragma unroll
    for (int c = 0; c < kStages - 1; c++) R.fetch(c);
    int flags = 1;
    if (rem) {
        const uint64_t i = (uint64_t)full * 32 + lane;
        const bool active = lane < (int)rem;
        const uint32_t s = active ? sym(i) : 0u;
        uint32_t up = 0;
        if (CTX) up = active && i > 0 ? sym(i - 1) : 0u;
        const uint32_t m = pipe.open();
        sts_u16(m + 2 * lane, x);
        const uint32_t bits = active && enc_step(x, entry(s, up)) ? 1u : 0u;
        pipe.close(m, bits, job, full ? 1 : 3);
        flags = 0;
    }
    const int64_t tail = plan.tail;  // rounds below the whole chunks
    // Symbols of chunk c, whose next chunk is on its way; past the whole
    // chunks, of the rounds below them. `low`: the round below the lowest.
    struct Symbols {
        uint32_t s[kEncChunk], low;
    };
    auto look = [&](int64_t c, Symbols &S) {
        S.low = 0;
        if (c < R.chunks) {
            // keyless order-1 also reads the top round of chunk c + 1
            SymbolRing<E>::template wait<CTX ? 0 : 1>();
            const uint32_t st = R.stage(c);
#pragma unroll
            for (int k = 0; k < kEncChunk; k++) S.s[k] = R.at(st, k);
            if constexpr (CTX)
                S.low = c + 1 < R.chunks ? R.at(R.stage(c + 1), 0) : tail ? sym((uint64_t)(tail - 1) * 32 + lane) : 0u;
        } else {
#pragma unroll
            for (int k = 0; k < kEncChunk; k++)
                S.s[k] = c == R.chunks && k < tail ? sym((uint64_t)(tail - 1 - k) * 32 + lane) : 0u;
        }
    };
    auto step_of = [&](const Symbols &S, int k) {
        uint32_t up = 0;
        if constexpr (CTX) {
            const uint32_t below = (uint32_t)(lane + 31) & 31u;
            up = __shfl_sync(0xffffffffu, lane == 31 ? (k + 1 < kEncChunk ? S.s[(k + 1) % kEncChunk] : S.low) : S.s[k],
                             below);
        }
        return entry(S.s[k], up);
    };
    // A round's table entry is loaded kAhead rounds before its step, across
    // the chunks' edges (a ring of eight in registers), and a chunk's symbols
    // one chunk before: loaded where they are used, they cost every chunk
    // their latencies, about 240 cycles.
    constexpr int kAhead = 6;
    EncStep e[8];
    auto chunk = [&](int64_t c, const Symbols &S, Symbols &N, uint32_t on, bool all) {
        const bool last = c + 1 == R.chunks + (tail ? 1 : 0);
        const uint32_t m = pipe.open(), mine = m + 2 * lane;
        uint32_t bits = 0;
#pragma unroll
        for (int k = 0; k < kEncChunk; k++) {
            if (k == 2) {
                // chunk c's stage was read a chunk ago; the chunk kStages - 1
                // ahead takes the one before it
                look(c + 1, N);
                R.fetch(c + kStages - 1);
            }
            e[(k + kAhead) & 7] = k + kAhead < kEncChunk ? step_of(S, (k + kAhead) % kEncChunk)
                                                         : step_of(N, (k + kAhead) % kEncChunk);
            sts_u16(mine + 64 * k, x);
            if (all || (on >> k) & 1u)
                if (enc_step(x, e[k & 7])) bits |= 1u << k;
        }
        pipe.close(m, bits, job, flags | (last ? 2 : 0));
        flags = 0;
    };
    Symbols A, B;
    look(0, A);
#pragma unroll
    for (int k = 0; k < kAhead; k++) e[k] = step_of(A, k);
    int64_t c = 0;
    for (; c + 1 < R.chunks; c += 2) {
        chunk(c, A, B, 0u, true);
        chunk(c + 1, B, A, 0u, true);
    }
    // at most one whole chunk and the rounds below
    for (const int64_t end = R.chunks + (tail ? 1 : 0); c < end; c++) {
        chunk(c, A, B, c < R.chunks ? 0xffffffffu : (1u << tail) - 1u, false);
        A = B;
    }
    SymbolRing<E>::template wait<0>();
    return x;
}

// Order-1 tables are copied into the pair's slice of dynamic shared memory:
// unpacked for alphabets of up to kEncO1StepNu symbols, as they are in the
// arena for up to kEncO1SmemNu; larger ones are read through L1.
constexpr uint32_t kEncO1StepNu = 32;
constexpr uint32_t kEncO1SmemNu = 45;
constexpr uint32_t kEncO1TabBytes = kEncO1StepNu * kEncO1StepNu * 16;
static_assert(kEncO1SmemNu * kEncO1SmemNu * 8 <= kEncO1TabBytes, "a packed table fits the slice");

// Four CTAs per SM is the register limit; a fourth of its 228 KB of shared
// memory holds one, with 1 KB that the hardware reserves per CTA.
static_assert(kEncJobsPerCta * (256 * (sizeof(EncStep) + 1) + 2 * sizeof(EncMsg) +
                                kStages * SymbolRing<uint16_t>::kStage + kEncO1TabBytes) +
                      1024 <=
                  228 * 1024 / 4,
              "four encode CTAs per SM");

// Warps 0 .. kEncJobsPerCta - 1 are chain warps, the others emit warps, each
// of the next pair's number, so a pair's two warps sit on two schedulers.
__global__ void __launch_bounds__(kEncJobsPerCta * 64, 4)
    enc_run_kernel(const uint8_t *__restrict__ src, EncBlock *__restrict__ blocks,
                   const EncJob *__restrict__ jobs, int njobs, const uint8_t *__restrict__ tbl,
                   uint16_t *__restrict__ words, int *__restrict__ queue, const uint16_t *__restrict__ keys) {
    extern __shared__ __align__(16) uint8_t dsm[];
    __shared__ EncStep s_tab[kEncJobsPerCta][256];
    __shared__ uint8_t s_umap[kEncJobsPerCta][256];
    __shared__ __align__(16) EncMsg s_msg[kEncJobsPerCta][2];
    __shared__ __align__(16) uint8_t s_ring[kEncJobsPerCta][kStages * SymbolRing<uint16_t>::kStage];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp >= kEncJobsPerCta) {
        emit_words(s_msg[warp - kEncJobsPerCta], warp - kEncJobsPerCta, blocks, jobs, words);
        return;
    }
    WordPipe pipe(s_msg[warp], warp);
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(s_ring[warp]);
    for (;;) {
        int j = 0;
        if (lane == 0) j = atomicAdd(queue, 1);
        j = __shfl_sync(0xffffffffu, j, 0);
        if (j >= njobs) break;
        const EncJob job = jobs[j];
        EncBlock &B = blocks[job.block];
        const uint64_t n = B.n;
        const uint8_t *p = src + B.src_off;
        const uint8_t *T = tbl + B.tbl_off;
        uint32_t st = kRansL;
        if (n == 0) {
            if (lane == 0) B.nwords[job.order] = 0;
        } else if (job.order == 0) {
            const uint2 *T0 = reinterpret_cast<const uint2 *>(T + kTblO0);
            const uint32_t tab0 = (uint32_t)__cvta_generic_to_shared(s_tab[warp]);
#pragma unroll
            for (int k = 0; k < 8; k++) s_tab[warp][lane + 32 * k] = enc_unpack(T0[lane + 32 * k].x, T0[lane + 32 * k].y);
            __syncwarp();
            st = encode_chain<false>(n, p, [&](uint32_t s, uint32_t) { return lds_step(tab0 + 16 * s); }, pipe, j, ring);
        } else {
            const uint32_t nu = (uint32_t)B.nu;
            const uint2 *T1 = reinterpret_cast<const uint2 *>(T + kTblO1);
            const uint16_t *kp = keys ? keys + ((uintptr_t)src & 15u) + B.src_off : nullptr;
            const uint8_t *um = s_umap[warp];
            if (!keys) {
#pragma unroll
                for (int k = 0; k < 8; k++) s_umap[warp][lane * 8 + k] = T[kTblUmap + lane * 8 + k];
            }
            const uint32_t tab1 = (uint32_t)__cvta_generic_to_shared(dsm + warp * kEncO1TabBytes);
            auto index = [&](uint32_t s, uint32_t c) { return (uint32_t)um[c] * nu + um[s]; };
            auto global = [&](uint32_t i) {
                const uint2 e = __ldg(T1 + i);
                return enc_unpack(e.x, e.y);
            };
            if (nu <= kEncO1StepNu) {
                EncStep *t = reinterpret_cast<EncStep *>(dsm + warp * kEncO1TabBytes);
                for (uint32_t i = lane; i < nu * nu; i += 32) t[i] = enc_unpack(T1[i].x, T1[i].y);
            } else if (nu <= kEncO1SmemNu) {
                uint2 *t = reinterpret_cast<uint2 *>(dsm + warp * kEncO1TabBytes);
                for (uint32_t i = lane; i < nu * nu; i += 32) t[i] = T1[i];
            }
            __syncwarp();
            if (keys) {
                if (nu <= kEncO1StepNu)
                    st = encode_chain<false>(n, kp, [&](uint32_t s, uint32_t) { return lds_step(tab1 + 16 * s); }, pipe,
                                             j, ring);
                else if (nu <= kEncO1SmemNu)
                    st = encode_chain<false>(n, kp, [&](uint32_t s, uint32_t) { return lds_entry(tab1 + 8 * s); }, pipe,
                                             j, ring);
                else
                    st = encode_chain<false>(n, kp, [&](uint32_t s, uint32_t) { return global(s); }, pipe, j, ring);
            } else {
                if (nu <= kEncO1StepNu)
                    st = encode_chain<true>(
                        n, p, [&](uint32_t s, uint32_t c) { return lds_step(tab1 + 16 * index(s, c)); }, pipe, j, ring);
                else if (nu <= kEncO1SmemNu)
                    st = encode_chain<true>(
                        n, p, [&](uint32_t s, uint32_t c) { return lds_entry(tab1 + 8 * index(s, c)); }, pipe, j, ring);
                else
                    st = encode_chain<true>(
                        n, p, [&](uint32_t s, uint32_t c) { return global(index(s, c)); }, pipe, j, ring);
            }
        }
        B.states[job.order][lane] = st;
        __syncwarp();
    }
    pipe.finish();
}

__global__ void __launch_bounds__(1024)
    enc_select_scan_kernel(EncBlock *__restrict__ blocks, int nblocks, uint64_t *__restrict__ total) {
    __shared__ uint64_t wtot[32];
    __shared__ uint64_t carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nblocks; base += 1024) {
        const int b = base + tid;
        uint64_t size = 0;
        if (b < nblocks) {
            EncBlock &B = blocks[b];
            const uint64_t n = B.n;
            const uint64_t s0 = n ? kHdr + kO0Tables + kStatesBytes + 2 * B.nwords[0] : kHdr;
            const uint64_t s1 =
                n ? kHdr + kO1Bitmap + kO1Table * (uint64_t)B.nctx + kStatesBytes + 2 * B.nwords[1] : kHdr;
            int ch;
            switch (B.mode) {
                case FQXV_RANS_ORDER0: ch = 0; break;
                case FQXV_RANS_ORDER1: ch = 1; break;
                case FQXV_RANS_BEST_TIE0: ch = s1 < s0 ? 1 : 0; break;
                default: ch = s1 <= s0 ? 1 : 0; break;
            }
            B.out_size[0] = s0;
            B.out_size[1] = s1;
            B.chosen = ch;
            size = ch ? s1 : s0;
        }
        const uint64_t incl = warp_incl_scan_u64(size);
        if (lane == 31) wtot[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const uint64_t v = wtot[lane];
            const uint64_t vi = warp_incl_scan_u64(v);
            wtot[lane] = vi - v;
            if (lane == 31) wtot[31] = vi - v;  // keep exclusive; chunk total below
        }
        __syncthreads();
        const uint64_t excl = carry + wtot[warp] + incl - size;
        if (b < nblocks) blocks[b].out_off = excl;
        __syncthreads();
        if (tid == 1023) carry = excl + size;
        __syncthreads();
    }
    if (tid == 0) *total = carry;
}

// Bytes [lo, hi) of src to the same positions of dst, by the whole CTA:
// 4-byte stores at aligned destination addresses, each assembled from the
// two aligned source words it straddles (a load never leaves the aligned
// word of a byte it needs).
__device__ __forceinline__ void cta_copy(uint8_t *__restrict__ dst, const uint8_t *__restrict__ src, uint64_t lo,
                                         uint64_t hi) {
    const uint32_t tid = threadIdx.x;
    if (hi <= lo) return;
    const uint64_t lead = (4u - ((uintptr_t)(dst + lo) & 3u)) & 3u;
    const uint64_t head = lead < hi - lo ? lead : hi - lo;
    if (tid < head) dst[lo + tid] = src[lo + tid];
    const uint64_t a = lo + head;
    const uint64_t nw = (hi - a) / 4;
    const uint32_t sh = (uint32_t)((uintptr_t)(src + a) & 3u);
    const uint32_t *s4 = reinterpret_cast<const uint32_t *>((uintptr_t)(src + a) & ~(uintptr_t)3);
    uint32_t *d4 = reinterpret_cast<uint32_t *>(dst + a);
    if (sh == 0) {
        for (uint64_t j = tid; j < nw; j += blockDim.x) d4[j] = s4[j];
    } else {
        for (uint64_t j = tid; j < nw; j += blockDim.x) d4[j] = __funnelshift_r(s4[j], s4[j + 1], 8 * sh);
    }
    const uint64_t t = a + 4 * nw;
    if (tid < hi - t) dst[t + tid] = src[t + tid];
}

// One work item per (block, part): part 0 writes the header and states, and
// every part its share of the order-1 tables and of the renorm words (all
// tables by part 0 kept its CTA busy long after the others: 2048 x 128 KiB
// full-range blocks, 32 tables each, 376 us against 278).
__global__ void __launch_bounds__(kPackThreads)
    enc_pack_kernel(const EncBlock *__restrict__ blocks, int nblocks, const uint8_t *__restrict__ tbl,
                    const uint16_t *__restrict__ words, uint8_t *__restrict__ dst) {
    __shared__ uint8_t present[256];
    __shared__ uint8_t rowctx[256];
    __shared__ uint8_t s_um[256];
    __shared__ int s_k;
    const int tid = threadIdx.x;
    const int nitems = nblocks * kPackParts;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int b = item / kPackParts, part = item % kPackParts;
        const EncBlock &B = blocks[b];
        const int o = B.chosen;
        const uint64_t n = B.n;
        uint8_t *d = dst + B.out_off;
        if (n == 0 && part != 0) continue;
        if (part == 0) {
            if (tid == 0) d[0] = (uint8_t)o;
            if (tid >= 1 && tid <= 8) d[tid] = (uint8_t)(n >> (8 * (tid - 1)));
            if (n == 0) continue;
        }
        const uint8_t *T = tbl + B.tbl_off;
        uint64_t off = kHdr;
        if (o == 0) {
            if (part == 0) {
                const uint2 *T0 = reinterpret_cast<const uint2 *>(T + kTblO0);
                for (int s = tid; s < 256; s += blockDim.x) {
                    const uint32_t f = enc_freq(T0[s].y);
                    d[off + 2 * s] = (uint8_t)f;
                    d[off + 2 * s + 1] = (uint8_t)(f >> 8);
                }
            }
            off += kO0Tables;
        } else {
            // scalar.rs:96-107: presence bitmap, then one table per present
            // context in ascending context order.
            const int nu = B.nu;
            const uint2 *T1 = reinterpret_cast<const uint2 *>(T + kTblO1);
            // With all 256 byte values in U the map is the identity and 0xFF
            // is a real index, not the "absent" marker.
            const bool full = nu == 256;
            if (tid < 256) {
                const uint32_t u = T[kTblUmap + tid];
                bool pr = false;
                if (full || u != 0xffu)
                    for (int v = 0; v < nu && !pr; v++) pr = T1[(size_t)u * nu + v].y != 0;
                s_um[tid] = (uint8_t)u;
                present[tid] = pr;
            }
            __syncthreads();
            if (tid < 32) {
                uint32_t bits = 0, cntp = 0;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    bits |= (uint32_t)present[tid * 8 + k] << k;
                    cntp += present[tid * 8 + k];
                }
                if (part == 0) d[off + tid] = (uint8_t)bits;
                uint32_t base = warp_incl_scan(cntp) - cntp;
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (present[tid * 8 + k]) rowctx[base++] = (uint8_t)(tid * 8 + k);
                if (tid == 31) s_k = (int)base;
            }
            __syncthreads();
            off += kO1Bitmap;
            const int K = s_k;
            const int e1 = K * 256 * (part + 1) / kPackParts;
            for (int e = K * 256 * part / kPackParts + tid; e < e1; e += blockDim.x) {
                const uint32_t u = s_um[rowctx[e >> 8]];
                const uint32_t us = s_um[e & 255];
                const uint32_t f = (full || us != 0xffu) ? enc_freq(T1[(size_t)u * nu + us].y) : 0u;
                d[off + 2 * (uint64_t)e] = (uint8_t)f;
                d[off + 2 * (uint64_t)e + 1] = (uint8_t)(f >> 8);
            }
            off += kO1Table * (uint64_t)K;
        }
        if (part == 0 && tid < kStates) {
            const uint32_t x = B.states[o][tid];
#pragma unroll
            for (int k = 0; k < 4; k++) d[off + 4 * tid + k] = (uint8_t)(x >> (8 * k));
        }
        const uint64_t W2 = 2 * B.nwords[o];
        const uint64_t lo = (W2 * part / kPackParts) & ~(uint64_t)15;
        const uint64_t hi = part + 1 == kPackParts ? W2 : (W2 * (part + 1) / kPackParts) & ~(uint64_t)15;
        const uint8_t *ws = reinterpret_cast<const uint8_t *>(words + B.word_off[o] + n - B.nwords[o]);
        cta_copy(d + off + kStatesBytes, ws, lo, hi);
        __syncthreads();  // the next item rewrites the shared arrays
    }
}

cudaError_t launch_enc_model(const uint8_t *src, EncBlock *blocks, const uint32_t *order, int nblocks,
                             uint8_t *tbl, uint32_t *hist_scratch, uint16_t *keys, int grid, int cluster,
                             cudaStream_t s) {
    if (nblocks <= 0) return cudaSuccess;
    // `grid` clusters of `cluster` CTAs
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid * (unsigned)cluster, 1, 1);
    cfg.blockDim = dim3(kModelThreads, 1, 1);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, enc_model_kernel, src, blocks, order, nblocks, tbl, hist_scratch, keys);
}

void launch_enc_run(const uint8_t *src, EncBlock *blocks, const EncJob *jobs, int njobs,
                    const uint8_t *tbl, uint16_t *words, int *queue, const uint16_t *keys, int grid,
                    cudaStream_t s) {
    if (njobs <= 0) return;
    static std::mutex mu;
    static bool done[256];
    int dev = 0;
    cudaGetDevice(&dev);
    {
        // raised once per device: a per-launch setting would race between
        // host threads (see the decode launchers)
        std::lock_guard<std::mutex> lk(mu);
        if (dev >= 0 && dev < 256 && !done[dev]) {
            cudaFuncSetAttribute(enc_run_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(kEncJobsPerCta * kEncO1TabBytes));
            cudaFuncSetAttribute(enc_run_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared);
            cudaGetLastError();
            done[dev] = true;
        }
    }
    enc_run_kernel<<<grid, kEncJobsPerCta * 64, kEncJobsPerCta * kEncO1TabBytes, s>>>(src, blocks, jobs, njobs, tbl,
                                                                                     words, queue, keys);
}

void launch_enc_select_scan(EncBlock *blocks, int nblocks, uint64_t *total, cudaStream_t s) {
    enc_select_scan_kernel<<<1, 1024, 0, s>>>(blocks, nblocks, total);
}

void launch_enc_pack(EncBlock *blocks, int nblocks, const uint8_t *tbl, const uint16_t *words,
                     uint8_t *dst, int grid, cudaStream_t s) {
    if (nblocks <= 0) return;
    enc_pack_kernel<<<grid, kPackThreads, 0, s>>>(blocks, nblocks, tbl, words, dst);
}

}  // namespace fqxv

extern "C" int fqxv_rans_test_enc_map(uint32_t f, uint32_t cum, const uint32_t *v, size_t n, uint32_t *out) {
    if (f == 0 || f > fqxv::kTotFreq || (n && (!v || !out))) return FQXV_RANS_E_INVALID_ARG;
    const fqxv::EncEntry e = fqxv::enc_entry_of(f, cum);
    const fqxv::EncStep s = fqxv::enc_unpack(e.m, e.y);
    if (fqxv::enc_freq(e.y) != f || s.keep != (f << 20) - 1u) return FQXV_RANS_E_INVALID_ARG;
    for (size_t i = 0; i < n; i++) out[i] = fqxv::enc_map(v[i], s);
    return FQXV_RANS_OK;
}

extern "C" void fqxv_rans_test_enc_reads(uint64_t first, uint64_t n, uint32_t size, uint64_t *lo, uint64_t *hi) {
    // what SymbolRing::fetch copies: the lowest chunk's first granule up, and
    // chunk 0's last granule with the one behind it
    const fqxv::SymbolPlan p = fqxv::symbol_plan(first, n, size);
    *lo = *hi = first;
    if (p.chunks <= 0) return;
    const uint64_t bytes = (uint64_t)fqxv::kEncChunk * 32 * size;
    *lo = p.top - (uint64_t)(p.chunks - 1) * bytes;
    *hi = p.top + bytes + (p.mis ? p.behind : 0u);
}
