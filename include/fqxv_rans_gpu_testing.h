/*
 * fqxv_rans_gpu_testing.h -- test-only controls of libfqxv_rans_gpu.so.
 *
 * Not part of the coder's API (fqxv_rans_gpu.h) and with no counterpart in
 * the reference: these calls exist so that tests can drive failure paths that
 * normal operation never reaches, without faulting or hanging a GPU.
 */
#ifndef FQXV_RANS_GPU_TESTING_H
#define FQXV_RANS_GPU_TESTING_H

#include <stddef.h>
#include <stdint.h>

#include "fqxv_rans_gpu.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Polls a decode kernel makes of its table copy's barrier before it gives up
 * (default 4194304). A wait that gives up is followed by a drain of the same
 * copy with the default bound; the stream then reports FQXV_RANS_E_TIMEOUT,
 * and a CTA whose drain also failed reports FQXV_RANS_E_TIMEOUT for every
 * stream it takes afterwards without issuing another copy. 0 makes every
 * first wait give up at once, so each stream of the order-0 and shared-memory
 * order-1 decoders reports FQXV_RANS_E_TIMEOUT while its copy still lands.
 * Applies to the context and its sub-contexts. */
int fqxv_rans_ctx_test_set_wait_polls(fqxv_rans_ctx *ctx, uint32_t polls);

/* The encoder's state map for a symbol of frequency f (1..4096) and cumulative
 * frequency cum: out[i] = (v[i] / f) * 4096 + v[i] % f + cum, from the table
 * entry's multiplication. Host arithmetic, the same functions as the kernels'.
 * FQXV_RANS_E_INVALID_ARG when the entry does not give back f and f << 20. */
int fqxv_rans_test_enc_map(uint32_t f, uint32_t cum, const uint32_t *v, size_t n, uint32_t *out);

/* The addresses [*lo, *hi) that the encoder's chunk copies read of a block of n
 * elements of `size` bytes at address `first`: the kernel's plan, on the host
 * (nothing is dereferenced; *lo = *hi = first when it makes no such copy). */
void fqxv_rans_test_enc_reads(uint64_t first, uint64_t n, uint32_t size, uint64_t *lo, uint64_t *hi);

/* Rounds that a decoder runs in one go, without a check of the words left,
 * from round r of `full` whole rounds and word wp of navail: the kernels'
 * function, on the host. */
int64_t fqxv_rans_test_fast_rounds(uint64_t navail, uint64_t wp, uint64_t full, uint64_t r);

#ifdef __cplusplus
}
#endif
#endif
