/*
 * tbmd_probe.h - measurement helper exported by libtbmd.so (no counterpart in the reference).
 *
 * The roofline of the triplet kernels is the FP32 pipe (mixed precision) or the FP64 pipe (FP64
 * drop-in), not a tensor core or HBM figure, so the benchmark measures those pipe peaks on the
 * device it runs on with a dependent-chain-free FMA loop.
 *
 * And two handles for tests on limits that no run reaches.
 */
#ifndef TBMD_PROBE_H
#define TBMD_PROBE_H

#include <stdint.h>

#include "tbmd.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Measured FMA throughput of `device` in TFLOP/s (an FMA counts 2 FLOP): fp64 = 0 for the FP32
 * pipe, 1 for the FP64 pipe.  Runs about 0.1-0.3 s; returns a negative value on a CUDA error.  The
 * calling thread's current device is the same afterwards. */
double tbmd_probe_fma_tflops(int32_t device, int32_t fp64);

/* 1 if the forces of the context's particles go through the pair-tensor product, 0 if they go through a sweep or
 * the neighbour lists (after an evaluation: a workspace that was not to be had counts as the sweep). */
int32_t tbmd_probe_pairs(const tbmd_ctx *ctx);

/* Waits inside the pair-tensor kernels (no cutoff) of this context give up after `cycles` clock cycles (4e9 in a
 * new context); with 0 the first one does, and the evaluation ends with TBMD_TIMEOUT. */
tbmd_status tbmd_probe_pair_waits(tbmd_ctx *ctx, int64_t cycles);

/* A workspace of the pair-tensor product (no cutoff) that would take more than `bytes` is not to be had in this
 * context, as if the device's memory were full; takes effect with the next sizes. */
tbmd_status tbmd_probe_pair_workspace(tbmd_ctx *ctx, int64_t bytes);

#ifdef __cplusplus
}
#endif

#endif
