// Launchers of the RLC kernels that run one serial chain per segment or
// window (rlc_serial.cu): few threads, so latency-bound.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "rlc_dev.cuh"

namespace uf {

// Running sums over each (segment, window)'s buckets in sub-ranges, their
// combination per window, and Horner over the windows per segment:
// segok[s] = 1 when segment s's sum is infinity, | 2 when it holds an item
// that failed to parse; segpt[s] = the sum.  schedulers: the device's, four per SM.
cudaError_t launch_rlc_windows(const rlcdev::RoundGeo& g, const uint4* buckets, uint4* wins,
                               const uint32_t* segbad, uint8_t* segok, uint4* segpt, int schedulers,
                               cudaStream_t s);

// Buckets of two or more chunks: the sum of their chunk partials, by a thread
// per bucket, or by a warp per bucket of more than heavy_from >= kHeavyChunks
// chunks (their keys listed in heavy[1..heavy[0]] by the first kernel).
cudaError_t launch_rlc_bucket_merge(const uint32_t* coff, uint32_t K, uint32_t heavy_from, const uint4* partials,
                                    uint4* buckets, uint32_t* heavy, int heavy_grid, cudaStream_t s);

}  // namespace uf
