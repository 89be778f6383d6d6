// Values of eight 32-bit limbs (field elements, scalars) across a warp, for the
// product scans of the RLC's batch inversion.
#pragma once
#include "common.cuh"

namespace uf {

template <class V>
__device__ __forceinline__ V grp_shfl_up(const V& a, int d) {
    V r;
    UF_UNROLL
    for (int i = 0; i < 8; ++i) r.v[i] = __shfl_up_sync(0xFFFFFFFFu, a.v[i], d);
    return r;
}

template <class V>
__device__ __forceinline__ V grp_shfl_down(const V& a, int d) {
    V r;
    UF_UNROLL
    for (int i = 0; i < 8; ++i) r.v[i] = __shfl_down_sync(0xFFFFFFFFu, a.v[i], d);
    return r;
}

template <class V>
__device__ __forceinline__ V grp_shfl(const V& a, int src) {
    V r;
    UF_UNROLL
    for (int i = 0; i < 8; ++i) r.v[i] = __shfl_sync(0xFFFFFFFFu, a.v[i], src);
    return r;
}

}  // namespace uf
