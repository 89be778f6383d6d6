// Small calls by four or two warps per 32 signatures (team.cuh).
#include "kernels.h"
#include "team.cuh"

namespace uf {
namespace {

template <int kKind, int kWarps>
__global__ void __launch_bounds__(kWarps * kTeamLanes, 8 / kWarps)
k_verify_team(const uint8_t* __restrict__ msgs, const uint8_t* __restrict__ pubs, const uint8_t* __restrict__ sigs,
              uint32_t n, const uint4* __restrict__ gt, const uint4* __restrict__ comb, uint8_t* __restrict__ out,
              int collect) {
    extern __shared__ uint4 smem[];
    const uint32_t i = blockIdx.x * kTeamLanes + (threadIdx.x & 31u);
    const bool ok = team_verify<kKind, kWarps>(msgs + 32ull * i, pubs + (kKind == 1 ? 32ull : 33ull) * i, sigs + 64ull * i,
                                       i < n, gt, comb, smem);
    if (threadIdx.x < kTeamLanes && i < n) {
        if (collect) {
            if (ok) out[i] = 0;
        } else {
            out[i] = ok ? 1 : 0;
        }
    }
}

}  // namespace

template <int kWarps>
static void launch_team(int kind, const uint8_t* msgs, const uint8_t* pubs, const uint8_t* sigs, uint32_t n,
                        const uint4* gt, const uint4* comb, uint8_t* out, int collect, cudaStream_t s) {
    const uint32_t grid = (n + kTeamLanes - 1) / kTeamLanes;
    constexpr int threads = kWarps * kTeamLanes;
    if (kind == 0)
        k_verify_team<0, kWarps><<<grid, threads, kTeamSmem, s>>>(msgs, pubs, sigs, n, gt, comb, out, collect);
    else if (kind == 2)
        k_verify_team<2, kWarps><<<grid, threads, kTeamSmem, s>>>(msgs, pubs, sigs, n, gt, comb, out, collect);
    else
        k_verify_team<1, kWarps><<<grid, threads, kTeamSmem, s>>>(msgs, pubs, sigs, n, gt, comb, out, collect);
}

cudaError_t launch_verify_team(int kind, const uint8_t* msgs, const uint8_t* pubs, const uint8_t* sigs, uint32_t n,
                               const void* d_gtab, const void* d_comb, uint8_t* out, int collect, int sms,
                               cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint4* gt = reinterpret_cast<const uint4*>(d_gtab);
    const uint4* comb = reinterpret_cast<const uint4*>(d_comb);
    // more than a block per SM: two warps per 32 signatures, so that a second
    // block still finds idle schedulers (6,011 signatures 440 us by four warps, 338
    // by two; up to a block per SM 269 by four)
    if (n > (uint32_t)sms * kTeamLanes) launch_team<2>(kind, msgs, pubs, sigs, n, gt, comb, out, collect, s);
    else launch_team<4>(kind, msgs, pubs, sigs, n, gt, comb, out, collect, s);
    return cudaGetLastError();
}

cudaError_t verify_team_init() {
    cudaError_t e = cudaSuccess;
    auto opt_in = [&](auto f) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTeamSmem);
    };
    opt_in(k_verify_team<0, 4>);
    opt_in(k_verify_team<1, 4>);
    opt_in(k_verify_team<2, 4>);
    opt_in(k_verify_team<0, 2>);
    opt_in(k_verify_team<1, 2>);
    opt_in(k_verify_team<2, 2>);
    return e;
}

}  // namespace uf
