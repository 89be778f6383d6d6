// The RLC kernels with one serial chain per bucket, segment or window: the
// merge of a bucket's chunk sums, the running sums, the window combination and
// Horner.  All but the merge run a few thousand threads at most, so a chain's
// latency, not the issue rate, sets their time: they use the FP64 field
// arithmetic (fd.cuh), whose products are independent where the limb form is a
// chain of carries (a doubling alone on its scheduler 2.3 k cycles against
// 5.0 k), as many sub-ranges as a warp has lanes, and a tree instead of a chain
// to combine them.  64 segments of 4,096 items, window 10, per round: running
// sums 365 -> 232 us, combination 288 -> 216 us, Horner 368 -> 214 us.
#include "rlc_serial.h"

#include "jacd.cuh"
#include "point.cuh"

namespace uf {

namespace {

using namespace rlcdev;

__device__ __forceinline__ Fd shfl_fd(const Fd& a, int src) {
    Fd r;
    UF_UNROLL
    for (int k = 0; k < 5; ++k) r.v[k] = __shfl_sync(0xFFFFFFFFu, a.v[k], src);
    return r;
}

// Point of lane `src` of the warp (every lane calls it).
__device__ __forceinline__ JacD shfl_jacd(const JacD& a, int src) {
    JacD b;
    b.X = shfl_fd(a.X, src);
    b.Y = shfl_fd(a.Y, src);
    b.Z = shfl_fd(a.Z, src);
    b.inf = __shfl_sync(0xFFFFFFFFu, a.inf ? 1 : 0, src) != 0;
    return b;
}

// One thread per (segment, window, sub-range j of m buckets):
// T_j = sum_b bucket_b, U_j = sum_b (b - j m + 1) bucket_b by running sums.
__global__ void __launch_bounds__(128)
k_rlc_wpart(RoundGeo g, const uint4* __restrict__ buckets, uint4* __restrict__ wu, uint4* __restrict__ wt) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= g.n_seg * (uint32_t)(g.W * g.S)) return;
    const uint32_t sw = q / (uint32_t)g.S, j = q - sw * (uint32_t)g.S;
    const int m = g.B / g.S;
    const uint4* base = buckets + kJacQ * ((uint64_t)sw * g.B + (uint64_t)j * m);
    JacD run, tot, b;
    jacd_set_inf(run);
    jacd_set_inf(tot);
    for (int k = m - 1; k >= 0; --k) {
        load_jacd(base + kJacQ * k, b);
        run = jacd_add(run, b);
        tot = jacd_add(tot, run);
    }
    store_jacd(wu + kJacQ * (uint64_t)q, tot);
    store_jacd(wt + kJacQ * (uint64_t)q, run);
}

// S lanes per (segment, window), a power of two of at most 32: window sum =
// sum_j U_j + m sum_j j T_j by a tree over neighbouring ranges.  A range of
// 2^k sub-ranges keeps T = sum of its T_j and U = its sum of (bucket - first
// bucket + 1) weights, so two neighbours join as U + U' + m 2^k T', T + T'.
__global__ void __launch_bounds__(128)
k_rlc_wcomb(RoundGeo g, const uint4* __restrict__ wu, const uint4* __restrict__ wt, uint4* __restrict__ wins) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t total = g.n_seg * (uint32_t)(g.W * g.S);
    const int lane = (int)(threadIdx.x & 31u);
    JacD U, T;
    jacd_set_inf(U);
    jacd_set_inf(T);
    if (q < total) {
        load_jacd(wu + kJacQ * (uint64_t)q, U);
        load_jacd(wt + kJacQ * (uint64_t)q, T);
    }
    int log2len = 0;
    while ((g.B / g.S) >> (log2len + 1)) ++log2len;            // m = B / S
    for (int d = 1; d < g.S; d <<= 1, ++log2len) {
        // lanes that are not a range's first compute along and are not used
        const int src = lane + d < 32 ? lane + d : lane;
        const JacD U2 = shfl_jacd(U, src);
        const JacD T2 = shfl_jacd(T, src);
        U = jacd_add(U, U2);
        U = jacd_add(U, jacd_dbl_n(T2, log2len));
        if (2 * d < g.S) T = jacd_add(T, T2);
    }
    if (q < total && q % (uint32_t)g.S == 0) store_jacd(wins + kJacQ * (uint64_t)(q / (uint32_t)g.S), U);
}

// One thread per segment: Horner over the windows; ok = 1 if the sum is
// infinity, | 2 if the segment holds an item that failed to parse.
__global__ void __launch_bounds__(32)
k_rlc_finish(RoundGeo g, const uint4* __restrict__ wins, const uint32_t* __restrict__ segbad,
             uint8_t* __restrict__ segok, uint4* __restrict__ segpt) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.n_seg) return;
    const uint4* base = wins + kJacQ * (uint64_t)s * g.W;
    JacD acc, w;
    load_jacd(base + kJacQ * (g.W - 1), acc);
    for (int k = g.W - 2; k >= 0; --k) {
        acc = jacd_dbl_n(acc, g.c);
        load_jacd(base + kJacQ * k, w);
        acc = jacd_add(acc, w);
    }
    segok[s] = (uint8_t)((acc.inf ? 1 : 0) | (segbad[s] ? 2 : 0));
    store_jacd(segpt + kJacQ * (uint64_t)s, acc);
}

// Buckets with 0 or >= 2 chunks: infinity, or the sum of their partials.
// A bucket of more than kHeavyChunks chunks (skewed digits: the top windows
// of a locate round's j-scaled magnitudes put most points of a segment into a
// few buckets) is left to k_rlc_bucket_heavy: its key goes to `heavy`.
__device__ __forceinline__ void add_partial(JacD& acc, const uint4* q) {
    JacD p;
    load_jacd(q, p);
    acc = jacd_add(acc, p);
}

__global__ void __launch_bounds__(128)
k_rlc_bucket_fin(const uint32_t* __restrict__ coff, uint32_t K, const uint4* __restrict__ partials,
                 uint4* __restrict__ buckets, uint32_t* __restrict__ heavy) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    const uint32_t c0 = coff[k], c1 = coff[k + 1];
    if (c1 - c0 == 1) return;
    if (c1 - c0 > kHeavyChunks) {
        heavy[1 + atomicAdd(&heavy[0], 1u)] = k;
        return;
    }
    JacD acc;
    jacd_set_inf(acc);
    for (uint32_t c = c0; c < c1; ++c) add_partial(acc, partials + kJacQ * (uint64_t)c);
    store_jacd(buckets + kJacQ * (uint64_t)k, acc);
}

// One warp per heavy bucket (heavy[0] of them, keys in heavy[1..]): lane l
// sums partials l, l + 32, ..., then the 32 lane sums meet in a shuffle tree:
// about chunks / 32 + 5 serial additions instead of chunks.
__global__ void __launch_bounds__(128)
k_rlc_bucket_heavy(const uint32_t* __restrict__ coff, const uint4* __restrict__ partials,
                   uint4* __restrict__ buckets, const uint32_t* __restrict__ heavy) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < heavy[0]; w += warps) {
        const uint32_t k = heavy[1 + w];
        const uint32_t c0 = coff[k], c1 = coff[k + 1];
        JacD acc;
        jacd_set_inf(acc);
        for (uint32_t c = c0 + lane; c < c1; c += 32) add_partial(acc, partials + kJacQ * (uint64_t)c);
        for (int o = 16; o > 0; o >>= 1) {
            const JacD other = shfl_jacd(acc, (int)(lane ^ (uint32_t)o));
            acc = jacd_add(acc, other);
        }
        if (lane == 0) store_jacd(buckets + kJacQ * (uint64_t)k, acc);
    }
}

constexpr uint64_t kWarpHornerSegments = 592;      // one warp per scheduler of a 148-SM device

// The same with a warp per segment (at most 32 windows): lane w doubles window
// w's sum c w times, all windows at once, and a tree adds them: the chain has the
// same doublings but log2(W) additions instead of W - 1.  For rounds of few
// segments; many fill the device with a thread each.
__global__ void __launch_bounds__(32)
k_rlc_finish_warp(RoundGeo g, const uint4* __restrict__ wins, const uint32_t* __restrict__ segbad,
                  uint8_t* __restrict__ segok, uint4* __restrict__ segpt) {
    const uint32_t s = blockIdx.x;
    const int lane = (int)threadIdx.x;
    JacD acc;
    jacd_set_inf(acc);
    if (lane < g.W) {
        load_jacd(wins + kJacQ * ((uint64_t)s * g.W + lane), acc);
        acc = jacd_dbl_n(acc, g.c * lane);
    }
    __syncwarp();
    for (int d = 1; d < g.W; d <<= 1) {
        const JacD o = shfl_jacd(acc, lane + d < 32 ? lane + d : lane);
        if (lane + d < 32) acc = jacd_add(acc, o);
    }
    if (lane == 0) {
        segok[s] = (uint8_t)((acc.inf ? 1 : 0) | (segbad[s] ? 2 : 0));
        store_jacd(segpt + kJacQ * (uint64_t)s, acc);
    }
}

inline unsigned grid_of(uint64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace

cudaError_t launch_rlc_windows(const RoundGeo& g, const uint4* buckets, uint4* wu, uint4* wt, uint4* wins,
                               const uint32_t* segbad, uint8_t* segok, uint4* segpt, cudaStream_t s) {
    const uint64_t n_seg = g.n_seg;
    k_rlc_wpart<<<grid_of(n_seg * g.W * g.S, 128), 128, 0, s>>>(g, buckets, wu, wt);
    k_rlc_wcomb<<<grid_of(n_seg * g.W * g.S, 128), 128, 0, s>>>(g, wu, wt, wins);
    if (g.W <= 32 && n_seg <= kWarpHornerSegments)
        k_rlc_finish_warp<<<(unsigned)n_seg, 32, 0, s>>>(g, wins, segbad, segok, segpt);
    else
        k_rlc_finish<<<grid_of(n_seg, 32), 32, 0, s>>>(g, wins, segbad, segok, segpt);
    return cudaGetLastError();
}

cudaError_t launch_rlc_bucket_merge(const uint32_t* coff, uint32_t K, const uint4* partials, uint4* buckets,
                                    uint32_t* heavy, int heavy_grid, cudaStream_t s) {
    k_rlc_bucket_fin<<<grid_of(K, 128), 128, 0, s>>>(coff, K, partials, buckets, heavy);
    k_rlc_bucket_heavy<<<heavy_grid, 128, 0, s>>>(coff, partials, buckets, heavy);
    return cudaGetLastError();
}

}  // namespace uf
