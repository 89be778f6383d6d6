// The RLC kernels with one serial chain per bucket, segment or window: the
// merge of a bucket's chunk sums, the window sums and Horner.  All but the merge run a few thousand threads at most, so a chain's
// latency, not the issue rate, sets their time: they use the FP64 field
// arithmetic (fd.cuh), whose products are independent where the limb form is a
// chain of carries (a doubling alone on its scheduler 2.3 k cycles against
// 5.0 k), and trees over a warp's lanes instead of chains.  64 segments of 4,096
// items, window 10: window sums 653 -> 329 us, Horner 368 -> 155 us.
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

// Window sums: S lanes per (segment, window), lane j over m = B / S buckets.
//   T_j = sum_b bucket_b, U_j = sum_b (b - j m + 1) bucket_b by running sums,
//   window = sum_j U_j + m sum_j j T_j,  sum_j j T_j = sum_(j >= 1) T'_j
// with the suffix sums T'_j = T_j + T_(j+1) + ...: a scan, log2(m) doublings of
// every lane's T'_j at once, and a tree.  (A tree over (U, T) pairs alone doubles
// T by each range's length: 30 doublings and 10 additions where this takes 4 and
// 11 for m = 16.)  Blocks are one warp, or the S / 32 warps of one window.
__global__ void __launch_bounds__(256)
k_rlc_window(RoundGeo g, const uint4* __restrict__ buckets, uint4* __restrict__ wins) {
    __shared__ JacD part[8];
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t sw = q / (uint32_t)g.S, j = q - sw * (uint32_t)g.S;
    const bool live = sw < g.n_seg * (uint32_t)g.W;
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5), warps = (int)(blockDim.x >> 5);
    const int width = g.S < 32 ? g.S : 32, at = lane & (width - 1);     // this window's lanes of the warp
    const int m = g.B / g.S;
    JacD run, tot, b;
    jacd_set_inf(run);
    jacd_set_inf(tot);
    if (live) {
        const uint4* base = buckets + kJacQ * ((uint64_t)sw * g.B + (uint64_t)j * m);
        for (int k = m - 1; k >= 0; --k) {
            load_jacd(base + kJacQ * k, b);
            run = jacd_add(run, b);
            tot = jacd_add(tot, run);
        }
    }
    __syncwarp();
    for (int d = 1; d < width; d <<= 1) {
        const JacD o = shfl_jacd(run, at + d < width ? lane + d : lane);
        if (at + d < width) run = jacd_add(run, o);
        __syncwarp();
    }
    if (warps > 1) {
        if (lane == 0) part[warp] = run;
        __syncthreads();
        JacD above;
        jacd_set_inf(above);
        for (int v = warps - 1; v > warp; --v) above = jacd_add(above, part[v]);
        run = jacd_add(run, above);
        __syncthreads();
    }
    int log2m = 0;
    while (m >> (log2m + 1)) ++log2m;
    if (j == 0) jacd_set_inf(run);
    tot = jacd_add(tot, jacd_dbl_n(run, log2m));
    __syncwarp();
    for (int d = 1; d < width; d <<= 1) {
        const JacD o = shfl_jacd(tot, at + d < width ? lane + d : lane);
        if (at + d < width) tot = jacd_add(tot, o);
        __syncwarp();
    }
    if (warps > 1) {
        if (lane == 0) part[warp] = tot;
        __syncthreads();
        for (int v = 1; threadIdx.x == 0 && v < warps; ++v) tot = jacd_add(tot, part[v]);
    }
    if (live && j == 0) store_jacd(wins + kJacQ * (uint64_t)sw, tot);
}

// Horner over the windows, `lanes` (a power of two of at most 32) per segment: a
// lane takes ceil(W / lanes) neighbouring windows by Horner's rule, doubles the
// result up to its place, all lanes at once, and a tree adds them: the chain
// keeps its 129 doublings but has about W / lanes + log2(lanes) additions instead
// of W - 1.  ok = 1 if the sum is infinity, | 2 if the segment holds an item that
// failed to parse.
__global__ void __launch_bounds__(32)
k_rlc_finish(RoundGeo g, int lanes, const uint4* __restrict__ wins, const uint32_t* __restrict__ segbad,
             uint8_t* __restrict__ segok, uint4* __restrict__ segpt) {
    const uint32_t q = blockIdx.x * 32 + threadIdx.x, s = q / (uint32_t)lanes;
    const int lane = (int)threadIdx.x, at = lane & (lanes - 1);
    const int per = (g.W + lanes - 1) / lanes, first = at * per, last = first + per < g.W ? first + per : g.W;
    JacD acc, w;
    jacd_set_inf(acc);
    if (s < g.n_seg && first < last) {
        const uint4* base = wins + kJacQ * (uint64_t)s * g.W;
        load_jacd(base + kJacQ * (last - 1), acc);
        for (int k = last - 2; k >= first; --k) {
            acc = jacd_dbl_n(acc, g.c);
            load_jacd(base + kJacQ * k, w);
            acc = jacd_add(acc, w);
        }
        acc = jacd_dbl_n(acc, g.c * first);
    }
    __syncwarp();
    for (int d = 1; d < lanes; d <<= 1) {
        const JacD o = shfl_jacd(acc, at + d < lanes ? lane + d : lane);
        if (at + d < lanes) acc = jacd_add(acc, o);
        __syncwarp();
    }
    if (s < g.n_seg && at == 0) {
        segok[s] = (uint8_t)((acc.inf ? 1 : 0) | (segbad[s] ? 2 : 0));
        store_jacd(segpt + kJacQ * (uint64_t)s, acc);
    }
}

// Buckets with 0 or >= 2 chunks: infinity, or the sum of their partials.
// A bucket of more than heavy_from chunks (skewed digits: the top windows
// of a locate round's j-scaled magnitudes put most points of a segment into a
// few buckets) is left to k_rlc_bucket_heavy: its key goes to `heavy`.
__device__ __forceinline__ void add_partial(JacD& acc, const uint4* q) {
    JacD p;
    load_jacd(q, p);
    acc = jacd_add(acc, p);
}

__global__ void __launch_bounds__(128)
k_rlc_bucket_fin(const uint32_t* __restrict__ coff, uint32_t K, uint32_t heavy_from,
                 const uint4* __restrict__ partials, uint4* __restrict__ buckets, uint32_t* __restrict__ heavy) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    const uint32_t c0 = coff[k], c1 = coff[k + 1];
    if (c1 - c0 == 1) return;
    if (c1 - c0 > heavy_from) {
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

inline unsigned grid_of(uint64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace

cudaError_t launch_rlc_windows(const RoundGeo& g, const uint4* buckets, uint4* wins, const uint32_t* segbad,
                               uint8_t* segok, uint4* segpt, int schedulers, cudaStream_t s) {
    const uint64_t n_seg = g.n_seg;
    const int threads = g.S > 32 ? g.S : 32;
    k_rlc_window<<<grid_of(n_seg * g.W * g.S, threads), threads, 0, s>>>(g, buckets, wins);
    int lanes = 32;                                // while the warps stay at one per scheduler
    while (lanes > 1 && (n_seg * lanes > (uint64_t)schedulers * 32 || lanes >= 2 * g.W)) lanes >>= 1;
    k_rlc_finish<<<grid_of(n_seg * lanes, 32), 32, 0, s>>>(g, lanes, wins, segbad, segok, segpt);
    return cudaGetLastError();
}

cudaError_t launch_rlc_bucket_merge(const uint32_t* coff, uint32_t K, uint32_t heavy_from, const uint4* partials,
                                    uint4* buckets, uint32_t* heavy, int heavy_grid, cudaStream_t s) {
    k_rlc_bucket_fin<<<grid_of(K, 128), 128, 0, s>>>(coff, K, heavy_from, partials, buckets, heavy);
    k_rlc_bucket_heavy<<<heavy_grid, 128, 0, s>>>(coff, partials, buckets, heavy);
    return cudaGetLastError();
}

}  // namespace uf
