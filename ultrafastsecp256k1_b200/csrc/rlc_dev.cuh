// Device-side pieces shared by the RLC translation units (rlc.cu and
// rlc_serial.cu): point storage in global memory and the round geometry.
#pragma once
#include "common.cuh"
#include "fe.cuh"
#include "jacd.cuh"
#include "point.cuh"

namespace uf {
namespace rlcdev {

__device__ __forceinline__ void store_aff(uint4* q, const Fe& x, const Fe& y) {
    q[0] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
    q[1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
    q[2] = make_uint4(y.v[0], y.v[1], y.v[2], y.v[3]);
    q[3] = make_uint4(y.v[4], y.v[5], y.v[6], y.v[7]);
}

__device__ __forceinline__ void load_aff(const uint4* q, Fe& x, Fe& y) {
    const uint4 a = q[0], b = q[1], c = q[2], d = q[3];
    x.v[0] = a.x; x.v[1] = a.y; x.v[2] = a.z; x.v[3] = a.w;
    x.v[4] = b.x; x.v[5] = b.y; x.v[6] = b.z; x.v[7] = b.w;
    y.v[0] = c.x; y.v[1] = c.y; y.v[2] = c.z; y.v[3] = c.w;
    y.v[4] = d.x; y.v[5] = d.y; y.v[6] = d.z; y.v[7] = d.w;
}

// Jacobian point in global memory: X, Y, Z and the infinity flag (7 x uint4).
constexpr int kJacQ = 7;

__device__ __forceinline__ void load_jac(const uint4* q, Jac& P) {
    load_aff(q, P.X, P.Y);
    const uint4 a = q[4], b = q[5];
    P.Z.v[0] = a.x; P.Z.v[1] = a.y; P.Z.v[2] = a.z; P.Z.v[3] = a.w;
    P.Z.v[4] = b.x; P.Z.v[5] = b.y; P.Z.v[6] = b.z; P.Z.v[7] = b.w;
    P.inf = q[6].x != 0;
}

// The same storage for points in digit form (jacd.cuh): any 256-bit representative
// is read, canonical ones are written where the point was computed in that form.
__device__ __forceinline__ void load_limbs(Fd& r, const uint4* q) {
    const uint4 a = q[0], b = q[1];
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    fd_unpack(r, w);
    fd_strict(r);
}

__device__ __forceinline__ void store_limbs(uint4* q, const Fd& a) {
    uint32_t w[8];
    fd_pack(w, a);
    q[0] = make_uint4(w[0], w[1], w[2], w[3]);
    q[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

__device__ __forceinline__ void load_jacd(const uint4* q, JacD& p) {
    load_limbs(p.X, q);
    load_limbs(p.Y, q + 2);
    load_limbs(p.Z, q + 4);
    p.inf = q[6].x != 0;
}

__device__ __forceinline__ void store_jacd(uint4* q, const JacD& p) {
    store_limbs(q, p.X);
    store_limbs(q + 2, p.Y);
    store_limbs(q + 4, p.Z);
    q[6] = make_uint4(p.inf ? 1u : 0u, 0u, 0u, 0u);
}

// Round geometry in device memory: seg[2s], seg[2s+1] = first item, length of
// segment s; pwf[s] = first (point, window) index of segment s, pwf[S] = total.
struct RoundGeo {
    const uint32_t* seg;
    const uint32_t* pwf;
    uint32_t n_seg;
    uint32_t n3;             // 3 * items of the call: index of the first generator point
    int c, W, B, S;          // window bits, windows, buckets per window, sub-ranges per window
};

// A bucket of more chunks than this, and than twice the average bucket's, is merged
// by a warp (k_rlc_bucket_heavy): six additions of a warp for one bucket, against
// one per chunk for the 32 buckets of a warp of k_rlc_bucket_fin, so it pays for a
// few skewed buckets only.  With 8 alone, chunks shorter than an eighth of the
// average bucket sent most buckets there (262,144 items at 512 and chunks of 6: 9.1
// ms, at 1,000 9.7).
constexpr uint32_t kHeavyChunks = 8;

// The most chunks that one thread merges, in a round of `entries` over `buckets`.
inline uint32_t heavy_chunks(uint64_t entries, uint64_t buckets, uint32_t chunk) {
    const uint64_t twice = 2 * entries / (buckets * chunk);
    return twice > kHeavyChunks ? (uint32_t)twice : kHeavyChunks;
}

}  // namespace rlcdev
}  // namespace uf
