// Verify kernels for mixed ECDSA / BIP-340 batches.
//
// No reference counterpart: the reference launches one kernel per batch call
// (src/gpu/src/gpu_backend_cuda.cu:972, :1085).  Here many caller batches of
// both kinds are packed into one staging region (see QueueLayout in
// kernels.h): per kind contiguous msg / key / signature arrays.  Each kind has
// its own kernel (so a warp never holds both verify paths, and each kernel's code
// stays small for the instruction cache); the two launches run as parallel
// branches (fork / join events), so a mixed request costs one verify latency, not
// two.
//
// The item counts are read from a header in device memory (copied with the
// inputs), so a CUDA graph captured for one capacity bucket replays unchanged
// for any fill level of that bucket: the grid covers the bucket, and blocks
// beyond the count return at once.
//
// With the resident key table (pubcache.cuh) two passes run before the verify
// kernels: k_key_resolve gives every item its key's slot (claiming slots for
// new keys), k_key_build builds the claimed slots' tables; the verify kernels
// then copy an item's table.  Small launches (four warps per 32 signatures,
// team.cuh) build the table beside the scalars anyway: there the passes run
// beside the verify kernels and only keep the keys for later launches.
#include "kernels.h"
#include "team.cuh"

namespace uf {

// One thread per item slot of both kinds (ECDSA items first, cap_e of them,
// then BIP-340): parse the key, find or claim its slot, record the slot index.
// Keys that fail to parse (prefix, x >= p) get kNoSlot: their verdict is 0
// either way.  Per warp one pair of atomics adds the lookups and the hits
// (keys found in a slot that was not claimed in this pass).
__global__ void __launch_bounds__(128)
k_key_resolve(QueueArgs a) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n_e = min(a.counts[0], a.cap_e), n_s = min(a.counts[1], a.cap_s);
    bool looked = false, hit = false;
    const bool is_e = t < a.cap_e;
    const uint32_t i = is_e ? t : t - a.cap_e;
    if (is_e ? i < n_e : (t < a.cap_e + a.cap_s && i < n_s)) {
        Fe x;
        bool odd = false, ok;
        if (is_e) {
            const uint8_t* pub = a.e_pubs + 33ull * i;
            ok = pub[0] == 0x02 || pub[0] == 0x03;
            odd = pub[0] == 0x03;
            be32_to_limbs(x.v, pub + 1);
        } else {
            uint32_t pw[8];
            load_words8(pw, a.s_pubs + 32ull * i);
            words_be_to_limbs(x.v, pw);
            ok = true;
        }
        ok = ok && limbs_lt_p(x.v);
        uint32_t slot = kNoSlot;
        if (ok) {
            bool claimed;
            slot = key_resolve(a.cache, a.cache_mask, x, odd, &claimed);
            if (claimed) a.todo[atomicAdd(a.todo_count, 1u)] = slot;
            looked = true;
            hit = slot != kNoSlot && !claimed;
        }
        (is_e ? a.e_slot : a.s_slot)[i] = slot;
    }
    if (a.cache_stats) {
        const uint32_t nl = __reduce_add_sync(0xFFFFFFFFu, looked ? 1u : 0u);
        const uint32_t nh = __reduce_add_sync(0xFFFFFFFFu, hit ? 1u : 0u);
        if ((threadIdx.x & 31u) == 0 && nl) {
            atomicAdd(&a.cache_stats[0], (unsigned long long)nl);
            atomicAdd(&a.cache_stats[1], (unsigned long long)nh);
        }
    }
}

// A thread per entry of this launch's to-do list, strided over the grid:
// decompress the slot's key and build its table in place (READY), or mark an x
// off the curve BAD.  Every thread runs the same instruction stream.
constexpr int kBuildThreads = 128;

__global__ void __launch_bounds__(kBuildThreads)
k_key_build(QueueArgs a) {
    extern __shared__ uint4 smem[];
    const EisTab tab{reinterpret_cast<double2*>(smem) + threadIdx.x, kBuildThreads};
    const uint32_t n = *a.todo_count;
    for (uint32_t k = blockIdx.x * kBuildThreads + threadIdx.x; k < n; k += gridDim.x * kBuildThreads) {
        PubCacheSlot* slot = a.cache + a.todo[k];
        Fe x, y;
        for (int q = 0; q < 8; ++q) x.v[q] = slot->key[q];
        if (!lift_x_parity(y, x, slot->key[8] != 0)) {
            slot_publish(*slot, kSlotBad);
            continue;
        }
        Fd px, py;
        fd_unpack(px, x.v);
        fd_unpack(py, y.v);
        fd_strict(px);
        fd_strict(py);
        const Fd zc = eis_table(tab, px, py);
        Fe zi;
        fd_pack(zi.v, zc);
        fe_inv(zi, zi);
        Fd z1, z2, z3;
        fd_unpack(z1, zi.v);
        fd_strict(z1);
        z2 = fdc_sqr(z1);
        z3 = fdc_mul(z2, z1);
        UF_NOUNROLL
        for (int e = 0; e < kEisTab; ++e) {
            Fd ex, ey;
            Fe wx = x, wy = y;          // entry 0 is the key itself
            if (e > 0) {
                tab.load(e, ex, ey);
                fd_pack(wx.v, fdc_mul(ex, z2));
                fd_pack(wy.v, fdc_mul(ey, z3));
            }
            uint4* q = slot->tab + 4 * e;
            q[0] = make_uint4(wx.v[0], wx.v[1], wx.v[2], wx.v[3]);
            q[1] = make_uint4(wx.v[4], wx.v[5], wx.v[6], wx.v[7]);
            q[2] = make_uint4(wy.v[0], wy.v[1], wy.v[2], wy.v[3]);
            q[3] = make_uint4(wy.v[4], wy.v[5], wy.v[6], wy.v[7]);
        }
        slot_publish(*slot, kSlotReady);
    }
}

static cudaError_t launch_key_passes(const QueueArgs& a, int sms, cudaStream_t s) {
    const uint64_t items = (uint64_t)a.cap_e + a.cap_s;
    if (!a.cache || items == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((items + 127) / 128);
    k_key_resolve<<<blocks, 128, 0, s>>>(a);
    const unsigned grid = blocks < 2u * (unsigned)sms ? blocks : 2u * (unsigned)sms;
    k_key_build<<<grid, kBuildThreads, kBuildThreads * kFpSmemPerThread, s>>>(a);
    return cudaGetLastError();
}

// kKind 0 ECDSA, 1 BIP-340.  kCached: the item's key table may come from its
// resolved slot.
constexpr int kQueueThreads = 256;

template <bool kCached, int kKind>
__global__ void __launch_bounds__(kQueueThreads, 1)
k_verify_queue(QueueArgs a, const uint4* __restrict__ gt, const uint4* __restrict__ comb) {
    extern __shared__ uint4 smem[];
    const uint32_t total = kKind == 0 ? min(a.counts[0], a.cap_e) : min(a.counts[1], a.cap_s);
    if (blockIdx.x * blockDim.x >= total) return;          // the whole block
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < total;
    const PubCacheSlot* slot = nullptr;
    if (kCached && valid) {
        const uint32_t si = (kKind == 0 ? a.e_slot : a.s_slot)[i];
        if (si != kNoSlot) slot = a.cache + si;
    }
    const bool ok = fp_verify<kKind, kCached>((kKind == 0 ? a.e_msgs : a.s_msgs) + 32ull * i,
                                              kKind == 0 ? a.e_pubs + 33ull * i : a.s_pubs + 32ull * i,
                                              (kKind == 0 ? a.e_sigs : a.s_sigs) + 64ull * i, valid, slot, gt, comb,
                                              smem);
    if (valid) (kKind == 0 ? a.e_out : a.s_out)[i] = ok ? 1 : 0;
}

template <int kKind, int kWarps>
__global__ void __launch_bounds__(kWarps * kTeamLanes, 8 / kWarps)
k_verify_queue_team(QueueArgs a, const uint4* __restrict__ gt, const uint4* __restrict__ comb) {
    extern __shared__ uint4 smem[];
    const uint32_t total = kKind == 0 ? min(a.counts[0], a.cap_e) : min(a.counts[1], a.cap_s);
    if (blockIdx.x * kTeamLanes >= total) return;          // the whole block
    const uint32_t i = blockIdx.x * kTeamLanes + (threadIdx.x & 31u);
    const bool ok = team_verify<kKind, kWarps>((kKind == 0 ? a.e_msgs : a.s_msgs) + 32ull * i,
                                       kKind == 0 ? a.e_pubs + 33ull * i : a.s_pubs + 32ull * i,
                                       (kKind == 0 ? a.e_sigs : a.s_sigs) + 64ull * i, i < total, gt, comb, smem);
    if (threadIdx.x < kTeamLanes && i < total) (kKind == 0 ? a.e_out : a.s_out)[i] = ok ? 1 : 0;
}

cudaError_t launch_verify_queue(const QueueArgs& a, int team_warps, const void* d_gtab, const void* d_comb, int sms,
                                const QueueStreams& q) {
    const uint4* gt = reinterpret_cast<const uint4*>(d_gtab);
    const uint4* comb = reinterpret_cast<const uint4*>(d_comb);
    cudaError_t e = cudaSuccess;
    const bool team = team_warps != 0;
    const bool both = a.cap_e > 0 && a.cap_s > 0;
    if (!team && (e = launch_key_passes(a, sms, q.main)) != cudaSuccess) return e;
    const bool beside = team && a.cache;                   // the key passes on a branch of their own
    if (both || beside) {
        if ((e = cudaEventRecord(q.fork, q.main)) != cudaSuccess) return e;
        if (both && (e = cudaStreamWaitEvent(q.second, q.fork, 0)) != cudaSuccess) return e;
        if (beside && (e = cudaStreamWaitEvent(q.third, q.fork, 0)) != cudaSuccess) return e;
    }
    cudaStream_t ss = both ? q.second : q.main;
    if (team) {
        const unsigned ge = (a.cap_e + kTeamLanes - 1) / kTeamLanes, gs = (a.cap_s + kTeamLanes - 1) / kTeamLanes;
        if (team_warps == 4) {
            if (ge) k_verify_queue_team<0, 4><<<ge, kTeamThreads, kTeamSmem, q.main>>>(a, gt, comb);
            if (gs) k_verify_queue_team<1, 4><<<gs, kTeamThreads, kTeamSmem, ss>>>(a, gt, comb);
        } else {
            if (ge) k_verify_queue_team<0, 2><<<ge, kDuoThreads, kTeamSmem, q.main>>>(a, gt, comb);
            if (gs) k_verify_queue_team<1, 2><<<gs, kDuoThreads, kTeamSmem, ss>>>(a, gt, comb);
        }
    } else {
        // full blocks, one per SM, for launches that fill the device; two half
        // blocks per SM where both kinds or a part of a wave share it
        const uint32_t threads = (a.cap_e > a.cap_s ? a.cap_e : a.cap_s) > (uint32_t)sms * 128u ? kQueueThreads : 128;
        const size_t smem = threads * kFpSmemPerThread;
        const unsigned ge = (a.cap_e + threads - 1) / threads, gs = (a.cap_s + threads - 1) / threads;
        if (ge && a.cache) k_verify_queue<true, 0><<<ge, threads, smem, q.main>>>(a, gt, comb);
        else if (ge) k_verify_queue<false, 0><<<ge, threads, smem, q.main>>>(a, gt, comb);
        if (gs && a.cache) k_verify_queue<true, 1><<<gs, threads, smem, ss>>>(a, gt, comb);
        else if (gs) k_verify_queue<false, 1><<<gs, threads, smem, ss>>>(a, gt, comb);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (both) {
        if ((e = cudaEventRecord(q.join, q.second)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(q.main, q.join, 0)) != cudaSuccess) return e;
    }
    if (beside) {
        if ((e = launch_key_passes(a, sms, q.third)) != cudaSuccess) return e;
        if ((e = cudaEventRecord(q.join3, q.third)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(q.main, q.join3, 0)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t verify_queue_init() {
    cudaError_t e = cudaSuccess;
    auto opt_in = [&](auto f, size_t bytes) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    const size_t full = kQueueThreads * kFpSmemPerThread;
    opt_in(k_verify_queue<false, 0>, full);
    opt_in(k_verify_queue<false, 1>, full);
    opt_in(k_verify_queue<true, 0>, full);
    opt_in(k_verify_queue<true, 1>, full);
    opt_in(k_verify_queue_team<0, 4>, kTeamSmem);
    opt_in(k_verify_queue_team<1, 4>, kTeamSmem);
    opt_in(k_verify_queue_team<0, 2>, kTeamSmem);
    opt_in(k_verify_queue_team<1, 2>, kTeamSmem);
    opt_in(k_key_build, kBuildThreads * kFpSmemPerThread);
    return e;
}

}  // namespace uf
