// Per-signature verify kernel on the FP64 pipe, the path of large calls.
//
// A thread verifies one signature: R = a G + b P with the key's multiple summed
// by joint digits of its GLV halves (eis.cuh) on the curve scaled by the key's
// unknown y, so that no square root is taken (isocheck.cuh), the generator's
// multiple summed from a table of all windows, the field arithmetic in doubles
// (fd.cuh).  The verdicts are those of ecdsa_verify_one / ecdsa_verify_opaque_one
// / schnorr_verify_one (verify.cuh); sums that meet or vanish and an ECDSA r that
// may stand for r + n are decided in the scaled form too (isocheck.cuh), and those
// functions themselves take only a BIP-340 challenge of 0.
//
// One block of 256 threads per SM, one item per thread: a thread's table is 11
// points of ten doubles, 880 bytes of shared memory, read without conversion.
// The kernel is bound by register-file reads (a 64-bit operand takes both banks
// for a cycle; an FP64 multiply-add of three registers issues every 3.1 cycles)
// and by instruction fetch: the main loop alone is 60 KB of code, so the block's
// warps are kept at the same place by a barrier before each phase, which serves
// nothing else.  Measured over 16 rounds (BIP-340, sigs/s): 43.5 M with two
// independent blocks of 128 threads, 46.2 M with barriers in them, 55.5 M with one
// block of 256; the integer kernel with shared inversions that this replaces ran
// at 36.5 M.
#include "kernels.h"
#include "verify.cuh"
#include "dev_tables.cuh"
#include "isocheck.cuh"
#include "verify_fp.cuh"

namespace uf {
namespace {

constexpr int kFpThreads = 256;

// kKind: 0 ECDSA (compact r || s, low-S), 1 BIP-340, 2 ECDSA (opaque
// little-endian r, s; high-S normalised).
template <int kKind>
__global__ void __launch_bounds__(kFpThreads, 1)
k_verify_fp(const uint8_t* __restrict__ msgs, const uint8_t* __restrict__ pubs, const uint8_t* __restrict__ sigs,
             uint32_t n, const uint4* __restrict__ gt, const uint4* __restrict__ comb, uint8_t* __restrict__ out,
             int collect) {
    extern __shared__ uint4 smem[];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool ok = fp_verify<kKind, false>(msgs + 32ull * i, pubs + (kKind == 1 ? 32ull : 33ull) * i, sigs + 64ull * i,
                                            i < n, nullptr, gt, comb, smem);
    if (i < n) {
        if (collect) {
            if (ok) out[i] = 0;
        } else {
            out[i] = ok ? 1 : 0;
        }
    }
}

}  // namespace

cudaError_t launch_verify_fp(int kind, const uint8_t* msgs, const uint8_t* pubs, const uint8_t* sigs, uint32_t n,
                             const void* d_gtab, const void* d_comb, uint8_t* out, int collect, int sms,
                             cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint4* gt = reinterpret_cast<const uint4*>(d_gtab);
    const uint4* comb = reinterpret_cast<const uint4*>(d_comb);
    // fewer items than one full block per SM: smaller blocks on every SM
    const uint32_t per_sm = (n + (uint32_t)sms - 1) / (uint32_t)sms;
    const uint32_t threads = per_sm >= (uint32_t)kFpThreads ? (uint32_t)kFpThreads : (per_sm + 31) / 32 * 32;
    const uint32_t grid = (n + threads - 1) / threads;
    const size_t smem = (size_t)threads * kFpSmemPerThread;
    if (kind == 0) k_verify_fp<0><<<grid, threads, smem, s>>>(msgs, pubs, sigs, n, gt, comb, out, collect);
    else if (kind == 2) k_verify_fp<2><<<grid, threads, smem, s>>>(msgs, pubs, sigs, n, gt, comb, out, collect);
    else k_verify_fp<1><<<grid, threads, smem, s>>>(msgs, pubs, sigs, n, gt, comb, out, collect);
    return cudaGetLastError();
}

cudaError_t verify_fp_init() {
    cudaError_t e = cudaSuccess;
    auto opt_in = [&](auto f) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(kFpThreads * kFpSmemPerThread));
    };
    opt_in(k_verify_fp<0>);
    opt_in(k_verify_fp<1>);
    opt_in(k_verify_fp<2>);
    return e;
}

}  // namespace uf
