// Per-signature verify kernel on the FP64 pipe, the path of large calls.
//
// A thread verifies one signature: R = a G + b P with the key's multiple summed
// by joint digits of its GLV halves (eis.cuh) on the curve scaled by the key's
// unknown y, so that no square root is taken (isocheck.cuh), the generator's
// multiple summed from a table of all windows, the field arithmetic in doubles
// (fd.cuh).  The verdicts are those of ecdsa_verify_one / ecdsa_verify_opaque_one
// / schnorr_verify_one (verify.cuh); what the scaled form does not cover (a sum
// or an operand at infinity, equal x coordinates, an ECDSA r that may stand for
// r + n) takes those functions themselves.
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

namespace uf {
namespace {

constexpr int kFpThreads = 256;
constexpr size_t kFpSmemPerThread = (size_t)kEisTab * 80;

// A thread's 11-point table: [entry][5 pairs of doubles][thread], so that a
// thread's reads stay in its own 16-byte column (no bank conflict whatever the
// lanes' digits are).
struct EisTab {
    double2* base;
    uint32_t stride;
    __device__ __forceinline__ void store(int k, const Fd& x, const Fd& y) const {
        double2* p = base + (uint32_t)(k * 5) * stride;
        p[0] = make_double2(x.v[0], x.v[1]);
        p[stride] = make_double2(x.v[2], x.v[3]);
        p[2 * stride] = make_double2(x.v[4], y.v[0]);
        p[3 * stride] = make_double2(y.v[1], y.v[2]);
        p[4 * stride] = make_double2(y.v[3], y.v[4]);
    }
    __device__ __forceinline__ void load(int k, Fd& x, Fd& y) const {
        const double2* p = base + (uint32_t)(k * 5) * stride;
        const double2 a = p[0], b = p[stride], c = p[2 * stride], d = p[3 * stride], e = p[4 * stride];
        x.v[0] = a.x; x.v[1] = a.y; x.v[2] = b.x; x.v[3] = b.y; x.v[4] = c.x;
        y.v[0] = c.y; y.v[1] = d.x; y.v[2] = d.y; y.v[3] = e.x; y.v[4] = e.y;
    }
};

// One item by the plain per-thread verification (rare): its 512-byte table lies
// in the thread's own column of the same shared memory.
template <int kKind>
__device__ __noinline__ bool plain_verify(const uint8_t* msgs, const uint8_t* pubs, const uint8_t* sigs, uint32_t i,
                                          const uint4* gt, uint4* smem) {
    SmemTab tab{smem + threadIdx.x, blockDim.x};
    const GlobalGT g{gt};
    uint32_t mw[8], sw[16];
    load_words8(mw, msgs + 32ull * i);
    load_words8(sw, sigs + 64ull * i);
    load_words8(sw + 8, sigs + 64ull * i + 32);
    if (kKind == 0) return ecdsa_verify_one(mw, pubs + 33ull * i, sw, tab, g);
    if (kKind == 2) return ecdsa_verify_opaque_one(mw, pubs + 33ull * i, sw, tab, g);
    uint32_t pw[8];
    load_words8(pw, pubs + 32ull * i);
    return schnorr_verify_one(mw, pw, sw, tab, g);
}

// kKind: 0 ECDSA (compact r || s, low-S), 1 BIP-340, 2 ECDSA (opaque
// little-endian r, s; high-S normalised).
template <int kKind>
__global__ void __launch_bounds__(kFpThreads, 1)
k_verify_fp(const uint8_t* __restrict__ msgs, const uint8_t* __restrict__ pubs, const uint8_t* __restrict__ sigs,
             uint32_t n, const uint4* __restrict__ gt, const uint4* __restrict__ comb, uint8_t* __restrict__ out,
             int collect) {
    extern __shared__ uint4 smem[];
    const EisTab tab{reinterpret_cast<double2*>(smem) + threadIdx.x, blockDim.x};
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool ok = i < n, odd = false;
    uint32_t px[8], r[8];
    Sc s, b;             // R = s G + b P
    uint8_t dig[kEisDigits];
    if (kKind == 1) {
        // BIP-340: parse and challenge (schnorr_verify_one)
        if (ok) {
            uint32_t mw[8], sw[16], pw[8];
            load_words8(mw, msgs + 32ull * i);
            load_words8(sw, sigs + 64ull * i);
            load_words8(sw + 8, sigs + 64ull * i + 32);
            load_words8(pw, pubs + 32ull * i);
            words_be_to_limbs(r, sw);
            words_be_to_limbs(s.v, sw + 8);
            words_be_to_limbs(px, pw);
            ok = limbs_lt_p(r) && !sc_is_zero(s) && limbs_lt_n(s.v) && limbs_lt_p(px);
            uint32_t rbe[8], pbe[8], mbe[8], h[8];
            UF_UNROLL
            for (int k = 0; k < 8; ++k) {
                rbe[k] = bswap32(sw[k]);
                pbe[k] = bswap32(pw[k]);
                mbe[k] = bswap32(mw[k]);
            }
            bip340_challenge(h, rbe, pbe, mbe);
            Sc e;
            UF_UNROLL
            for (int k = 0; k < 8; ++k) e.v[k] = h[7 - k];
            sc_reduce_once(e);
            sc_neg(b, e);
        }
    } else {
        // ECDSA: parse, u1 and u2
        if (ok) {
            uint32_t sw[16];
            load_words8(sw, sigs + 64ull * i);
            load_words8(sw + 8, sigs + 64ull * i + 32);
            if (kKind == 0) {
                words_be_to_limbs(r, sw);
                words_be_to_limbs(s.v, sw + 8);
            } else {
                UF_UNROLL
                for (int k = 0; k < 8; ++k) {
                    r[k] = sw[k];
                    s.v[k] = sw[8 + k];
                }
            }
            ok = !is_zero256(r) && limbs_lt_n(r) && !sc_is_zero(s) && limbs_lt_n(s.v);
            if (ok) {
                if (kKind == 0) ok = sc_is_low(s.v);
                else if (!sc_is_low(s.v)) sc_neg(s, s);
            }
            const uint8_t* pub = pubs + 33ull * i;
            const uint8_t prefix = pub[0];
            odd = prefix == 0x03;
            be32_to_limbs(px, pub + 1);
            ok = ok && (prefix == 0x02 || prefix == 0x03) && limbs_lt_p(px);
        }
        if (ok) {
            uint32_t mw[8];
            load_words8(mw, msgs + 32ull * i);
            Sc z, rs;
            words_be_to_limbs(z.v, mw);
            sc_reduce_once(z);
            UF_UNROLL
            for (int k = 0; k < 8; ++k) rs.v[k] = r[k];
            Sc w;
            sc_inv(w, s);
            sc_mul(s, z, w);
            sc_mul(b, rs, w);
        }
    }
    Fd c, den, zc;
    JacD A;
    bool plain = false;      // left to the plain verification
    __syncthreads();
    if (ok) {
        GlvSplit split;
        glv_split(split, b);
        eis_recode(dig, split);
        Fd kx, ky;
        iso_key(kx, ky, c, px);
        zc = eis_table(tab, kx, ky);
    }
    jacd_set_inf(A);
    __syncthreads();
    UF_NOUNROLL
    for (int q = kEisDigits - 1; q >= 0; --q) {
        if (ok) eis_add_digit(A, dig[q], q == kEisDigits - 1, tab);
    }
    __syncthreads();
    if (ok) {
        A.Z = fdc_mul(A.Z, zc);
        if (kKind == 1) {
            uint32_t sw[8];
            load_words8(sw, sigs + 64ull * i + 32);
            words_be_to_limbs(s.v, sw);
        }
        const JacD B = comb_mul(s, comb);
        if (kKind == 1) {
            // s went into B; r from the signature again
            uint32_t sw[8];
            load_words8(sw, sigs + 64ull * i);
            words_be_to_limbs(r, sw);
        }
        plain = !iso_prepare<kKind == 1>(tab, den, A, B, c, r);
    }
    __syncthreads();
    if (ok && !plain) {
        Fe inv;
        fd_pack(inv.v, den);
        if (is_zero256(inv.v)) {
            plain = true;
        } else {
            fe_inv(inv, inv);
            ok = iso_finish<kKind == 1>(tab, inv, odd);
            // x(R) may be r + n: the plain check looks at both
            if (kKind != 1 && !ok && r_below_p_minus_n(r)) ok = plain = true;
        }
    }
    if (ok && plain) ok = plain_verify<kKind>(msgs, pubs, sigs, i, gt, smem);
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
