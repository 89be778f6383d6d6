// The verify kernels' body on the FP64 pipe (kernels_verify_fp.cu, kernels_queue.cu)
// and the pieces it shares with the small-call form (team.cuh).
#pragma once
#include "dev_tables.cuh"
#include "isocheck.cuh"
#include "pubcache.cuh"
#include "verify.cuh"

#if defined(__CUDACC__)
namespace uf {

constexpr size_t kFpSmemPerThread = (size_t)kEisTab * 80;   // one point table

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
// in the thread's own column (smem, stride) of the same shared memory.
template <int kKind>
static __device__ __noinline__ bool plain_verify(const uint8_t* msg, const uint8_t* pub, const uint8_t* sig,
                                                 const uint4* gt, uint4* column, uint32_t stride) {
    SmemTab tab{column, stride};
    const GlobalGT g{gt};
    uint32_t mw[8], sw[16];
    load_words8(mw, msg);
    load_words8(sw, sig);
    load_words8(sw + 8, sig + 32);
    if (kKind == 0) return ecdsa_verify_one(mw, pub, sw, tab, g);
    if (kKind == 2) return ecdsa_verify_opaque_one(mw, pub, sw, tab, g);
    uint32_t pw[8];
    load_words8(pw, pub);
    return schnorr_verify_one(mw, pw, sw, tab, g);
}

// Key and signature of one item: px the key's x, odd its wanted parity, r and s
// (ECDSA's opaque form with high s normalised); false when the item fails a
// range check (verify.cuh).
template <int kKind>
__device__ __forceinline__ bool fp_parse_key(uint32_t px[8], bool& odd, const uint8_t* pub) {
    if (kKind == 1) {
        uint32_t pw[8];
        load_words8(pw, pub);
        words_be_to_limbs(px, pw);
        odd = false;
        return limbs_lt_p(px);
    }
    const uint8_t prefix = pub[0];
    odd = prefix == 0x03;
    be32_to_limbs(px, pub + 1);
    return (prefix == 0x02 || prefix == 0x03) && limbs_lt_p(px);
}

template <int kKind>
__device__ __forceinline__ bool fp_parse_sig(uint32_t r[8], Sc& s, const uint8_t* sig) {
    uint32_t sw[16];
    load_words8(sw, sig);
    load_words8(sw + 8, sig + 32);
    if (kKind == 2) {
        UF_UNROLL
        for (int k = 0; k < 8; ++k) {
            r[k] = sw[k];
            s.v[k] = sw[8 + k];
        }
    } else {
        words_be_to_limbs(r, sw);
        words_be_to_limbs(s.v, sw + 8);
    }
    if (sc_is_zero(s) || !limbs_lt_n(s.v)) return false;
    if (kKind == 1) return limbs_lt_p(r);
    if (is_zero256(r) || !limbs_lt_n(r)) return false;
    if (!sc_is_low(s.v)) {
        if (kKind == 0) return false;
        sc_neg(s, s);
    }
    return true;
}

// The two scalars of R = a G + b P from a parsed signature.
template <int kKind>
__device__ __forceinline__ void fp_scalars(Sc& a, Sc& b, const uint32_t r[8], const Sc& s, const uint8_t* msg,
                                           const uint8_t* pub, const uint8_t* sig) {
    uint32_t mw[8];
    load_words8(mw, msg);
    if (kKind == 1) {
        uint32_t rw[8], pw[8], h[8];
        load_words8(rw, sig);
        load_words8(pw, pub);
        UF_UNROLL
        for (int k = 0; k < 8; ++k) {
            rw[k] = bswap32(rw[k]);
            pw[k] = bswap32(pw[k]);
            mw[k] = bswap32(mw[k]);
        }
        bip340_challenge(h, rw, pw, mw);
        Sc e;
        UF_UNROLL
        for (int k = 0; k < 8; ++k) e.v[k] = h[7 - k];
        sc_reduce_once(e);
        a = s;
        sc_neg(b, e);
    } else {
        Sc z, rs, w;
        words_be_to_limbs(z.v, mw);
        sc_reduce_once(z);
        UF_UNROLL
        for (int k = 0; k < 8; ++k) rs.v[k] = r[k];
        sc_inv(w, s);
        sc_mul(a, z, w);
        sc_mul(b, rs, w);
    }
}

// One item per thread; every thread of the block calls it (ok false for threads
// without one, whose pointers are not read).  smem: blockDim.x point tables.
// The barriers keep the block's warps at the same place in the code and serve
// nothing else.  kCached: `slot` may hold the key's table (pubcache.cuh); null
// or a slot that is not ready yet: the key's table is built here.
template <int kKind, bool kCached>
__device__ __forceinline__ bool fp_verify(const uint8_t* msg, const uint8_t* pub, const uint8_t* sig, bool ok,
                                          const PubCacheSlot* slot, const uint4* gt, const uint4* comb, uint4* smem) {
    const EisTab tab{reinterpret_cast<double2*>(smem) + threadIdx.x, blockDim.x};
    bool odd = false;
    uint32_t px[8], r[8];
    Sc a, b;             // R = a G + b P
    uint8_t dig[kEisDigits];
    if (ok) {
        Sc s;
        ok = fp_parse_sig<kKind>(r, s, sig) && fp_parse_key<kKind>(px, odd, pub);
        if (ok) fp_scalars<kKind>(a, b, r, s, msg, pub, sig);
    }
    Fd c, den, zc;
    JacD A;
    int st = kIsoNo;
    bool unit = false;       // the key's table comes from its slot
    if (kCached && ok && slot) {
        const uint32_t state = slot_state(*slot);
        unit = state == kSlotReady;
        if (state == kSlotBad) ok = false;
    }
    __syncthreads();
    if (ok) {
        GlvSplit split;
        glv_split(split, b);
        eis_recode(dig, split);
        if (kCached && unit) {
            UF_NOUNROLL
            for (int k = 0; k < kEisTab; ++k) {
                const uint4 x0 = slot->tab[4 * k], x1 = slot->tab[4 * k + 1], y0 = slot->tab[4 * k + 2],
                            y1 = slot->tab[4 * k + 3];
                const uint32_t xw[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
                const uint32_t yw[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
                Fd x, y;
                fd_unpack(x, xw);
                fd_unpack(y, yw);
                tab.store(k, x, y);
            }
            fd_set_u32(c, 1);
            fd_set_u32(zc, 1);
        } else {
            Fd kx, ky;
            iso_key(kx, ky, c, px);
            zc = eis_table(tab, kx, ky);
            ok = !fd_is_zero(zc);        // 0: the key is not on the curve (isocheck.cuh)
        }
    }
    jacd_set_inf(A);
    __syncthreads();
    UF_NOUNROLL
    for (int q = kEisDigits - 1; q >= 0; --q) {
        if (ok) eis_add_digit<false>(A, dig[q], q == kEisDigits - 1, tab);
    }
    __syncthreads();
    if (ok) {
        A.Z = fdc_mul(A.Z, zc);
        if (kKind == 1) {
            // the scalar and r again from the signature: not held over the main loop
            uint32_t sw[8];
            load_words8(sw, sig + 32);
            words_be_to_limbs(a.v, sw);
        }
        const JacD B = comb_mul<false>(a, comb);
        if (kKind == 1) {
            uint32_t sw[8];
            load_words8(sw, sig);
            words_be_to_limbs(r, sw);
        }
        st = iso_prepare<kKind == 1>(tab, den, A, B, c, r);
        if (kKind == 1 && st == kIsoKeyInf) {
            st = kIsoPlain;                     // e = 0, unless the key is not on the curve
            for (int q = 0; q < kEisDigits; ++q)
                if (dig[q] != kEisZero) st = kIsoNo;
        }
    }
    __syncthreads();
    bool holds = false;
    if (st == kIsoSolve) {
        Fe inv;
        fd_pack(inv.v, den);
        if (is_zero256(inv.v)) {
            st = kIsoPlain;
        } else {
            fe_inv(inv, inv);
            holds = iso_finish<kKind == 1>(tab, inv, odd, unit, kKind != 1 && r_below_p_minus_n(r));
        }
    }
    if (kKind != 1 && st == kIsoOnCurve) holds = iso_on_curve(tab);
    if (st == kIsoPlain) holds = plain_verify<kKind>(msg, pub, sig, gt, smem + threadIdx.x, blockDim.x);
    return holds;
}

}  // namespace uf
#endif  // __CUDACC__
