// k P for one variable point by joint digits of the two GLV halves.
//
// k = k1 + k2 lambda with lambda^2 + lambda + 1 = 0, so k1 + k2 lambda is an
// element z of the Eisenstein integers Z[w] (w = lambda), and w P = (beta x, y).
// z is written in base 8 with digits from the 63 nonzero residues mod 8, each
// represented by its element of least norm: the six units +-1, +-w, +-w^2 act on
// a point by a sign and a factor beta^e of x, and up to them 11 digits remain.
// So a table of 11 points gives one addition per three doublings for both
// halves: 43 + 1 additions for 129 doublings, where two 4-bit window streams
// take 66 additions (and 33 multiplications by beta, against 44 here).
//
// The 11 table points form a path with unit steps,
//   1, 1-w, 2-w, 3-w, 3, 4, 4+w, 5+2w, 4+2w, 3+w, 2,
// so each is the one before plus a unit multiple of P: ten mixed additions, no
// doubling.
#pragma once
#include "common.cuh"
#include "fn.cuh"
#include "jacd.cuh"

namespace uf {

constexpr int kEisDigits = 44;      // |z| < 2^128.8: 43 base-8 digits and a last one of 0 or a unit
constexpr int kEisTab = 11;
constexpr uint32_t kEisZero = 15;   // digit byte of 0

// A digit byte: table entry in bits 0..3, e of beta^e in bits 4..5, sign in bit 6.
// LUT by (k1 mod 8) + 8 (k2 mod 8): the digit byte, and in bits 7 and 8 what the
// digit borrows from the next windows of k1 and k2.
#if defined(__CUDACC__)
__device__ const
#else
static const
#endif
uint16_t kEisLut[64] = {
    15, 0, 10, 4, 5, 196, 202, 192, 16, 96, 97, 9, 6, 195, 194, 193, 26, 17, 106, 98, 8, 7,
    152, 153, 20, 18, 105, 100, 99, 423, 151, 150, 21, 19, 104, 102, 421, 422, 424, 467, 340, 342,
    343, 103, 419, 420, 425, 466, 346, 345, 344, 455, 456, 418, 426, 465, 336, 257, 258, 259, 454, 457,
    417, 416};

// Steps of the table path: e | sign << 2 of the unit added to reach entry
// k = 1..10 (5, 0, 0, 1, 0, 1, 6, 4, 2, 2), three bits each.
UF_HD uint32_t eis_step(int k) {
    const uint32_t steps = 05u | 00u << 3 | 00u << 6 | 01u << 9 | 00u << 12 | 01u << 15 | 06u << 18 | 04u << 21 |
                           02u << 24 | 02u << 27;
    return (steps >> (3 * (k - 1))) & 7u;
}

// Signed 132-bit window source of a GLV half.
UF_HD void eis_signed(uint32_t w[5], const uint32_t k[4], bool neg) {
    const uint32_t m = neg ? 0xFFFFFFFFu : 0u;
    uint64_t c = neg ? 1 : 0;
    UF_UNROLL
    for (int i = 0; i < 4; ++i) {
        c += (uint64_t)(k[i] ^ m);
        w[i] = lo32(c);
        c >>= 32;
    }
    w[4] = lo32(c + m);
}

// Digit bytes of z = k1 + k2 w, least significant first.
UF_HDI void eis_recode(uint8_t dig[kEisDigits], const GlvSplit& s) {
    uint32_t a[5], b[5], ca = 0, cb = 0;
    eis_signed(a, s.k1, s.neg1);
    eis_signed(b, s.k2, s.neg2);
    UF_NOUNROLL
    for (int i = 0; i < kEisDigits; ++i) {
        const uint32_t u = (a[0] & 7u) + ca, v = (b[0] & 7u) + cb;
        const uint32_t e = kEisLut[(u & 7u) + 8u * (v & 7u)];
        dig[i] = (uint8_t)(e & 0x7Fu);
        ca = (u >> 3) + ((e >> 7) & 1u);
        cb = (v >> 3) + (e >> 8);
        UF_UNROLL
        for (int j = 0; j < 4; ++j) {
            a[j] = (a[j] >> 3) | (a[j + 1] << 29);
            b[j] = (b[j] >> 3) | (b[j + 1] << 29);
        }
        a[4] = (uint32_t)((int32_t)a[4] >> 3);
        b[4] = (uint32_t)((int32_t)b[4] >> 3);
    }
}

// beta^e as strict digits (e = 0, 1, 2), padded to 48 bytes.
#if defined(__CUDACC__)
__device__ const
#else
static const
#endif
double kBetaPow[3][6] = {
    {1.0, 0.0, 0.0, 0.0, 0.0, 0.0},
    {-1851403876892178.0, 2059588628732948.0, -1068498044522423.0, 124274446989803.0, 135142927197564.0, 0.0},
    {1851403876892177.0, -2059588628732948.0, 1068498044522423.0, -124274446989803.0, -135142927197564.0, 0.0}};

UF_HD void fd_beta_pow(Fd& r, uint32_t e) {
    const double* p = kBetaPow[e];
    UF_UNROLL
    for (int i = 0; i < 5; ++i) r.v[i] = p[i];
}

// (x, y) times the unit beta^e, sign: x2 strict, y2 negated where neg.
template <bool kCalls>
UF_HD void eis_unit(Fd& x, Fd& y, uint32_t e, bool neg) {
    Fd b;
    fd_beta_pow(b, e);
    x = jf_mul<kCalls>(x, b);
    const double s = neg ? -1.0 : 1.0;
    UF_UNROLL
    for (int i = 0; i < 5; ++i) y.v[i] *= s;
}

// The table of P = (x, y) (strict digits, on any curve y^2 = x^3 + b) with every
// entry brought to the common Z of the last one: as affine points they lie on
// the curve scaled by that Z, which is returned; the point that eis_mul sums
// from them has its own Z times that one.  No inversion.
//
// The path's additions are co-Z additions: T and the step U = unit P share their
// Z, and U + T comes with U rescaled to the sum's Z (4M + 2S, the Z's themselves
// are never formed: Z grows by the factor H = x_U - x_T each time).  A second
// pass from the last entry down multiplies the entries up by the later H's
// (4M + 1S each).  (If an addition meets equal or opposite points, which a point
// of order n never does, H becomes 0 and everything computed from it too.)
//
// eis_path is the first pass (hs[k]: Z of entry k over Z of entry k - 1),
// eis_scale multiplies one entry by rho = Z of the last entry over its own.
template <class Tab>
UF_HDI void eis_path(const Tab& tab, const Fd& px, const Fd& py, Fd hs[kEisTab]) {
    Fd ux = px, uy = py, X = px, Y = py;
    uint32_t cur = 0;            // the unit that U holds
    tab.store(0, X, Y);
    UF_NOUNROLL
    for (int k = 1; k < kEisTab; ++k) {
        const uint32_t st = eis_step(k);
        uint32_t turn = (st & 3u) + 3u - (cur & 3u);
        turn -= turn >= 3u ? 3u : 0u;
        if (turn != 0) {         // the same step in every lane: no divergence
            Fd bt;
            fd_beta_pow(bt, turn);
            ux = fdc_mul(ux, bt);
        }
        if ((st ^ cur) & 4u) uy = fd_neg(uy);
        cur = st;
        const Fd H = fdc_sub(ux, X), G = fdc_sub(uy, Y);
        hs[k] = H;
        const Fd C = fdc_sqr(H);
        const Fd W1 = fdc_mul(ux, C), W2 = fdc_mul(X, C);
        uy = fdc_mul(fd_sub_l(W1, W2), uy);
        X = fdc_sqr_sub_sub(G, W1, W2);
        Y = fdc_mul_sub(fd_sub_l(W1, X), G, uy);
        ux = W1;
        tab.store(k, X, Y);
    }
}

template <class Tab>
UF_HDI void eis_scale(const Tab& tab, int k, const Fd& rho) {
    Fd X, Y;
    const Fd r2 = fdc_sqr(rho);
    tab.load(k, X, Y);
    X = fdc_mul(X, r2);
    Y = fdc_mul(Y, fdc_mul(r2, rho));
    tab.store(k, X, Y);
}

template <class Tab>
UF_HDI Fd eis_table(const Tab& tab, const Fd& px, const Fd& py) {
    Fd hs[kEisTab];
    eis_path(tab, px, py, hs);
    Fd rho = hs[kEisTab - 1];
    UF_NOUNROLL
    for (int k = kEisTab - 2; k >= 0; --k) {
        eis_scale(tab, k, rho);
        if (k > 0) rho = fdc_mul(rho, hs[k]);
    }
    return rho;
}

// One digit of the sum over the table, most significant first: R <- 8 R + digit
// (129 doublings and at most 44 additions in all).  kCalls as in jacd.cuh.
template <bool kCalls, class Tab>
UF_HD void eis_add_digit(JacD& R, uint32_t e, bool top, const Tab& tab) {
    if (!top) {
        UF_NOUNROLL
        for (int k = 0; k < 3; ++k) R = jacd_dbl_t<kCalls>(R);
    }
    if (e != kEisZero) {
        Fd x, y;
        tab.load((int)(e & 15u), x, y);
        eis_unit<kCalls>(x, y, (e >> 4) & 3u, (e & 64u) != 0);
        R = jacd_add_aff_t<kCalls>(R, x, y);
    }
}

template <class Tab>
UF_HD JacD eis_mul(const uint8_t* dig, const Tab& tab) {
    JacD R;
    jacd_set_inf(R);
    UF_NOUNROLL
    for (int i = kEisDigits - 1; i >= 0; --i) eis_add_digit<false>(R, dig[i], i == kEisDigits - 1, tab);
    return R;
}

}  // namespace uf
