// Signature check without the key's square root.
//
// A compressed or x-only key gives x and y^2 = c = x^3 + 7, and lift_x pays a
// 253-squaring chain for y.  Scaling secp256k1 by y (x -> x y^2, y -> y y^3)
// sends the key to (x c, c^2), which needs only c, on the isomorphic curve
// Y^2 = X^3 + 7 c^3.  So the key's multiple A = b P is summed there, the
// generator's multiple B = a G on secp256k1 itself from a table of all windows
// (no doublings), and the equation x(A + B) = r is solved for the unknown y:
// with Jacobian A = (a, b, za) on the scaled curve and B = (d, f, zb),
//   x_A = a / (c za^2),  y_A = y b / (c^2 za^3),  x_B = d / zb^2,  y_B = f / zb^3,
//   (y_B - y_A)^2 = (r + x_A + x_B)(x_B - x_A)^2 and y_A^2 = b^2 / (c^3 za^6)
// is linear in y:
//   y = M / (2 f b c za^3 zb^3),
//   M = f^2 cz^3 + b^2 zb^6 - (r cz zb^2 + a zb^2 + d cz) N^2,
//   cz = c za^2,  N = d cz - a zb^2.
// The signature's x-equation holds for the key with that parity exactly when
// this y satisfies y^2 = c and has the parity; y^2 = c also shows that x is on
// the curve (for a c that is no square no y passes).  BIP-340's y(R) follows as
//   y_R = [(f c^2 za^3 - y b zb^3)(d - r zb^2) - f c za N] / (c za zb^3 N).
// One inversion serves both.
//
// It needs A, B finite and x_A != x_B, and ECDSA's r may stand for r + n.  Only
// crafted items meet these cases, but anyone can craft them, and one such item in
// a block that verified it again alone held the block's SM for a second verify's
// latency (1 % of them in 2^20 device-resident signatures: 47.4 - 49.4 ms against
// 18.6).  So they take the same inversion, or none:
//   x(R) = r + n: M is linear in r, so y(r + n) = (M - n cz zb^2 N^2) / g1.
//   N = 0: y_A^2 = y_B^2 holds for either square root of c, so A = B or A = -B
//     according to the parity of  y = f c^2 za^3 / (b zb^3);  then R = 2 B or
//     infinity, and x(2 B), y(2 B) are compared (iso_meet; 1 % 19.1 ms).
//   B infinite (ECDSA of a digest 0 mod n): x_A = r; that c is a square is looked at
//     only where it holds (kIsoOnCurve; 1 % of such valid items 22.7 ms).
//   A table whose Z is 0, or A infinite with b != 0: on secp256k1, whose order is a
//     prime, neither happens (the table's path adds multiples of different small
//     norm), so the key is not on it (1 % of points of small order 18.5 ms).
#pragma once
#include "common.cuh"
#include "eis.cuh"
#include "verify.cuh"

namespace uf {

// Generator windows: s G = sum of 16 table points, table[i][m - 1] = m 2^(16 i) G
// for m = 1..2^15 (signed 16-bit digits; 32 MB, resident in L2).  Against the
// interleaved 20-bit G and lambda G windows (14 additions) two more additions,
// but no doubling is tied to them, so they can follow a key sum on another curve.
constexpr int kCombWindows = 16;
constexpr int kCombTab = 1 << 15;
constexpr size_t kCombBytes = (size_t)kCombWindows * kCombTab * 64;

#if defined(__CUDACC__)

// Windows [first, last) of s G (all of them: 0, kCombWindows).  kCalls as in jacd.cuh.
template <bool kCalls>
__device__ __forceinline__ JacD comb_mul(Sc s, const uint4* __restrict__ comb, int first = 0,
                                         int last = kCombWindows) {
    JacD B;
    Sc k = s;
    const bool flip = !sc_is_low(s.v);         // |k| < 2^255: the last window takes no carry out
    if (flip) sc_neg(k, s);
    jacd_set_inf(B);
    uint32_t carry = 0;
    UF_NOUNROLL
    for (int i = 0; i < last; ++i) {
        const uint32_t w = (k.v[0] & 0xFFFFu) + carry;
        carry = w > (uint32_t)kCombTab ? 1u : 0u;
        const int d = (int)w - (int)(carry << 16);
        UF_UNROLL
        for (int j = 0; j < 7; ++j) k.v[j] = (k.v[j] >> 16) | (k.v[j + 1] << 16);
        k.v[7] >>= 16;
        if (d != 0 && i >= first) {
            const uint4* q = comb + 4 * ((size_t)i * kCombTab + (size_t)((d < 0 ? -d : d) - 1));
            const uint4 x0 = __ldg(q), x1 = __ldg(q + 1), y0 = __ldg(q + 2), y1 = __ldg(q + 3);
            const uint32_t xw[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
            const uint32_t yw[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
            Fd x, y;
            fd_unpack(x, xw);
            fd_unpack(y, yw);
            const double sg = (d < 0) != flip ? -1.0 : 1.0;
            UF_UNROLL
            for (int j = 0; j < 5; ++j) y.v[j] *= sg;
            B = kCalls ? jacd_add_aff_t<true>(B, x, y) : jacd_add_aff(B, x, y);
        }
    }
    return B;
}

#endif  // __CUDACC__

// The key on its scaled curve: (x c, c^2), c = x^3 + 7, from canonical limbs.
UF_HD void iso_key(Fd& kx, Fd& ky, Fd& c, const uint32_t x[8]) {
    Fd fx;
    fd_unpack(fx, x);
    fd_strict(fx);
    c = fdc_mul(fdc_sqr(fx), fx);
    c.v[0] += 7.0;
    fd_strict(c);
    kx = fdc_mul(fx, c);
    ky = fdc_sqr(c);
}

// The check around its inversion.  The values that cross the inversion wait in
// `tab`, the thread's point table, which is free by then: in registers they made
// ptxas spill, and with the spills it schedules the whole kernel for register
// pressure instead of latency (BIP-340: 49.4 against 55 M sigs/s).
//   slots 0: m, g1   1: p1, g2   2: p2, p3   3: p4, c
// y = m / g1 and y_R = ((p1 - y p2) p3 - p4) / g2, p3 kept negated.
//
// A key whose table is known in affine coordinates on secp256k1 itself (the
// resident key table) goes through the same check with c = 1: its scale is one,
// so the equation holds exactly when y comes out as 1.
//
// iso_prepare's den = g1, for BIP-340 g1 g2; slot 1 of an ECDSA item whose r may
// stand for r + n holds what m loses for it.  Its result:
enum : int {
    kIsoNo = 0,        // the item is invalid
    kIsoSolve = 1,     // iso_finish with 1 / den decides
    kIsoOnCurve = 2,   // valid if the key is on the curve (iso_on_curve)
    kIsoKeyInf = 3,    // BIP-340, b P infinite: b = 0, or the key is not on the curve
    kIsoPlain = 4      // left to the plain verification (no item is known to get here)
};

// r + n as digits (r < p - n).
UF_HD void iso_r_plus_n(Fd& f, const uint32_t r[8]) {
    uint32_t w[8];
    sc_n(w);
    uint64_t t = 0;
    UF_UNROLL
    for (int i = 0; i < 8; ++i) {
        t = (uint64_t)r[i] + w[i] + (t >> 32);
        w[i] = lo32(t);
    }
    fd_unpack(f, w);
    fd_strict(f);
}

// x(P) = r or, where alt, r + n, for a finite P (x = X / zz).
UF_COLD bool iso_x_is(Fd X, Fd zz, Fd r, Fd rn, bool alt) {
    if (fd_is_zero(fdc_mul_sub(r, zz, X))) return true;
    return alt && fd_is_zero(fdc_mul_sub(rn, zz, X));
}

struct IsoDen {
    Fd den;
    int st;
};

// x_A = x_B.  y = u / v by the same slots and one more inverse, 1 / Z(2 B)^3, for
// y(2 B): in iso_finish's terms m = u, g1 = v, g2 = Z^3, p1 = p2 = 0, p4 = -Y.
// About 20 products more in a warp that holds such an item.
template <bool kSchnorr, class Tab>
UF_COLD IsoDen iso_meet(Tab tab, JacD A, JacD B, Fd c, Fd r, Fd rn, bool alt) {
    IsoDen o;
    o.st = kIsoNo;
    const JacD D = jacd_dbl_n(B, 1);
    const Fd z2 = fdc_sqr(D.Z);
    if (!iso_x_is(D.X, z2, r, rn, alt)) return o;
    const Fd za3 = fdc_mul(fdc_sqr(A.Z), A.Z), zb3 = fdc_mul(fdc_sqr(B.Z), B.Z);
    const Fd u = fdc_mul(fdc_mul(B.Y, c), fdc_mul(c, za3)), v = fdc_mul(A.Y, zb3);
    Fd zero;
    fd_set_u32(zero, 0);
    o.st = kIsoSolve;
    o.den = v;
    tab.store(0, u, v);
    if (kSchnorr) {
        const Fd z3 = fdc_mul(z2, D.Z);
        tab.store(1, zero, z3);
        tab.store(2, zero, zero);
        tab.store(3, fd_neg(D.Y), c);
        o.den = fdc_mul(v, z3);
    } else {
        tab.store(1, zero, zero);
        tab.store(3, c, c);
    }
    return o;
}

template <bool kSchnorr, class Tab>
UF_HD int iso_prepare(const Tab& tab, Fd& den, const JacD& A, const JacD& B, const Fd& c, const uint32_t r[8]) {
    if (A.inf) return kSchnorr ? kIsoKeyInf : kIsoNo;
    Fd fr, frn;
    fd_unpack(fr, r);
    fd_strict(fr);
    const bool alt = !kSchnorr && r_below_p_minus_n(r);
    if (alt) iso_r_plus_n(frn, r);
    else frn = fr;
    const Fd za2 = fdc_sqr(A.Z);
    const Fd cz = fdc_mul(c, za2);
    if (B.inf) {
        if (kSchnorr) return kIsoPlain;
        tab.store(3, c, c);
        return iso_x_is(A.X, cz, fr, frn, alt) ? kIsoOnCurve : kIsoNo;
    }
    const Fd zb2 = fdc_sqr(B.Z);
    const Fd p2 = fdc_mul(A.X, zb2);
    const Fd N = fdc_mul_sub(B.X, cz, p2);
    if (fd_is_zero(N)) {
        const IsoDen o = iso_meet<kSchnorr>(tab, A, B, c, fr, frn, alt);
        den = o.den;
        return o.st;
    }
    const Fd za3 = fdc_mul(za2, A.Z), zb3 = fdc_mul(zb2, B.Z);
    const Fd c1 = fdc_mul(c, za3);
    const Fd g1 = fdc_mul(fdc_mul(fd_add_l(B.Y, B.Y), A.Y), fdc_mul(c1, zb3));
    den = g1;
    if (kSchnorr) {
        const Fd cza = fdc_mul(c, A.Z);
        const Fd g2 = fdc_mul(fdc_mul(cza, zb3), N);
        tab.store(1, fdc_mul(B.Y, fdc_mul(c, c1)), g2);
        tab.store(2, fdc_mul(A.Y, zb3), fdc_mul_sub(fr, zb2, B.X));
        tab.store(3, fdc_mul(fdc_mul(B.Y, cza), N), c);
        den = fdc_mul(g1, g2);
    } else {
        tab.store(3, c, c);
    }
    // r cz zb^2 + a zb^2 + d cz, the last two as N + 2 a zb^2
    const Fd czb = fdc_mul(cz, zb2), N2 = fdc_sqr(N);
    const Fd K = fdc_add(fdc_add(fdc_mul(fr, czb), N), fd_add_l(p2, p2));
    Fd m = fdc_mul(fdc_sqr(B.Y), fdc_mul(fdc_sqr(cz), cz));
    m = fdc_add(m, fdc_mul(fdc_sqr(A.Y), fdc_mul(fdc_sqr(zb2), zb2)));
    m = fdc_sub(m, fdc_mul(K, N2));
    tab.store(0, m, g1);
    if (alt) tab.store(1, fdc_mul(fdc_mul(czb, N2), fd_sub_l(frn, fr)), c);
    return kIsoSolve;
}

template <class Tab>
UF_HD bool iso_on_curve(const Tab& tab) {
    Fd c, x;
    tab.load(3, c, x);
    return fd_is_square(c);
}

// Second half, with inv = 1 / den (canonical limbs).  unit: the key was given on
// secp256k1 (c = 1); alt: r < p - n (ECDSA).
template <bool kSchnorr, class Tab>
UF_HD bool iso_finish(const Tab& tab, const Fe& inv, bool odd, bool unit, bool alt) {
    Fd fi, m, g1, p1, g2, p4, c;
    fd_unpack(fi, inv.v);
    fd_strict(fi);
    tab.load(0, m, g1);
    tab.load(1, p1, g2);
    tab.load(3, p4, c);
    uint32_t w[8];
    Fd y = fdc_mul(m, kSchnorr ? fdc_mul(fi, g2) : fi);
    bool good = fd_is_zero(fdc_mul_sub(y, y, c));
    if (kSchnorr && !good) return false;
    fd_pack(w, y);
    good = good && ((w[0] & 1u) != 0) == (odd || unit);          // of +-1, 1 is the odd one
    if (!kSchnorr && !good && alt) {
        y = fdc_mul(fdc_sub(m, p1), fi);
        good = fd_is_zero(fdc_mul_sub(y, y, c));
        fd_pack(w, y);
        good = good && ((w[0] & 1u) != 0) == (odd || unit);
    }
    if (!good) return false;
    if (kSchnorr) {
        Fd p2, p3;
        tab.load(2, p2, p3);
        const Fd s = fdc_sub(fdc_mul(y, p2), p1);            // times p3: both negated
        const Fd num = fdc_mul_sub(s, p3, p4);
        fd_pack(w, fdc_mul(num, fdc_mul(fi, g1)));
        if (w[0] & 1u) return false;
    }
    return true;
}

}  // namespace uf
