// Points of y^2 = x^3 + b in Jacobian coordinates over fd.cuh (a = 0, any b:
// the formulas do not use it, so they serve secp256k1 and the curves isomorphic
// to it that the verify kernels compute on).
#pragma once
#include "common.cuh"
#include "fd.cuh"

namespace uf {

// Strict digits; the identity is flagged.
struct JacD { Fd X, Y, Z; bool inf; };

UF_HD void jacd_set_inf(JacD& a) {
    fd_set_u32(a.X, 0);
    fd_set_u32(a.Y, 1);
    fd_set_u32(a.Z, 0);
    a.inf = true;
}

// E = 3 X^2, B = 2 Y^2, S = 2 X B, X3 = E^2 - 2 S, Y3 = E (S - X3) - 2 B^2,
// Z3 = 2 Y Z: 3M + 4S with the two products of Y3 reduced together.  The
// identity stays flagged (its coordinates only stay bounded).  Y = 0 has no point
// of odd order; on another curve it gives Z = 0, which the callers reject.
UF_HD JacD jacd_dbl_c(JacD a) {
    if (a.inf) return a;
    const Fd E = fd_sqr_x<3>(a.X);
    const Fd B = fd_sqr_x<2>(a.Y);
    a.Z = fd_mul(fd_add_l(a.Y, a.Y), a.Z);
    const Fd S = fd_mul(fd_add_l(B, B), a.X);
    a.X = fd_sqr_sub2(E, S);
    a.Y = fd_mul_sub_2sqr(fd_sub_l(S, a.X), E, B);
    return a;
}

// The same for a warp alone on its scheduler (kCalls as below): the two plain
// products through the out-of-line form that the additions call too, so that a
// digit's doublings and addition fit the instruction cache better.  4,096
// signatures by four warps per 32: ECDSA 288 -> 280 us, BIP-340 289 -> 271; with
// the squarings out of line as well 297 and 301.
template <bool kCalls>
UF_HD JacD jacd_dbl_t(JacD a) {
    if (!kCalls) return jacd_dbl_c(a);
    if (a.inf) return a;
    const Fd E = fd_sqr_x<3>(a.X);
    const Fd B = fd_sqr_x<2>(a.Y);
    a.Z = fdc_mul(fd_add_l(a.Y, a.Y), a.Z);
    const Fd S = fdc_mul(fd_add_l(B, B), a.X);
    a.X = fd_sqr_sub2(E, S);
    a.Y = fd_mul_sub_2sqr(fd_sub_l(S, a.X), E, B);
    return a;
}

// n doublings in one call.  Point operations are out of line with the field
// operations inlined into them: all inlined, four doublings and two additions
// take 18.3 k cycles per warp and scheduler at two blocks per SM, with the field
// operations out of line 21.2 k.
UF_COLD JacD jacd_dbl_n(JacD a, int n) {
    UF_NOUNROLL
    for (int i = 0; i < n; ++i) a = jacd_dbl_c(a);
    return a;
}

// A field operation inlined or, with kCalls, through its out-of-line form.
template <bool kCalls>
UF_HD Fd jf_mul(const Fd& a, const Fd& b) { return kCalls ? fdc_mul(a, b) : fd_mul(a, b); }
template <bool kCalls>
UF_HD Fd jf_sqr(const Fd& a) { return kCalls ? fdc_sqr(a) : fd_sqr(a); }
template <bool kCalls>
UF_HD Fd jf_mul_sub(const Fd& a, const Fd& b, const Fd& x) {
    return kCalls ? fdc_mul_sub(a, b, x) : fd_mul_sub(a, b, x);
}

// a += (x2, y2), digits unsigned or strict, y2 also negated: U2 = x2 Z1^2,
// S2 = y2 Z1^3, H = U2 - X1, r = S2 - Y1, V = X1 H^2, X3 = r^2 - H^3 - 2 V,
// Y3 = r (V - X3) - Y1 H^3, Z3 = Z1 H: 8M + 3S, the products of Y3 reduced
// together and the differences taken inside their product's reduction.  Exact
// for every input: equal points double, opposite ones give the identity.
// kCalls: the products out of line (25 KB of code instead of 37): a warp alone
// on its scheduler takes 5.1 k cycles that way and 6.3 k inlined, two warps in
// step 8.5 k and 8.3 k.
template <bool kCalls>
UF_HD JacD jacd_add_aff_t(JacD a, Fd x2, Fd y2) {
    if (a.inf) {
        fd_strict(x2);
        fd_strict(y2);
        a.X = x2;
        a.Y = y2;
        fd_set_u32(a.Z, 1);
        a.inf = false;
        return a;
    }
    const Fd ZZ = jf_sqr<kCalls>(a.Z);
    const Fd H = jf_mul_sub<kCalls>(x2, ZZ, a.X);
    const Fd ZZZ = jf_mul<kCalls>(a.Z, ZZ);
    const Fd r = jf_mul_sub<kCalls>(y2, ZZZ, a.Y);
    if (fd_is_zero(H)) {
        if (fd_is_zero(r)) a = jacd_dbl_n(a, 1);
        else a.inf = true;
        return a;
    }
    a.Z = jf_mul<kCalls>(a.Z, H);
    const Fd HH = jf_sqr<kCalls>(H);
    const Fd HHH = jf_mul<kCalls>(H, HH);
    const Fd V = jf_mul<kCalls>(a.X, HH);
    a.X = fd_sqr_sub_sub2(r, HHH, V);
    a.Y = fd_mul_mul_sub(fd_sub_l(V, a.X), r, a.Y, HHH);
    return a;
}

UF_COLD JacD jacd_add_aff(JacD a, Fd x2, Fd y2) { return jacd_add_aff_t<false>(a, x2, y2); }

// (X, Y, ZZ = Z^2, ZZZ = Z^3): for long runs of mixed additions, one squaring
// less each than in Jacobian form.
struct XyzzD { Fd X, Y, ZZ, ZZZ; bool inf; };

UF_HD void xyzzd_set_inf(XyzzD& a) {
    fd_set_u32(a.X, 0);
    fd_set_u32(a.Y, 1);
    fd_set_u32(a.ZZ, 0);
    fd_set_u32(a.ZZZ, 0);
    a.inf = true;
}

// 2 (x, y) of an affine point, strict digits.
UF_COLD XyzzD xyzzd_dbl_aff(Fd x, Fd y) {
    XyzzD r;
    const Fd M = fd_sqr_x<3>(x), H = fd_sqr_x<2>(y);       // 3 x^2, 2 y^2
    r.ZZ = fd_add_l(H, H);                                 // (2 y)^2
    fd_strict(r.ZZ);
    r.ZZZ = fdc_mul(fd_add_l(y, y), r.ZZ);
    const Fd S = fdc_mul(x, r.ZZ);
    r.X = fd_sqr_sub2(M, S);
    r.Y = fdc_mul_sub(fd_sub_l(S, r.X), M, fdc_mul(y, r.ZZZ));
    r.inf = false;
    return r;
}

// a += (x2, y2), digits as in jacd_add_aff_t, exact for every input: 8M + 2S, the
// products of Y3 reduced together.
UF_HD void xyzzd_add_aff(XyzzD& a, Fd x2, Fd y2) {
    if (a.inf) {
        fd_strict(x2);
        fd_strict(y2);
        a.X = x2;
        a.Y = y2;
        fd_set_u32(a.ZZ, 1);
        fd_set_u32(a.ZZZ, 1);
        a.inf = false;
        return;
    }
    const Fd H = fd_mul_sub(x2, a.ZZ, a.X);
    const Fd r = fd_mul_sub(y2, a.ZZZ, a.Y);
    if (fd_is_zero(H)) {
        if (fd_is_zero(r)) {
            fd_strict(x2);
            fd_strict(y2);
            a = xyzzd_dbl_aff(x2, y2);
        } else {
            a.inf = true;
        }
        return;
    }
    const Fd HH = fd_sqr(H);
    const Fd HHH = fd_mul(H, HH);
    const Fd V = fd_mul(a.X, HH);
    a.ZZ = fd_mul(a.ZZ, HH);
    a.ZZZ = fd_mul(a.ZZZ, HHH);
    a.X = fd_sqr_sub_sub2(r, HHH, V);
    a.Y = fd_mul_mul_sub(fd_sub_l(V, a.X), r, a.Y, HHH);
}

// The same point in Jacobian form: Z' = Z ZZ = ZZZ, so X' = X ZZ^2, Y' = Y ZZ^3.
UF_HD JacD xyzzd_to_jac(const XyzzD& a) {
    JacD p;
    const Fd w = fdc_sqr(a.ZZ);
    p.X = fdc_mul(a.X, w);
    p.Y = fdc_mul(a.Y, fdc_mul(w, a.ZZ));
    p.Z = a.ZZZ;
    p.inf = a.inf;
    return p;
}

// General addition, exact for every input (a few per signature).
UF_COLD JacD jacd_add(JacD a, JacD b) {
    if (b.inf) return a;
    if (a.inf) return b;
    const Fd za2 = fdc_sqr(a.Z), zb2 = fdc_sqr(b.Z);
    const Fd U = fdc_mul(a.X, zb2);
    const Fd H = fdc_mul_sub(b.X, za2, U);
    const Fd S = fdc_mul(a.Y, fdc_mul(b.Z, zb2));
    const Fd r = fdc_mul_sub(b.Y, fdc_mul(a.Z, za2), S);
    if (fd_is_zero(H)) {
        if (fd_is_zero(r)) a = jacd_dbl_n(a, 1);
        else a.inf = true;
        return a;
    }
    const Fd HH = fdc_sqr(H);
    const Fd HHH = fdc_mul(H, HH), V = fdc_mul(U, HH);
    a.Z = fdc_mul(fdc_mul(a.Z, b.Z), H);
    a.X = fdc_sqr_sub_sub2(r, HHH, V);         // one reduction: a difference of two may leave (-p, p)
    a.Y = fdc_mul_sub(fd_sub_l(V, a.X), r, fdc_mul(S, HHH));
    return a;
}

}  // namespace uf
