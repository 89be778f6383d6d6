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

// n doublings in one call.  Point operations are out of line with the field
// operations inlined into them: all inlined, four doublings and two additions
// take 18.3 k cycles per warp and scheduler at two blocks per SM, with the field
// operations out of line 21.2 k.
UF_COLD JacD jacd_dbl_n(JacD a, int n) {
    UF_NOUNROLL
    for (int i = 0; i < n; ++i) a = jacd_dbl_c(a);
    return a;
}

// a += (x2, y2), digits unsigned or strict, y2 also negated: U2 = x2 Z1^2,
// S2 = y2 Z1^3, H = U2 - X1, r = S2 - Y1, V = X1 H^2, X3 = r^2 - H^3 - 2 V,
// Y3 = r (V - X3) - Y1 H^3, Z3 = Z1 H: 8M + 3S, the products of Y3 reduced
// together and the differences taken inside their product's reduction.  Exact
// for every input: equal points double, opposite ones give the identity.
UF_HD JacD jacd_add_aff_c(JacD a, Fd x2, Fd y2) {
    if (a.inf) {
        fd_strict(x2);
        fd_strict(y2);
        a.X = x2;
        a.Y = y2;
        fd_set_u32(a.Z, 1);
        a.inf = false;
        return a;
    }
    const Fd ZZ = fd_sqr(a.Z);
    const Fd H = fd_mul_sub(x2, ZZ, a.X);
    const Fd ZZZ = fd_mul(a.Z, ZZ);
    const Fd r = fd_mul_sub(y2, ZZZ, a.Y);
    if (fd_is_zero(H)) {
        if (fd_is_zero(r)) a = jacd_dbl_n(a, 1);
        else a.inf = true;
        return a;
    }
    a.Z = fd_mul(a.Z, H);
    const Fd HH = fd_sqr(H);
    const Fd HHH = fd_mul(H, HH);
    const Fd V = fd_mul(a.X, HH);
    a.X = fd_sqr_sub_sub2(r, HHH, V);
    a.Y = fd_mul_mul_sub(fd_sub_l(V, a.X), r, a.Y, HHH);
    return a;
}

UF_COLD JacD jacd_add_aff(JacD a, Fd x2, Fd y2) { return jacd_add_aff_c(a, x2, y2); }

}  // namespace uf
