// Host build of the FP64 point additions (csrc/jacd.cuh) for
// tests/test_fp_digits.py; values are 8 little-endian 32-bit limbs.
#include "../../ultrafastsecp256k1_b200/csrc/jacd.cuh"

using namespace uf;

namespace {
Fd in(const uint32_t* w) {
    Fd r;
    fd_unpack(r, w);
    fd_strict(r);
    return r;
}
JacD point(const uint32_t* w) {
    JacD p;
    p.X = in(w);
    p.Y = in(w + 8);
    p.Z = in(w + 16);
    p.inf = false;
    return p;
}
}  // namespace

// a + b (X, Y, Z each) as digits and as packed limbs
extern "C" void jd_add(const uint32_t* a, const uint32_t* b, double* digits, uint32_t* packed) {
    const JacD s = jacd_add(point(a), point(b));
    const Fd v[3] = {s.X, s.Y, s.Z};
    for (int c = 0; c < 3; ++c) {
        for (int i = 0; i < 5; ++i) digits[5 * c + i] = v[c].v[i];
        fd_pack(packed + 8 * c, v[c]);
    }
}

extern "C" void jd_add_sub(const double* a, const double* b, double* sum, double* diff) {
    Fd x, y;
    for (int i = 0; i < 5; ++i) {
        x.v[i] = a[i];
        y.v[i] = b[i];
    }
    const Fd s = fdc_add(x, y), d = fdc_sub(x, y);
    for (int i = 0; i < 5; ++i) {
        sum[i] = s.v[i];
        diff[i] = d.v[i];
    }
}

extern "C" int jd_is_square(const uint32_t* a) { return fd_is_square(in(a)) ? 1 : 0; }
