// Host build of the FP64 field, point and digit headers (csrc/fd.cuh, jacd.cuh,
// eis.cuh) for tests/test_fp_verify.py.  Operands are digit vectors or 8
// little-endian 32-bit limbs.
#include "../../ultrafastsecp256k1_b200/csrc/eis.cuh"

using namespace uf;

namespace {
Fd in(const double* d) {
    Fd r;
    for (int i = 0; i < 5; ++i) r.v[i] = d[i];
    return r;
}
struct Table {
    Fd* p;
    void store(int k, const Fd& x, const Fd& y) const { p[2 * k] = x; p[2 * k + 1] = y; }
    void load(int k, Fd& x, Fd& y) const { x = p[2 * k]; y = p[2 * k + 1]; }
};
}  // namespace

extern "C" void fp_op(int op, const double* a, const double* b, const double* x, const double* y, double* out) {
    const Fd A = in(a), B = in(b), X = in(x), Y = in(y);
    Fd r = A;
    switch (op) {
        case 0: r = fd_mul(A, B); break;
        case 1: r = fd_sqr(A); break;
        case 2: r = fd_mul_sub(A, B, X); break;
        case 3: r = fd_sqr_x<2>(A); break;
        case 4: r = fd_sqr_x<3>(A); break;
        case 5: r = fd_sqr_sub2(A, X); break;
        case 6: r = fd_sqr_sub_sub(A, X, Y); break;
        case 7: r = fd_sqr_sub_sub2(A, X, Y); break;
        case 8: r = fd_mul_mul_sub(A, B, X, Y); break;
        case 9: r = fd_mul_sub_2sqr(A, B, X); break;
        case 10: fd_strict(r); break;
    }
    for (int i = 0; i < 5; ++i) out[i] = r.v[i];
}

extern "C" void fp_unpack(const uint32_t* w, double* out) {
    Fd r;
    fd_unpack(r, w);
    for (int i = 0; i < 5; ++i) out[i] = r.v[i];
}

extern "C" void fp_pack(const double* d, uint32_t* w) { fd_pack(w, in(d)); }

// k (x, y) in Jacobian coordinates X, Y, Z (canonical limbs); 0 for infinity
extern "C" int fp_point_mul(const uint32_t* k, const uint32_t* x, const uint32_t* y, uint32_t* out) {
    Sc s;
    for (int i = 0; i < 8; ++i) s.v[i] = k[i];
    GlvSplit g;
    glv_split(g, s);
    uint8_t dig[kEisDigits];
    eis_recode(dig, g);
    Fd px, py, cells[2 * kEisTab];
    fd_unpack(px, x);
    fd_unpack(py, y);
    fd_strict(px);
    fd_strict(py);
    const Table t{cells};
    const Fd zc = eis_table(t, px, py);
    JacD R = eis_mul(dig, t);
    if (R.inf) return 0;
    R.Z = fd_mul(R.Z, zc);
    fd_pack(out, R.X);
    fd_pack(out + 8, R.Y);
    fd_pack(out + 16, R.Z);
    return 1;
}
