// Host build of the signature check without a square root (csrc/isocheck.cuh)
// for tests/test_edge_items.py.  Values are 8 little-endian 32-bit limbs.
#include "../../ultrafastsecp256k1_b200/csrc/isocheck.cuh"

using namespace uf;

namespace {
struct Table {
    Fd* p;
    void store(int k, const Fd& x, const Fd& y) const { p[2 * k] = x; p[2 * k + 1] = y; }
    void load(int k, Fd& x, Fd& y) const { x = p[2 * k]; y = p[2 * k + 1]; }
};

Fd in(const uint32_t* w) {
    Fd r;
    fd_unpack(r, w);
    fd_strict(r);
    return r;
}

template <bool kSchnorr>
int check(const Table& t, const JacD& A, const JacD& B, const Fd& c, const uint32_t* r, bool odd, bool unit) {
    Fd den;
    int st = iso_prepare<kSchnorr>(t, den, A, B, c, r);
    bool holds = false;
    if (st == kIsoSolve) {
        Fe inv;
        fd_pack(inv.v, den);
        if (is_zero256(inv.v)) return kIsoPlain;
        fe_inv(inv, inv);
        holds = iso_finish<kSchnorr>(t, inv, odd, unit, !kSchnorr && r_below_p_minus_n(r));
    }
    if (st == kIsoOnCurve) holds = iso_on_curve(t);
    return st | (holds ? 256 : 0);
}
}  // namespace

// x(A + B) = r, with A = b P for the key P of that x and parity (py: its y, given
// with `unit` only) and B = (X / Z^2, Y / Z^3), infinite where Z = 0; BIP-340 also
// wants an even y.  iso_prepare's result, | 256 where the item is valid.
extern "C" int iso_check(int schnorr, int unit, const uint32_t* px, const uint32_t* py, int odd, const uint32_t* b,
                         const uint32_t* bj, const uint32_t* r) {
    Sc s;
    for (int i = 0; i < 8; ++i) s.v[i] = b[i];
    GlvSplit g;
    glv_split(g, s);
    uint8_t dig[kEisDigits];
    eis_recode(dig, g);
    Fd cells[2 * kEisTab], kx, ky, c;
    const Table t{cells};
    if (unit) {
        kx = in(px);
        ky = in(py);
        fd_set_u32(c, 1);
    } else {
        iso_key(kx, ky, c, px);
    }
    const Fd zc = eis_table(t, kx, ky);
    if (fd_is_zero(zc)) return kIsoNo;
    JacD A = eis_mul(dig, t), B;
    A.Z = fd_mul(A.Z, zc);
    B.X = in(bj);
    B.Y = in(bj + 8);
    B.Z = in(bj + 16);
    B.inf = is_zero256(bj + 16);
    return schnorr ? check<true>(t, A, B, c, r, odd != 0, unit != 0) : check<false>(t, A, B, c, r, odd != 0, unit != 0);
}
