// Field arithmetic mod p = 2^256 - 2^32 - 977 on the FP64 pipe: five signed
// 52-bit digits held as doubles, every operation exact.
//
// Why.  B200 issues 64 FP64 fused multiply-adds per SM and clock, as many lanes
// as its 32-bit integer multiply-adds, and a 52 x 52-bit product needs two of
// them where the integer pipe needs about four half-rate wide multiply-adds.
// A field multiplication on 8 x 32-bit limbs (fe.cuh) is bound by the integer
// multiply-add pipe; here the products run on the FP64 pipe and the column sums
// on the integer ALU pipe, which the carry chains leave idle, and the 25
// products of a multiplication are independent where the limb form is a chain
// of carries.
//
// Product of two digits (Emmart, Zheng, Weems, "Faster Modular Exponentiation
// Using Double Precision Floating Point Arithmetic on the GPU", 2018: the
// high / low split of a product by two fused multiply-adds).  With
// C1 = 1.5 * 2^104, whose last place is 2^52, and |a b| <= 2^103:
//   h = fma_rd(a, b, C1)            = C1 + 2^52 q,  q = floor(a b / 2^52)
//   l = fma(a, b, (C1 + 2^52) - h)  = 2^52 + (a b mod 2^52)
// exactly, so the bit patterns of h and l, read as 64-bit integers, are a
// constant plus q and a constant plus the low half: they are summed per column
// as integers and the constants leave with the column's initial value.
//
// Digits.  "Strict" digits d_0..d_3 lie in [-2^51, 2^51]; every function below
// returns strict digits unless it says otherwise, and a multiplication's result
// has |d_4| <= 2^47 + 2^12 and its value in (-p, p), which fd_pack and fd_is_zero
// need.  A product may take strict digits times sums or differences of two strict
// values (2^52 * 2^51 = 2^103), or times the unsigned digits [0, 2^52) of an
// unpacked table coordinate.
//
// The top digit of other values is larger: 2^48 for a coordinate just below p,
// 2^49 for sums of a few results.  Products take |d_4| up to 2^50: the column of
// weight 2^468 holds the top products' high halves alone, so those of one
// reduction have to stay below 2^103 together (a b - 2 x^2: 3 * 2^100).
#pragma once
#include "common.cuh"
#include "fe.cuh"
#if !defined(__CUDACC__)
#include <cfenv>
#include <cmath>
#include <string.h>
#endif

namespace uf {

struct Fd { double v[5]; };

#if defined(__CUDACC__)
#define UF_HDC __host__ __device__ static constexpr
#else
#define UF_HDC static constexpr
#endif

UF_HD double fd_fma_rd(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
    return __fma_rd(a, b, c);
#elif defined(__CUDACC__)
    return a * b + c;   // host pass of nvcc: never run
#else
    const int mode = fegetround();
    fesetround(FE_DOWNWARD);
    volatile double x = a, y = b, z = c;
    volatile double r = std::fma(x, y, z);
    fesetround(mode);
    return r;
#endif
}

UF_HD double fd_fma(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
    return __fma_rn(a, b, c);
#elif defined(__CUDACC__)
    return a * b + c;
#else
    return std::fma(a, b, c);
#endif
}

UF_HD uint64_t fd_bits(double d) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(d);
#else
    uint64_t u;
    memcpy(&u, &d, 8);
    return u;
#endif
}

UF_HD double fd_from_bits(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double d;
    memcpy(&d, &u, 8);
    return d;
#endif
}

UF_HD double fd_mk(uint32_t hi, uint32_t lo) { return fd_from_bits(((uint64_t)hi << 32) | lo); }

#define UF_FD_C1 30423614405477505635920876929024.0       /* 1.5 * 2^104 */
#define UF_FD_C2 30423614405477510139520504299520.0       /* 1.5 * 2^104 + 2^52 */
#define UF_FD_2P104 20282409603651670423947251286016.0
#define UF_FD_2P52 4503599627370496.0
#define UF_FD_2P51 2251799813685248.0
#define UF_FD_EXP 0x43300000u                              /* high word of 2^52 */
// what a low and a high half's bit pattern add to a column beside their value
constexpr uint64_t kFdBiasLo = 0x4330000000000000ull;
constexpr uint64_t kFdBiasHi = 0x4670000000000000ull + (1ull << 51);
// and a digit x converted as 1.5 * 2^52 - x, beside -x
constexpr uint64_t kFdBiasIn = 0x4330000000000000ull + (1ull << 51);
constexpr double kFdR = 68719492368.0;                     // 2^260 mod p = 2^36 + 15632
constexpr double kFdK = 4294968273.0;                      // 2^256 mod p = 2^32 + 977

// Low and high halves per column of a full product and of a square: column k
// holds the low halves of the digit products of weight k and the high halves of
// weight k - 1.
UF_HDC int fd_nmul(int k) { return k < 0 || k > 8 ? 0 : (k < 5 ? k + 1 : 9 - k); }
UF_HDC int fd_nsq(int k) { return k < 0 || k > 8 ? 0 : (k < 4 ? k / 2 + 1 : (10 - k) / 2); }

// What a sum of columns holds beside its value, as compile-time constants:
// M full products, Q squares (2 for a doubled square), I injected digits, the
// low columns taken S times, and the terms of fd_reduce.
template <int M, int Q, int I, int S>
struct FdBias {
    UF_HDC uint64_t col0(int k) {
        return (uint64_t)(M * fd_nmul(k) + Q * fd_nsq(k)) * kFdBiasLo +
               (uint64_t)(M * fd_nmul(k - 1) + Q * fd_nsq(k - 1)) * kFdBiasHi + (uint64_t)(k < 5 ? I : 0) * kFdBiasIn;
    }
    // columns 6..8: one more from the high half of digit product (k - 5, 4), whose
    // small top digit leaves the room, where fd_reduce's constant would be odd
    UF_HDC uint64_t dl(int k) { return k >= 6 && k <= 8 ? (col0(k - 1) >> 52) & 1 : 0; }
    UF_HDC uint64_t col(int k) { return col0(k) + dl(k); }
    // high columns: carry constant and fraction
    UF_HDC uint32_t top(int k) { return (uint32_t)(col(k) >> 52); }
    UF_HDC uint64_t frac(int k) { return col(k) & ((1ull << 52) - 1); }
    // low columns, without the fold's free constant, in fd_reduce's order
    UF_HDC uint64_t low0(int k) {
        return (uint64_t)S * col(k) + kFdBiasLo + (k == 0 ? kFdBiasLo : 0x4670000000000000ull) +
               (k == 1 ? kFdBiasHi : 0ull);
    }
    // whether column k takes + 2^51 by an integer add (k = 0, and where the
    // fraction is already odd)
    UF_HDC bool odd(int k) { return ((low0(k) >> 51) & 1) != 0; }
    UF_HDC bool add51(int k) { return k == 0 ? !odd(0) : (k < 4 && odd(k)); }
    // free constant of the fold's high half entering column k = 1..4
    UF_HDC uint64_t x(int k) {
        return (k < 4 ? 1ull << 51 : (1ull << 51) + (1ull << 47)) - cin(k);
    }
    // constant arriving with column k - 1's carry
    UF_HDC uint64_t cin(int k) { return k == 0 ? 0 : (uint64_t)dtop(k - 1); }
    UF_HDC uint64_t total(int k) {
        return low0(k) + (k > 0 ? x(k) : 0ull) + (add51(k) ? 1ull << 51 : 0ull) + (k < 4 ? cin(k) : 0ull);
    }
    UF_HDC uint32_t dtop(int k) { return (uint32_t)(total(k) >> 52); }
    // column 4 from bit 48 on
    UF_HDC uint32_t dtop48() { return (uint32_t)((low0(4) + x(4)) >> 48); }
};

// C1 of digit product (i, j): with B's extra one where column i + 5 asks for it
template <class B>
UF_HDC double fd_c1(int i, int j, bool acc) {
    return !acc && j == 4 && i < 4 && B::dl(i + 5) ? UF_FD_C2 : UF_FD_C1;
}

struct FdNoBias {
    UF_HDC uint64_t dl(int) { return 0; }
};

// c = a b (kAcc = false) or c += a b
template <class B, bool kAcc>
UF_HD void fd_mac(uint64_t c[10], const Fd& a, const Fd& b) {
    UF_UNROLL
    for (int i = 0; i < 5; ++i) {
        double h[5], d[5];
        uint64_t l[5];
        UF_UNROLL
        for (int j = 0; j < 5; ++j) h[j] = fd_fma_rd(a.v[i], b.v[j], fd_c1<B>(i, j, kAcc));
        UF_UNROLL
        for (int j = 0; j < 5; ++j) d[j] = (fd_c1<B>(i, j, kAcc) + UF_FD_2P52) - h[j];
        UF_UNROLL
        for (int j = 0; j < 5; ++j) l[j] = fd_bits(fd_fma(a.v[i], b.v[j], d[j]));
        c[i] = (kAcc || i > 0) ? c[i] + l[0] : l[0];
        UF_UNROLL
        for (int j = 1; j < 5; ++j) {
            const uint64_t t = l[j] + fd_bits(h[j - 1]);
            c[i + j] = (kAcc || i > 0) ? c[i + j] + t : t;
        }
        c[i + 5] = kAcc ? c[i + 5] + fd_bits(h[4]) : fd_bits(h[4]);
    }
}

// c = a^2 (strict a), the cross products once with a doubled digit
template <class B>
UF_HD void fd_sac(uint64_t c[10], const Fd& a) {
    UF_UNROLL
    for (int i = 0; i < 5; ++i) {
        double h[5], d[5];
        uint64_t l[5];
        const double t2 = a.v[i] + a.v[i];
        UF_UNROLL
        for (int j = i; j < 5; ++j) h[j] = fd_fma_rd(j == i ? a.v[i] : t2, a.v[j], fd_c1<B>(i, j, false));
        UF_UNROLL
        for (int j = i; j < 5; ++j) d[j] = (fd_c1<B>(i, j, false) + UF_FD_2P52) - h[j];
        UF_UNROLL
        for (int j = i; j < 5; ++j) l[j] = fd_bits(fd_fma(j == i ? a.v[i] : t2, a.v[j], d[j]));
        c[2 * i] = i > 0 ? c[2 * i] + l[i] : l[i];
        UF_UNROLL
        for (int j = i + 1; j < 5; ++j) {
            const uint64_t t = l[j] + fd_bits(h[j - 1]);
            c[i + j] = i > 0 ? c[i + j] + t : t;
        }
        c[i + 5] = fd_bits(h[4]);
    }
}

// c -= x (strict x)
UF_HD void fd_inject_neg(uint64_t c[10], const Fd& x) {
    UF_UNROLL
    for (int k = 0; k < 5; ++k) c[k] += fd_bits(1.5 * UF_FD_2P52 - x.v[k]);
}

// c -= 2 x (counts as two injected values)
UF_HD void fd_inject_neg2(uint64_t c[10], const Fd& x) {
    UF_UNROLL
    for (int k = 0; k < 5; ++k) {
        const uint64_t b = fd_bits(1.5 * UF_FD_2P52 - x.v[k]);
        c[k] += b + b;
    }
}

// S times the column sums (S = 1, 2, 3), reduced mod p to strict digits.
// Columns 5..9 become digits h_j of value 2^260 each step up by one parallel
// carry, are folded with 2^260 = R (mod p) through the same high / low split,
// what lies above 2^256 is folded once more with K, and one carry pass over
// columns 0..4 gives the digits.  Every constant that the bit patterns bring
// along is known at compile time (B) and leaves in an operation that is there
// anyway; sums stay below 2^58 in magnitude.
template <class B, int S>
UF_HD Fd fd_reduce(const uint64_t c[10]) {
    static_assert(B::top(5) >= 100 && B::top(5) <= 3996 && B::top(6) >= 100 && B::top(6) <= 3996 &&
                  B::top(7) >= 100 && B::top(7) <= 3996 && B::top(8) >= 100 && B::top(8) <= 3996, "high carries");
    static_assert(B::dtop(0) >= 100 && B::dtop(0) <= 3996 && B::dtop(1) >= 100 && B::dtop(1) <= 3996 &&
                  B::dtop(2) >= 100 && B::dtop(2) <= 3996 && B::dtop(3) >= 100 && B::dtop(3) <= 3996, "low carries");
    static_assert(B::dtop48() >= 2000 && B::dtop48() <= 63000, "top carry");
    double h[5];
    h[0] = fd_mk((hi32(c[5]) & 0xFFFFFu) | UF_FD_EXP, lo32(c[5])) - (UF_FD_2P52 + (double)B::frac(5));
    UF_UNROLL
    for (int k = 6; k < 9; ++k) {
        const double K = 2.0 * UF_FD_2P52 + (double)(B::top(k - 1) + B::frac(k));
        h[k - 5] = fd_mk((hi32(c[k]) & 0xFFFFFu) | UF_FD_EXP, lo32(c[k])) +
                   (fd_mk(UF_FD_EXP, hi32(c[k - 1]) >> 20) - K);
    }
    // column 9 holds high halves only: as 2^52 + 2^51 + value
    h[4] = fd_from_bits(c[9] + (kFdBiasIn + (B::top(8) & 1) - B::col(9))) +
           (fd_mk(UF_FD_EXP, hi32(c[8]) >> 20) -
            (2.0 * UF_FD_2P52 + UF_FD_2P51 + (double)(B::top(8) + (B::top(8) & 1))));
    const double R = S * kFdR;
    uint64_t e[5], d[5];
    double top = 0;
    UF_UNROLL
    for (int j = 0; j < 5; ++j) {
        const double C = j < 4 ? UF_FD_2P104 + UF_FD_2P52 * (double)B::x(j < 4 ? j + 1 : 4) : UF_FD_C1;
        const double hh = fd_fma_rd(h[j], R, C);
        const uint64_t l = fd_bits(fd_fma(h[j], R, (C + UF_FD_2P52) - hh));
        d[j] = (S == 1 ? c[j] : S == 2 ? c[j] + c[j] : c[j] + c[j] + c[j]) + l;
        if (j > 0) d[j] += e[j - 1];
        if (j < 4) e[j] = fd_bits(hh);
        else top = hh - C;
    }
    const double q = fd_fma(top, 1.0 / 281474976710656.0,
                            fd_mk(UF_FD_EXP, hi32(d[4]) >> 16) - (UF_FD_2P52 + (double)B::dtop48()));
    const double qh = fd_fma_rd(q, kFdK, UF_FD_C1);
    d[0] += fd_bits(fd_fma(q, kFdK, UF_FD_C2 - qh));
    d[1] += fd_bits(qh);
    Fd r;
    uint32_t cy = 0;
    UF_UNROLL
    for (int k = 0; k < 4; ++k) {
        if (k > 0) d[k] += cy;
        if (B::add51(k)) d[k] += 1ull << 51;
        r.v[k] = fd_mk((hi32(d[k]) & 0xFFFFFu) | UF_FD_EXP, lo32(d[k])) - (UF_FD_2P52 + UF_FD_2P51);
        cy = hi32(d[k]) >> 20;
    }
    // x(4) took column 3's carry constant out already
    r.v[4] = fd_mk((hi32(d[4]) & 0xFFFFu) | UF_FD_EXP, lo32(d[4])) +
             (fd_mk(UF_FD_EXP, cy) - (2.0 * UF_FD_2P52 + 140737488355328.0));
    return r;
}

// ---- values ---------------------------------------------------------------------

UF_HD void fd_set_u32(Fd& r, uint32_t a) {
    r.v[0] = (double)a;
    UF_UNROLL
    for (int i = 1; i < 5; ++i) r.v[i] = 0.0;
}

// 8 little-endian 32-bit limbs -> unsigned digits in [0, 2^52) (not strict).
UF_HD void fd_unpack(Fd& r, const uint32_t w[8]) {
    const uint32_t m = 0xFFFFFu;
    r.v[0] = fd_mk((w[1] & m) | UF_FD_EXP, w[0]) - UF_FD_2P52;
    r.v[1] = fd_mk((((w[2] >> 20) | (w[3] << 12)) & m) | UF_FD_EXP, (w[1] >> 20) | (w[2] << 12)) - UF_FD_2P52;
    r.v[2] = fd_mk((((w[4] >> 8) | (w[5] << 24)) & m) | UF_FD_EXP, (w[3] >> 8) | (w[4] << 24)) - UF_FD_2P52;
    r.v[3] = fd_mk((((w[5] >> 28) | (w[6] << 4)) & m) | UF_FD_EXP, (w[4] >> 28) | (w[5] << 4)) - UF_FD_2P52;
    r.v[4] = fd_mk((w[7] >> 16) | UF_FD_EXP, (w[6] >> 16) | (w[7] << 16)) - UF_FD_2P52;
}

// Any digits below 2^53 in magnitude -> strict digits of the same value (what the
// lower digits carry goes to the top one).
UF_HD void fd_strict(Fd& a) {
    UF_UNROLL
    for (int k = 0; k < 4; ++k) {
        const double u = (a.v[k] + UF_FD_C1) - UF_FD_C1;     // nearest multiple of 2^52
        a.v[k] -= u;
        a.v[k + 1] = fd_fma(u, 1.0 / UF_FD_2P52, a.v[k + 1]);
    }
}

// Strict digits of a value in (-p, p) -> canonical limbs of its residue.
UF_HD void fd_pack(uint32_t w[8], const Fd& a) {
    int64_t t[5];
    UF_UNROLL
    for (int k = 0; k < 5; ++k) t[k] = (int64_t)(fd_bits(a.v[k] + 1.5 * UF_FD_2P52) - kFdBiasIn);
    int64_t c = 0, u[5];
    UF_UNROLL
    for (int k = 0; k < 5; ++k) c = (t[k] + c) >> 52;
    // c < 0 exactly when the value is negative: + p
    const int64_t neg = c < 0 ? -1 : 0;
    t[0] -= neg & (int64_t)4294968273ll;
    t[4] += neg & (int64_t)(1ll << 48);
    c = 0;
    UF_UNROLL
    for (int k = 0; k < 5; ++k) {
        c += t[k];
        u[k] = c & ((1ll << 52) - 1);
        c >>= 52;
    }
    w[0] = (uint32_t)u[0];
    w[1] = (uint32_t)(u[0] >> 32) | (uint32_t)(u[1] << 20);
    w[2] = (uint32_t)(u[1] >> 12);
    w[3] = (uint32_t)(u[1] >> 44) | (uint32_t)(u[2] << 8);
    w[4] = (uint32_t)(u[2] >> 24) | (uint32_t)((uint64_t)u[3] << 28);
    w[5] = (uint32_t)(u[3] >> 4);
    w[6] = (uint32_t)(u[3] >> 36) | (uint32_t)((uint64_t)u[4] << 16);
    w[7] = (uint32_t)(u[4] >> 16);
}

// ---- operations -------------------------------------------------------------------

// Always inlined here (a multiplication is about 240 instructions); code that
// runs a few times per signature goes through the out-of-line wrappers below.
UF_HD Fd fd_mul(Fd a, Fd b) {
    uint64_t c[10];
    fd_mac<FdBias<1, 0, 0, 1>, false>(c, a, b);
    return fd_reduce<FdBias<1, 0, 0, 1>, 1>(c);
}

// S a^2
template <int S>
UF_HD Fd fd_sqr_x(Fd a) {
    uint64_t c[10];
    fd_sac<FdBias<0, 1, 0, S>>(c, a);
    return fd_reduce<FdBias<0, 1, 0, S>, S>(c);
}

UF_HD Fd fd_sqr(const Fd& a) { return fd_sqr_x<1>(a); }

// a b - x
UF_HD Fd fd_mul_sub(Fd a, Fd b, Fd x) {
    uint64_t c[10];
    fd_mac<FdBias<1, 0, 1, 1>, false>(c, a, b);
    fd_inject_neg(c, x);
    return fd_reduce<FdBias<1, 0, 1, 1>, 1>(c);
}

// a^2 - 2 x
UF_HD Fd fd_sqr_sub2(Fd a, Fd x) {
    uint64_t c[10];
    fd_sac<FdBias<0, 1, 2, 1>>(c, a);
    fd_inject_neg2(c, x);
    return fd_reduce<FdBias<0, 1, 2, 1>, 1>(c);
}

// a^2 - x - y
UF_HD Fd fd_sqr_sub_sub(Fd a, Fd x, Fd y) {
    uint64_t c[10];
    fd_sac<FdBias<0, 1, 2, 1>>(c, a);
    fd_inject_neg(c, x);
    fd_inject_neg(c, y);
    return fd_reduce<FdBias<0, 1, 2, 1>, 1>(c);
}

// a^2 - x - 2 y
UF_HD Fd fd_sqr_sub_sub2(Fd a, Fd x, Fd y) {
    uint64_t c[10];
    fd_sac<FdBias<0, 1, 3, 1>>(c, a);
    fd_inject_neg(c, x);
    fd_inject_neg2(c, y);
    return fd_reduce<FdBias<0, 1, 3, 1>, 1>(c);
}

// a b - x y
UF_HD Fd fd_mul_mul_sub(Fd a, Fd b, Fd x, Fd y) {
    uint64_t c[10];
    fd_mac<FdBias<2, 0, 0, 1>, false>(c, a, b);
    UF_UNROLL
    for (int i = 0; i < 5; ++i) x.v[i] = -x.v[i];
    fd_mac<FdBias<2, 0, 0, 1>, true>(c, x, y);
    return fd_reduce<FdBias<2, 0, 0, 1>, 1>(c);
}

// a b - 2 x^2 (as a b - (2 x) x: the doubled digits of the cross products would
// not fit, so the square's columns are doubled as integers)
UF_HD Fd fd_mul_sub_2sqr(Fd a, Fd b, Fd x) {
    uint64_t c[10], e[10];
    fd_mac<FdBias<1, -2, 0, 1>, false>(c, a, b);
    fd_sac<FdNoBias>(e, x);
    UF_UNROLL
    for (int k = 0; k < 10; ++k) c[k] -= e[k] + e[k];
    return fd_reduce<FdBias<1, -2, 0, 1>, 1>(c);
}

UF_COLD Fd fd_sqr_n(Fd a, int n) {
    UF_NOUNROLL
    for (int i = 0; i < n; ++i) {
        uint64_t c[10];
        fd_sac<FdBias<0, 1, 0, 1>>(c, a);
        a = fd_reduce<FdBias<0, 1, 0, 1>, 1>(c);
    }
    return a;
}

// a + b, a - b, 2 a by digits: not strict
UF_HD Fd fd_add_l(const Fd& a, const Fd& b) {
    Fd r;
    UF_UNROLL
    for (int i = 0; i < 5; ++i) r.v[i] = a.v[i] + b.v[i];
    return r;
}

UF_HD Fd fd_sub_l(const Fd& a, const Fd& b) {
    Fd r;
    UF_UNROLL
    for (int i = 0; i < 5; ++i) r.v[i] = a.v[i] - b.v[i];
    return r;
}

UF_HD Fd fd_neg(const Fd& a) {
    Fd r;
    UF_UNROLL
    for (int i = 0; i < 5; ++i) r.v[i] = -a.v[i];
    return r;
}

// Zero test for a result of a multiplication: its value is in (-p, p), so it is
// 0 mod p only as 0, whose only strict digits are zeros.
UF_HD bool fd_is_zero(const Fd& a) {
    return a.v[0] == 0.0 && a.v[1] == 0.0 && a.v[2] == 0.0 && a.v[3] == 0.0 && a.v[4] == 0.0;
}

// Out-of-line forms for code outside the main loops.
UF_COLD Fd fdc_mul(Fd a, Fd b) { return fd_mul(a, b); }
UF_COLD Fd fdc_sqr(Fd a) { return fd_sqr(a); }
UF_COLD Fd fdc_mul_sub(Fd a, Fd b, Fd x) { return fd_mul_sub(a, b, x); }
UF_COLD Fd fdc_sqr_sub_sub(Fd a, Fd x, Fd y) { return fd_sqr_sub_sub(a, x, y); }
UF_COLD Fd fdc_sqr_sub_sub2(Fd a, Fd x, Fd y) { return fd_sqr_sub_sub2(a, x, y); }

// a + b and a - b as strict digits
UF_COLD Fd fdc_add(Fd a, Fd b) {
    Fd r = fd_add_l(a, b);
    fd_strict(r);
    return r;
}
UF_COLD Fd fdc_sub(Fd a, Fd b) {
    Fd r = fd_sub_l(a, b);
    fd_strict(r);
    return r;
}

// Whether a is a square mod p: its candidate root a^((p + 1) / 4), by the blocks of
// ones of fe_sqrt_candidate (fe.cuh), squared.
UF_COLD bool fd_is_square(Fd a) {
    const Fd x2 = fdc_mul(fdc_sqr(a), a), x3 = fdc_mul(fdc_sqr(x2), a);
    Fd t = fdc_mul(fd_sqr_n(x3, 3), x3);
    t = fdc_mul(fd_sqr_n(t, 3), x3);
    t = fdc_mul(fd_sqr_n(t, 2), x2);
    const Fd x22 = fdc_mul(fd_sqr_n(t, 11), t), x44 = fdc_mul(fd_sqr_n(x22, 22), x22);
    t = fdc_mul(fd_sqr_n(x44, 44), x44);
    t = fdc_mul(fd_sqr_n(t, 88), t);
    t = fdc_mul(fd_sqr_n(t, 44), x44);
    t = fdc_mul(fd_sqr_n(t, 3), x3);
    t = fdc_mul(fd_sqr_n(t, 23), x22);
    t = fdc_mul(fd_sqr_n(t, 6), x2);
    t = fd_sqr_n(t, 2);
    return fd_is_zero(fdc_mul_sub(t, t, a));
}

}  // namespace uf
