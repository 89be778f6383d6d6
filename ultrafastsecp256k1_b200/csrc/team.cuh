// Small calls: four or two warps per 32 signatures.
//
// A call of a few thousand signatures fills a fraction of the device, so its
// time is one signature's chain of dependent operations.  Here lane l of each of
// a block's four warps works on signature l, and the chain is cut between them:
//
//   warp 0: the key's point table (eis.cuh), while warp 1 parses the signature
//           and computes the scalars and their digits (ECDSA's s^-1 is as long
//           as the table) and, for BIP-340, whose s is the generator's scalar,
//           warps 2 and 3 sum half of its windows each;
//   all:    the table's scaling, an entry each in turn, and for ECDSA a quarter of
//           the generator's windows each;
//   all:    a range of the 44 digits each, R_w = sum of its digits times 8^low:
//           the additions are shared out, the doublings below a range repeated,
//           so the ranges grow towards the low end;
//   the partial sums in two steps; warp 0 does the check (isocheck.cuh).
//
// The doublings (129 of about 2.2 k cycles) cannot be shared, the rest mostly
// can.  The warps run the same code at the same time wherever that can be had:
// with the whole generator sum on warp 0 beside the others' digits a third of
// the issue slots waited for instructions (digits 390 k cycles instead of 325 k).
// It pays up to 32 signatures per SM, a warp for each of its schedulers; up to 64
// two warps share 32 signatures the same way (kWarps = 2: the scalars beside the
// table, all of the generator's windows after them).
// Verdicts as in kernels_verify_fp.cu.
#pragma once
#include "verify_fp.cuh"

#if defined(__CUDACC__)
namespace uf {

constexpr int kTeamLanes = 32;
constexpr int kTeamThreads = 4 * kTeamLanes;
constexpr int kDuoThreads = 2 * kTeamLanes;
// digits [low, high) of each warp: equal times at 6.8 k cycles per three
// doublings and as many per addition
static __device__ const uint8_t kTeamLow[5] = {0, 23, 35, 41, kEisDigits};
static __device__ const uint8_t kDuoLow[3] = {0, 29, kEisDigits};

// Shared memory of a block, in 16-byte columns of one lane each.
constexpr int kTabCells = 5 * kEisTab;       // the table
constexpr int kRhoCells = 3 * (kEisTab - 1); // its scale factors, then the partial sums of warps 1..3
constexpr int kPartCells = 8;
constexpr int kGenCells = 4 * kPartCells;    // the warps' partial sums of the generator's multiple
constexpr int kScalCells = 2;                // the generator's scalar
constexpr int kDigCells = 3;                 // 44 digit bytes
constexpr int kTeamCells = kTabCells + kRhoCells + kGenCells + kScalCells + kDigCells;
static_assert(3 * kPartCells <= kRhoCells, "partial sums reuse the scale factors' cells");
static_assert(32 <= kTabCells, "the plain verification's table lies in the point table");
constexpr size_t kTeamSmem = (size_t)kTeamCells * 16 * kTeamLanes;

__device__ __forceinline__ void put_fd(double2* cell, const Fd& a) {
    cell[0] = make_double2(a.v[0], a.v[1]);
    cell[kTeamLanes] = make_double2(a.v[2], a.v[3]);
    cell[2 * kTeamLanes].x = a.v[4];
}

__device__ __forceinline__ void get_fd(Fd& a, const double2* cell) {
    const double2 x = cell[0], y = cell[kTeamLanes];
    a.v[0] = x.x; a.v[1] = x.y; a.v[2] = y.x; a.v[3] = y.y;
    a.v[4] = cell[2 * kTeamLanes].x;
}

__device__ __forceinline__ void put_part(double2* c, const JacD& p) {
    const double v[16] = {p.X.v[0], p.X.v[1], p.X.v[2], p.X.v[3], p.X.v[4], p.Y.v[0], p.Y.v[1], p.Y.v[2],
                          p.Y.v[3], p.Y.v[4], p.Z.v[0], p.Z.v[1], p.Z.v[2], p.Z.v[3], p.Z.v[4], p.inf ? 1.0 : 0.0};
    UF_UNROLL
    for (int k = 0; k < kPartCells; ++k) c[k * kTeamLanes] = make_double2(v[2 * k], v[2 * k + 1]);
}

__device__ __forceinline__ JacD get_part(const double2* c) {
    double v[16];
    UF_UNROLL
    for (int k = 0; k < kPartCells; ++k) {
        const double2 t = c[k * kTeamLanes];
        v[2 * k] = t.x;
        v[2 * k + 1] = t.y;
    }
    JacD p;
    UF_UNROLL
    for (int k = 0; k < 5; ++k) {
        p.X.v[k] = v[k];
        p.Y.v[k] = v[5 + k];
        p.Z.v[k] = v[10 + k];
    }
    p.inf = v[15] != 0.0;
    return p;
}

// One signature per lane, verified by the block's four warps together (every
// thread calls it; `valid` false for lanes without one, whose pointers are not
// read).  The verdict is meaningful on warp 0.
template <int kKind, int kWarps = 4>
__device__ __forceinline__ bool team_verify(const uint8_t* msg, const uint8_t* pub, const uint8_t* sig, bool valid,
                                            const uint4* gt, const uint4* comb, uint4* smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double2* col = reinterpret_cast<double2*>(smem) + lane;
    const EisTab tab{col, kTeamLanes};
    double2* rho_c = col + kTabCells * kTeamLanes;
    double2* part_c = rho_c;
    double2* gen_c = rho_c + kRhoCells * kTeamLanes;
    uint4* scal = smem + lane + (kTabCells + kRhoCells + kGenCells) * kTeamLanes;
    uint8_t* dig = reinterpret_cast<uint8_t*>(smem + (kTeamCells - kDigCells) * kTeamLanes) + lane;
    Fd c, zc;                // warp 0
    bool odd = false, ok = valid;
    if (warp == 0) {
        uint32_t px[8];
        ok = ok && fp_parse_key<kKind>(px, odd, pub);
        if (ok) {
            Fd kx, ky, hs[kEisTab];
            iso_key(kx, ky, c, px);
            eis_path(tab, kx, ky, hs);
            zc = hs[kEisTab - 1];
            UF_NOUNROLL
            for (int k = kEisTab - 2; k >= 0; --k) {
                put_fd(rho_c + 3 * k * kTeamLanes, zc);
                if (k > 0) zc = fdc_mul(zc, hs[k]);
            }
            ok = !fd_is_zero(zc);        // 0: the key is not on the curve (isocheck.cuh)
        }
    } else if (warp == 1) {
        uint32_t r[8];
        Sc s;
        ok = ok && fp_parse_sig<kKind>(r, s, sig);
        if (ok) {
            Sc a, b;
            fp_scalars<kKind>(a, b, r, s, msg, pub, sig);
            GlvSplit split;
            glv_split(split, b);
            uint8_t d[kEisDigits];
            eis_recode(d, split);
            for (int k = 0; k < kEisDigits; ++k) dig[k * kTeamLanes] = d[k];
            scal[0] = make_uint4(a.v[0], a.v[1], a.v[2], a.v[3]);
            scal[kTeamLanes] = make_uint4(a.v[4], a.v[5], a.v[6], a.v[7]);
        }
    } else if (kKind == 1 && kWarps == 4 && ok) {
        uint32_t sw[8];
        Sc s;
        load_words8(sw, sig + 32);
        words_be_to_limbs(s.v, sw);
        const int half = (warp - 2) * (kCombWindows / 2);
        put_part(gen_c + warp * kPartCells * kTeamLanes, comb_mul<true>(s, comb, half, half + kCombWindows / 2));
    }
    constexpr bool kGenAfter = kKind != 1 || kWarps == 2;      // the generator's windows shared by all warps
    // a lane goes on when no warp refused its item
    __shared__ uint32_t good[2];
    const uint32_t mine = __ballot_sync(0xFFFFFFFFu, ok);
    if (warp < 2 && lane == 0) good[warp] = mine;
    __syncthreads();
    ok = ((good[0] & good[1]) >> lane) & 1u;
    if (ok) {
        UF_NOUNROLL
        for (int k = warp; k < kEisTab - 1; k += kWarps) {
            Fd rho;
            get_fd(rho, rho_c + 3 * k * kTeamLanes);
            eis_scale(tab, k, rho);
        }
        if (kGenAfter) {
            const uint4 lo = scal[0], hi = scal[kTeamLanes];
            const Sc a = {{lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w}};
            const int first = warp * (kCombWindows / kWarps);
            put_part(gen_c + warp * kPartCells * kTeamLanes,
                     comb_mul<true>(a, comb, first, first + kCombWindows / kWarps));
        }
    }
    __syncthreads();
    JacD A;
    jacd_set_inf(A);
    if (ok) {
        const uint8_t* ranges = kWarps == 4 ? kTeamLow : kDuoLow;
        const int low = ranges[warp], high = ranges[warp + 1];
        UF_NOUNROLL
        for (int q = high - 1; q >= 0; --q)
            eis_add_digit<true>(A, q >= low ? (uint32_t)dig[q * kTeamLanes] : kEisZero, q == high - 1, tab);
        if (warp != 0) put_part(part_c + (warp - 1) * kPartCells * kTeamLanes, A);
    }
    __syncthreads();
    const int c1 = kPartCells * kTeamLanes;
    if (kWarps == 4) {
        // first step: warps 0 and 2 on the key's sums, 1 and 3 on the generator's
        if (ok) {
            if (warp == 0) A = jacd_add(A, get_part(part_c));
            if (warp == 2) put_part(part_c + c1, jacd_add(A, get_part(part_c + 2 * c1)));
            if (warp == 1 && kKind != 1) put_part(gen_c, jacd_add(get_part(gen_c), get_part(gen_c + c1)));
            if (warp == 3) put_part(gen_c + 2 * c1, jacd_add(get_part(gen_c + 2 * c1), get_part(gen_c + 3 * c1)));
        }
        __syncthreads();
        if (ok) {
            if (warp == 0) A = jacd_add(A, get_part(part_c + c1));
            if (warp == 1 && kKind != 1) put_part(gen_c + 2 * c1, jacd_add(get_part(gen_c), get_part(gen_c + 2 * c1)));
        }
    } else if (ok) {
        if (warp == 0) A = jacd_add(A, get_part(part_c));
        if (warp == 1) put_part(gen_c + 2 * c1, jacd_add(get_part(gen_c), get_part(gen_c + c1)));
    }
    __syncthreads();
    if (warp != 0 || !ok) return false;
    const JacD B = get_part(gen_c + 2 * c1);
    A.Z = fdc_mul(A.Z, zc);
    uint32_t r[8];
    {
        Sc s;
        fp_parse_sig<kKind>(r, s, sig);
    }
    Fd den;
    int st = iso_prepare<kKind == 1>(tab, den, A, B, c, r);
    if (kKind == 1 && st == kIsoKeyInf) {
        st = kIsoPlain;                         // e = 0, unless the key is not on the curve
        for (int q = 0; q < kEisDigits; ++q)
            if (dig[q * kTeamLanes] != kEisZero) st = kIsoNo;
    }
    bool holds = false;
    if (st == kIsoSolve) {
        Fe inv;
        fd_pack(inv.v, den);
        if (is_zero256(inv.v)) {
            st = kIsoPlain;
        } else {
            fe_inv(inv, inv);
            holds = iso_finish<kKind == 1>(tab, inv, odd, false, kKind != 1 && r_below_p_minus_n(r));
        }
    }
    if (kKind != 1 && st == kIsoOnCurve) holds = iso_on_curve(tab);
    if (st == kIsoPlain) holds = plain_verify<kKind>(msg, pub, sig, gt, smem + lane, kTeamLanes);
    return holds;
}

}  // namespace uf
#endif  // __CUDACC__
