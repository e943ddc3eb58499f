// Interval certifier of packings on the GPU, verdict for verdict and digit
// for digit the reference certifier (cuda/certifier.cpp:738-912).
//
// Pipeline of one batch:
//   host    envelope checks (row count, square ids), literal slices in
//           square-id order, optional pandas round-trip of every literal
//           (certifier.cpp:914-929), packings bucketed by n;
//   kernel  cert_packing_kernel, one CTA per packing:
//             literal syntax + exact double-range and bound checks
//             (certifier.cpp:764-791), float corners + padded AABBs, Fix<9>
//             side measurement with Taylor sin/cos of the squares that can
//             hold an extreme (:793-854), bitonic sort of the AABBs,
//             sort-and-sweep (:856-883) with a directed-rounding FP64
//             evaluation of each pair that settles the float check and the
//             pairs whose sign it certifies; the rest go to a global list;
//   kernels the 7-, 15- and 58-limb interval SAT of the pairs still open at
//           63, 135 and 522 decimal digits (:885-899), each stage taking the
//           pairs the previous one left open;
//   host    reason strings, area bound, score, 50-decimal side (:900-911).
// The kernel file is compiled without multiply-add contraction so its double
// arithmetic rounds exactly like the reference's host code.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <charconv>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "common.cuh"
#include "fixdev.cuh"

namespace sqs {
namespace cert {

using fx::Fix;
using fx::Iv;
using fx::Lit;

constexpr int kMaxN = 1000;
constexpr int kMaxLiteral = 100;
constexpr uint32_t kNoKey = 0xffffffffu;
constexpr unsigned long long kNoPair = ~0ull;

enum : uint32_t { kCertOverlap = 1u, kUndecidable = 2u, kPairOverflow = 4u };
enum : uint32_t { kErrParse = 0, kErrRange = 1, kErrCoord = 2, kErrAngle = 3 };

struct PkOut {
    uint32_t err_key;          // 4 * square + kind of the first failing check
    uint32_t flags;            // kCertOverlap | kUndecidable | kPairOverflow
    unsigned long long fkey;   // (ii << 32 | jj) of the first float overlap in sweep order
    int32_t fu, fv;            // that pair, as square ids
    uint32_t undecided;        // pairs sent to the interval stages
    uint32_t pad;
    Fix<9> side;               // max(span_x, span_y) of the corners, Fix<9>
};

struct Pair {
    int32_t pk;
    int16_t u, v;
};

// A square's literals x, y, angle: back to back from text offset `off`.
struct SqText {
    uint32_t off, len[3];
};
constexpr uint32_t kLenMax = 1u << 20;  // a longer literal is read as far as this
// The offsets have 32 bits, so the last literal a square's record names must
// start here at the latest; calls with more text are refused.
constexpr int64_t kOffMax = (1ll << 32) - kLenMax;

struct Consts {
    Fix<9> half_pi9, two_pi9, half9;
    Iv<7> half_pi7, half7;
    Iv<15> half_pi15, half15;
    Iv<58> half_pi58, half58;
};

__constant__ Consts c_consts;
// Decimal thresholds of the reference's double checks, exact:
//   strtod overflows      iff |v| >= 2^1024 - 2^970
//   |x| > 1e4 as a double iff |v| >  1e4 + 2^-40 (the tie rounds to 1e4)
//   |a| > 100 as a double iff |v| >  100 + 2^-47
__device__ const char c_inf_edge[] =
    "179769313486231580793728971405303415079934132710037826936173778980444968292764750946649017977587"
    "207096330286416692887910946555547851940402630657488671505820681908902000708383676273854845817711"
    "531764475730270069855571366959622842914819860834936475292719074168444365510704342711559699508093"
    "04222336";
__device__ const char c_coord_edge[] = "10000.0000000000009094947017729282379150390625";
__device__ const char c_angle_edge[] = "100.00000000000000710542735760100185871124267578125";

const char* kHalfPi =
    "1.5707963267948966192313216916397514420985846996875529104874722961539082031431044993140174126710585339"
    "9107404325664115332354692230477529111586267970406424055872514205135096926055277982231147447746519098"
    "2214405487832966723064237824116893391582635600954572824283161565386415559563044484210977355059400485"
    "7492389293099245510655716316154220989218499846888949675083019800051100514872368941154883214599416258"
    "7630228031340772652010253145121415210968393898212262598912242342639728019727481121132833606270987663"
    "3184560871636462872546121833290233099787539786414835847812261143213250625359595866490484368352035968";
const char* kTwoPi =
    "6.2831853071795864769252867665590057683943387987502116419498891846156328125724179972560696506842341359"
    "6429617302656461329418768921910116446345071881625696223490056820540387704221111928924589790986076392"
    "8857621951331866892256951296467573566330542403818291297132646261545662238252177936843909420237601942"
    "9969557172396982042622865264616883956873999387555798700332079200204402059489475764619532858397665035"
    "0520912125363090608041012580485660843873575592848905039564896937055891207890992448453133442508395065"
    "2738243486545851490184487333160932399150159145659343391249044572853002501438383465961937473408143872";

FX_HD bool is_space(char c) { return c == ' ' || c == '\t' || c == '\n' || c == '\v' || c == '\f' || c == '\r'; }
FX_HD bool is_digit(char c) { return c >= '0' && c <= '9'; }

// is_valid_decimal (certifier.cpp:505-529) + the digit/point analysis of
// parse_decimal_fix (:265-333).  `base` is the text offset of `s`.
FX_HD bool analyze(const char* s, int len, uint32_t base, Lit& L, int max_len = kMaxLiteral) {
    int a = 0, b = len;
    while (a < b && is_space(s[a])) ++a;
    while (b > a && is_space(s[b - 1])) --b;
    const int n = b - a;
    L.off = base + (uint32_t)a;
    L.point = 0;
    L.ndig = 0;
    L.dot = -1;
    L.neg = 0;
    L.dyadic = 0;
    L.zero_str = 0;
    L.pad = 0;
    if (n <= 0 || n > max_len) return false;
    const char* t = s + a;
    int i = 0;
    if (t[0] == '+' || t[0] == '-') {
        L.neg = t[0] == '-';
        ++i;
    }
    if (i >= n) return false;
    L.off = base + (uint32_t)(a + i);
    bool any = false;
    int nd = 0, frac = 0;
    while (i < n && is_digit(t[i])) { any = true; ++i; ++nd; }
    if (i < n && t[i] == '.') {
        L.dot = (int16_t)nd;
        ++i;
        while (i < n && is_digit(t[i])) { any = true; ++i; ++nd; ++frac; }
    }
    if (!any) return false;
    long long ex = 0;
    if (i < n && (t[i] == 'e' || t[i] == 'E')) {
        ++i;
        int es = 1;
        if (i < n && (t[i] == '+' || t[i] == '-')) es = t[i++] == '-' ? -1 : 1;
        bool ed = false;
        while (i < n && is_digit(t[i])) {
            ed = true;
            if (ex < 100000000LL) ex = ex * 10 + (t[i] - '0');
            ++i;
        }
        if (!ed) return false;
        ex *= es;
    }
    if (i != n) return false;
    L.ndig = (uint16_t)nd;
    L.point = (int32_t)((long long)nd - frac + ex);
    L.zero_str = (n == 1 && t[0] == '0') || (n == 3 && t[0] == '0' && t[1] == '.' && t[2] == '0');
    return true;
}

// is_dyadic_decimal_str (certifier.cpp:335-381).
FX_HD bool dyadic(const char* text, const Lit& L) {
    int nd = L.ndig;
    long long places = (long long)L.ndig - L.point;
    while (places > 0 && nd > 0 && fx::lit_digit(text, L, nd - 1) == 0) { --nd; --places; }
    if (places <= 0) return true;
    if (places > 25) return false;
    char dg[kMaxLiteral + 4];
    int m = 0;
    for (int k = 0; k < nd; ++k) dg[m++] = (char)fx::lit_digit(text, L, k);
    for (long long k = 0; k < places; ++k) {
        if (m == 0) return true;
        if (dg[m - 1] % 5) return false;
        int rem = 0, w = 0;
        for (int r = 0; r < m; ++r) {
            const int cur = rem * 10 + dg[r];
            if (w > 0 || cur / 5) dg[w++] = (char)(cur / 5);
            rem = cur % 5;
        }
        m = w;
    }
    return true;
}

// Compare |literal| with a positive decimal constant (no sign, no exponent)
// of cl characters with its point at cdot (-1: none).
__device__ int cmp_abs_const(const char* text, const Lit& L, const char* c, int cl, int cdot) {
    const int cint = cdot < 0 ? cl : cdot;           // constant's integer digit count
    const int cnd = cdot < 0 ? cl : cl - 1;
    auto cdig = [&](long long k) -> int {           // k-th digit of the constant
        if (k < 0 || k >= cnd) return 0;
        return c[(cdot >= 0 && k >= cdot) ? k + 1 : k] - '0';
    };
    int lz = 0;
    while (lz < L.ndig && fx::lit_digit(text, L, lz) == 0) ++lz;
    if (lz == L.ndig) return -1;  // zero
    const long long le = (long long)L.point - lz;    // digits before the point from the first non-zero
    int cz = 0;
    while (cz < cnd && cdig(cz) == 0) ++cz;
    const long long ce = (long long)cint - cz;
    if (le != ce) return le < ce ? -1 : 1;
    const long long len = (long long)(L.ndig - lz) > (long long)(cnd - cz) ? (L.ndig - lz) : (cnd - cz);
    for (long long k = 0; k < len; ++k) {
        const int a = fx::lit_digit(text, L, lz + k), b = cdig(cz + k);
        if (a != b) return a < b ? -1 : 1;
    }
    return 0;
}

// Float SAT prefilter (certifier.cpp:543-588) on squares with centre (x, y)
// and cached cos/sin (c, s) of the reduced angle.
struct FSq {
    double x, y, c, s;
};

__device__ __forceinline__ void fcorners(const FSq& q, double* cx, double* cy) {
    const double ux = 0.5 * q.c - 0.5 * q.s, uy = 0.5 * q.s + 0.5 * q.c;
    const double vx = -0.5 * q.c - 0.5 * q.s, vy = -0.5 * q.s + 0.5 * q.c;
    cx[0] = q.x + ux; cy[0] = q.y + uy;
    cx[1] = q.x + vx; cy[1] = q.y + vy;
    cx[2] = q.x - ux; cy[2] = q.y - uy;
    cx[3] = q.x - vx; cy[3] = q.y - vy;
}

__device__ __noinline__ int float_sat(const FSq& p, const FSq& q) {
    double px[4], py[4], qx[4], qy[4];
    fcorners(p, px, py);
    fcorners(q, qx, qy);
    const double ax[4][2] = {{p.c, p.s}, {-p.s, p.c}, {q.c, q.s}, {-q.s, q.c}};
    double worst = 1e300;
    for (int a = 0; a < 4; ++a) {
        double lo1 = 1e300, hi1 = -1e300, lo2 = 1e300, hi2 = -1e300;
        for (int k = 0; k < 4; ++k) {
            const double u = ax[a][0] * px[k] + ax[a][1] * py[k];
            const double v = ax[a][0] * qx[k] + ax[a][1] * qy[k];
            if (u < lo1) lo1 = u;
            if (u > hi1) hi1 = u;
            if (v < lo2) lo2 = v;
            if (v > hi2) hi2 = v;
        }
        const double ov = fmin(hi1, hi2) - fmax(lo1, lo2);
        if (ov < -1e-8) return 1;
        if (ov < worst) worst = ov;
    }
    return worst > 1e-8 ? -1 : 0;
}

// ------------------------------------------------------------ pair decision
// One directed-rounding FP64 evaluation of the exact overlap of two squares
// along the four axes.  Both squares have support 1/2 (own axes) and
// (|cos d| + |sin d|) / 2 (the other's, d the angle between them), so every
// axis's overlap is r - |v|, r = 1/2 + (|cos d| + |sin d|) / 2, v the centre
// difference along the axis: 12 products of enclosures instead of the 64 of
// two times four corners on four axes.  (Where one projection contains the
// other the reference's overlap is smaller than r - |v|, but both are at
// least 1 there.)  Enclosures are midpoint and radius, radii rounded up.
//
// It decides the reference's float check wherever that check's own rounding
// cannot matter (kTol around its +-1e-8 thresholds; the check itself runs on
// the rest), and of the pairs that leave open those the interval stages are
// certain to decide the same way:
//   * separated when some axis's overlap lies strictly below zero,
//     overlapping when every axis's lies strictly above: the exact overlap of
//     the exact decimal inputs then has that sign and is at least 2^-120 in
//     magnitude (the spacing of the doubles involved), which the 7-limb stage
//     (widths below 1e-60) resolves alike;
//   * two axis-aligned squares (angle literals exactly zero, the reference's
//     flat path) whose literals on an axis, and square 0's, are dyadic within
//     25 decimal places are compared exactly on it: touching edges count as
//     separated, as they do there.
// The rest goes to the 7-limb stage.
//
// Bounds.  A coordinate is kept as its integer part and its fraction, the
// latter within 2^-51 (one correctly rounded division, two additions), so a
// centre difference is within 2^-48 of exact.  The angle's double is within
// (|a| + 1) 2^-50, sin and cos (documented 2 ulp) within w of their exact
// values, w = (|a| + 1) 2^-49 + 2^-50.
struct MR {
    double m, r;  // |value - m| <= r
};
__device__ __forceinline__ double round_err(double m) { return __fma_ru(fabs(m), 0x1p-53, 0x1p-1000); }
__device__ __forceinline__ MR mr_mul(MR a, MR b) {
    const double m = __dmul_rn(a.m, b.m);
    const double r = __fma_ru(fabs(a.m), b.r, __fma_ru(fabs(b.m), a.r, __fma_ru(a.r, b.r, round_err(m))));
    return MR{m, r};
}
__device__ __forceinline__ MR mr_add(MR a, MR b) {
    const double m = __dadd_rn(a.m, b.m);
    return MR{m, __dadd_ru(__dadd_ru(a.r, b.r), round_err(m))};
}
__device__ __forceinline__ MR mr_neg(MR a) { return MR{-a.m, a.r}; }

enum : uint32_t { kSqFlat = 1u, kSqExactX = 2u, kSqExactY = 4u, kSqDyadicX = 8u, kSqDyadicY = 16u };

// A square as the pair decision reads it (shared memory, by square id).
struct PairSq {
    double* xf;     // fractions of the coordinates, with their sign
    double* yf;
    float* w;       // error bound of the cached cos / sin
    int16_t* xi;    // integer parts, with their sign
    int16_t* yi;
    uint8_t* fl;    // kSq* bits
};

// Whether two dyadic literals are at least 1 apart, exactly (27 decimals hold them).
__device__ __noinline__ bool apart_exact(const char* text, const Lit& p, const Lit& q) {
    Fix<3> d = fx::sub(fx::parse<3>(text, p, 0), fx::parse<3>(text, q, 0));
    d.neg = 0;
    return fx::cmp(d, fx::of_int<3>(1)) >= 0;
}

// 1 separated, -1 overlap by the float check, -2 overlap by the intervals,
// 2 left to the multi-limb stages.  u < v are the squares' ids in the packing
// whose literals start at L0.
__device__ __forceinline__ int decide_pair(const FSq* sq, const PairSq& ps, int u, int v, const char* text, const Lit* L0) {
    const FSq p = sq[u], q = sq[v];
    const double wp = ps.w[u], wq = ps.w[v];
    const MR dx{__dadd_rn((double)(ps.xi[v] - ps.xi[u]), __dsub_rn(ps.xf[v], ps.xf[u])), 0x1p-48};
    const MR dy{__dadd_rn((double)(ps.yi[v] - ps.yi[u]), __dsub_rn(ps.yf[v], ps.yf[u])), 0x1p-48};
    const MR cp{p.c, wp}, sp{p.s, wp}, cq{q.c, wq}, sq_{q.s, wq};
    const MR cd = mr_add(mr_mul(cp, cq), mr_mul(sp, sq_)), sd = mr_add(mr_mul(sp, cq), mr_neg(mr_mul(cp, sq_)));
    const MR sum = mr_add(MR{fabs(cd.m), cd.r}, MR{fabs(sd.m), sd.r});
    const MR rad = mr_add(MR{0.5, 0.0}, MR{0.5 * sum.m, 0.5 * sum.r});
    const MR vv[4] = {mr_add(mr_mul(dx, cp), mr_mul(dy, sp)), mr_add(mr_mul(dy, cp), mr_neg(mr_mul(dx, sp))),
                      mr_add(mr_mul(dx, cq), mr_mul(dy, sq_)), mr_add(mr_mul(dy, cq), mr_neg(mr_mul(dx, sq_)))};
    double hi = 1e300, lo = 1e300;  // bounds of the smallest overlap
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const MR ov = mr_add(rad, MR{-fabs(vv[k].m), vv[k].r});
        hi = fmin(hi, __dadd_ru(ov.m, ov.r));
        lo = fmin(lo, __dsub_rd(ov.m, ov.r));
    }
    // the float check's rounding: its corners and projections are within
    // 2^-45 of the coordinates' size of exact
    const double tol = 0x1p-44 * (fabs(p.x) + fabs(p.y) + fabs(q.x) + fabs(q.y) + 4.0);
    if (hi < -1e-8 - tol) return 1;
    if (lo > 1e-8 + tol) return -1;
    if (!(lo > -1e-8 + tol && hi < 1e-8 - tol)) {
        const int f = float_sat(p, q);
        if (f != 0) return f;
    }
    const uint32_t fl = ps.fl[u] & ps.fl[v];
    if (fl & kSqFlat) {
        // per axis: apart, overlapping, or open (the exact distances of exact
        // coordinates, the bounds above, or 3-limb arithmetic)
        const uint32_t fo = fl & ps.fl[0];
        bool open = false;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const double d = fabs(k ? dy.m : dx.m);
            if (fo & (k ? kSqExactY : kSqExactX)) {
                if (d >= 1.0) return 1;
            } else if (d - 0x1p-47 > 1.0) {
                return 1;
            } else if (!(d + 0x1p-47 < 1.0)) {
                if (!(fo & (k ? kSqDyadicY : kSqDyadicX))) open = true;
                else if (apart_exact(text, L0[3 * u + k], L0[3 * v + k])) return 1;
            }
        }
        return open ? 2 : -2;
    }
    if (hi < 0.0) return 1;
    return lo > 0.0 ? -2 : 2;
}

// The warp's largest (or smallest) value among the lanes that have one, on
// every lane: lanes drop out limb by limb, sign first, one warp reduction a
// limb (five rounds of exchanging and comparing whole values took 20,000
// cycles for the four extremes, most of it local memory).
template <int F>
__device__ __forceinline__ bool warp_extreme(Fix<F>& v, bool have, bool want_min) {
    if (!__any_sync(0xffffffffu, have)) return false;
    const bool flip = (v.neg != 0) != want_min;  // larger magnitude is worse
    bool in = have;
    const uint32_t s = (v.neg != 0) == want_min ? 2u : 1u;  // the wanted sign first
    const uint32_t best = __reduce_max_sync(0xffffffffu, in ? s : 0u);
    in = in && s == best;
#pragma unroll
    for (int i = 0; i <= F; ++i) {
        const uint32_t k = flip ? ~v.d[i] : v.d[i];
        const uint32_t m = __reduce_max_sync(0xffffffffu, in ? k : 0u);
        in = in && k == m;
    }
    const int src = __ffs(__ballot_sync(0xffffffffu, in)) - 1;
#pragma unroll
    for (int i = 0; i <= F; ++i) v.d[i] = __shfl_sync(0xffffffffu, v.d[i], src);
    v.neg = __shfl_sync(0xffffffffu, v.neg, src);
    return true;
}

// One CTA per packing: checks, side measurement, sort and sweep.
template <int T, int NMAX>
__global__ void __launch_bounds__(T, 512 / T) cert_packing_kernel(
    int count, const int32_t* __restrict__ bucket, const int32_t* __restrict__ pk_n,
    const int64_t* __restrict__ pk_sq0, const char* __restrict__ text, const SqText* __restrict__ raw,
    Lit* __restrict__ lits, PkOut* __restrict__ out,
    Pair* __restrict__ pairs, uint32_t* __restrict__ pair_count, uint32_t pair_cap) {
    constexpr int W = T / 32;
    constexpr int NP = NMAX;  // power of two
    extern __shared__ __align__(16) unsigned char dyn[];
    FSq* sq = reinterpret_cast<FSq*>(dyn);                    // by square id
    double* bx0 = reinterpret_cast<double*>(sq + NMAX);       // padded AABBs by square id
    double* bx1 = bx0 + NMAX;
    double* by0 = bx1 + NMAX;
    double* by1 = by0 + NMAX;
    double* key = by1 + NMAX;
    PairSq ps;
    ps.xf = key + NP;
    ps.yf = ps.xf + NMAX;
    ps.w = reinterpret_cast<float*>(ps.yf + NMAX);
    ps.xi = reinterpret_cast<int16_t*>(ps.w + NMAX);
    ps.yi = ps.xi + NMAX;
    int16_t* idx = ps.yi + NMAX;                              // candidates of the side, then the sort
    ps.fl = reinterpret_cast<uint8_t*>(idx + NP);
    __shared__ Fix<9> series[T];                              // sin and cos series of a pair of threads
    __shared__ double box[W][4];
    __shared__ int s_cand;
    __shared__ Fix<9> ext[W][4];
    __shared__ int ext_have[W][4];
    __shared__ Fix<9> org[2];
    __shared__ uint32_t s_err;
    __shared__ unsigned long long s_fkey;
    __shared__ uint32_t s_undecided;

    const int b = blockIdx.x;
    if (b >= count) return;
    const int pk = bucket[b];
    const int n = pk_n[pk];
    const int64_t s0 = pk_sq0[pk];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_err = kNoKey;
        s_fkey = kNoPair;
        s_undecided = 0;
        s_cand = 0;
    }
    __syncthreads();

    // 1. literal syntax and the double-range checks, first failure by square id
    for (int i = tid; i < n; i += T) {
        uint32_t kind = kNoKey;
        Lit Ls[3];
        const SqText st = raw[s0 + i];
        uint32_t off = st.off;
        for (int k = 0; k < 3; off += st.len[k], ++k) {
            const bool ok = analyze(text + off, (int)min(st.len[k], kLenMax), off, Ls[k]);
            if (!ok && kind == kNoKey) kind = kErrParse;
        }
        if (kind == kNoKey) {
            for (int k = 0; k < 3; ++k) {
                if (cmp_abs_const(text, Ls[k], c_inf_edge, sizeof(c_inf_edge) - 1, -1) >= 0) kind = kErrRange;
                Ls[k].dyadic = dyadic(text, Ls[k]);
            }
        }
        if (kind == kNoKey && (cmp_abs_const(text, Ls[0], c_coord_edge, sizeof(c_coord_edge) - 1, 5) > 0 ||
                               cmp_abs_const(text, Ls[1], c_coord_edge, sizeof(c_coord_edge) - 1, 5) > 0))
            kind = kErrCoord;
        if (kind == kNoKey && cmp_abs_const(text, Ls[2], c_angle_edge, sizeof(c_angle_edge) - 1, 3) > 0) kind = kErrAngle;
        for (int k = 0; k < 3; ++k) lits[3 * (s0 + i) + k] = Ls[k];
        if (kind != kNoKey) atomicMin(&s_err, 4u * (uint32_t)i + kind);
    }
    __syncthreads();
    if (s_err != kNoKey) {
        if (tid == 0) {
            out[pk].err_key = s_err;
            out[pk].fkey = kNoPair;
            out[pk].flags = 0;
            out[pk].undecided = 0;
        }
        return;
    }
    if (tid == 0) {
        org[0] = fx::parse<9>(text, lits[3 * s0], 0);
        org[1] = fx::parse<9>(text, lits[3 * s0 + 1], 0);
    }
    __syncthreads();

    // 2. float geometry of every square, and what the pair decision reads
    const Consts& C = c_consts;
    double gx0 = 1e300, gx1 = -1e300, gy0 = 1e300, gy1 = -1e300;
    for (int i = tid; i < n; i += T) {
        const Lit lx = lits[3 * (s0 + i)], ly = lits[3 * (s0 + i) + 1], la = lits[3 * (s0 + i) + 2];
        const Fix<9> x = fx::parse<9>(text, lx, 0), y = fx::parse<9>(text, ly, 0);
        const Fix<9> A = fx::parse<9>(text, la, 0);
        const double a = fx::approx(A);
        const long long turns = (long long)floor(a / 6.283185307179586476925);
        double ang = a;
        if (turns != 0 || A.neg || a > 6.28) {  // (else the reduction below would leave A as it is)
            Fix<9> red = fx::sub<9, true>(A, fx::mul(fx::of_int<9>(turns), C.two_pi9, 0));
            if (red.neg && !fx::is_zero(red)) red = fx::add<9, true>(red, C.two_pi9);
            if (fx::cmp<9, true>(red, C.two_pi9) >= 0) red = fx::sub<9, true>(red, C.two_pi9);
            ang = fx::approx(red);
        }
        FSq q;
        q.x = fx::approx(fx::sub<9, true>(x, org[0]));
        q.y = fx::approx(fx::sub<9, true>(y, org[1]));
        q.c = cos(ang);
        q.s = sin(ang);
        sq[i] = q;
        double cx[4], cy[4];
        fcorners(q, cx, cy);
        double x0 = cx[0], x1 = cx[0], y0 = cy[0], y1 = cy[0];
        for (int k = 1; k < 4; ++k) {
            x0 = fmin(x0, cx[k]); x1 = fmax(x1, cx[k]);
            y0 = fmin(y0, cy[k]); y1 = fmax(y1, cy[k]);
        }
        bx0[i] = x0 - 1e-7; by0[i] = y0 - 1e-7; bx1[i] = x1 + 1e-7; by1[i] = y1 + 1e-7;
        gx0 = fmin(gx0, x0); gx1 = fmax(gx1, x1);
        gy0 = fmin(gy0, y0); gy1 = fmax(gy1, y1);
        uint32_t fl = 0;
        auto split = [&](const Fix<9>& v, const Lit& L, double& f, int16_t& whole, uint32_t dy, uint32_t ex) {
            f = __ddiv_rn((double)v.d[1], 1e9) + ((double)v.d[2] * 1e-18 + (double)v.d[3] * 1e-27);
            f = v.neg ? -f : f;
            whole = (int16_t)(v.neg ? -(int)v.d[0] : (int)v.d[0]);  // |v| <= 1e4 (checked above)
            uint32_t rest = 0;
            for (int k = 2; k <= 9; ++k) rest |= v.d[k];
            if (L.dyadic) fl |= rest ? dy : dy | ex;
        };
        split(x, lx, ps.xf[i], ps.xi[i], kSqDyadicX, kSqExactX);
        split(y, ly, ps.yf[i], ps.yi[i], kSqDyadicY, kSqExactY);
        bool flat = true;  // every digit of the angle is zero
        for (int k = 0; k < la.ndig && flat; ++k) flat = fx::lit_digit(text, la, k) == 0;
        ps.fl[i] = (uint8_t)(fl | (flat ? kSqFlat : 0u));
        ps.w[i] = flat ? 0.f : __double2float_ru(__fma_ru(__dadd_ru(fabs(ang), 1.0), 0x1p-49, 0x1p-50));
    }
    for (int o = 16; o > 0; o >>= 1) {
        gx0 = fmin(gx0, __shfl_xor_sync(0xffffffffu, gx0, o));
        gx1 = fmax(gx1, __shfl_xor_sync(0xffffffffu, gx1, o));
        gy0 = fmin(gy0, __shfl_xor_sync(0xffffffffu, gy0, o));
        gy1 = fmax(gy1, __shfl_xor_sync(0xffffffffu, gy1, o));
    }
    if (lane == 0) {
        box[warp][0] = gx0;
        box[warp][1] = gx1;
        box[warp][2] = gy0;
        box[warp][3] = gy1;
    }
    __syncthreads();
    for (int w = 0; w < W; ++w) {
        gx0 = fmin(gx0, box[w][0]);
        gx1 = fmax(gx1, box[w][1]);
        gy0 = fmin(gy0, box[w][2]);
        gy1 = fmax(gy1, box[w][3]);
    }
    // The side: spans of the Fix<9> corners.  A double corner is within 1e-9
    // of its Fix<9> value, so only squares whose float box reaches within
    // 1e-8 of the packing's can hold an extreme: the 81-digit sin and cos are
    // taken of those alone (a tilted layout has a handful; all of them before,
    // which was most of this kernel), by two threads a square, one a series.
    for (int i = tid; i < n; i += T) {
        if (bx0[i] + 1e-7 <= gx0 + 1e-8 || bx1[i] - 1e-7 >= gx1 - 1e-8 || by0[i] + 1e-7 <= gy0 + 1e-8 ||
            by1[i] - 1e-7 >= gy1 - 1e-8)
            idx[atomicAdd(&s_cand, 1)] = (int16_t)i;
    }
    __syncthreads();
    Fix<9> ex[2];  // smallest and largest corner coordinate of this thread (an even one's x, an odd one's y)
    fx::set_zero(ex[0]);
    fx::set_zero(ex[1]);
    bool have[2] = {false, false};
    const double gext[4] = {gx0, gx1, gy0, gy1};
    const int ncand = s_cand;
    for (int base = 0; base < ncand; base += T / 2) {
        const int k = base + tid / 2;
        const bool in = k < ncand;
        const int i = in ? idx[k] : 0;
        const Lit la = lits[3 * (s0 + i) + 2];
        const Fix<9> A = fx::parse<9>(text, la, 0);
        const bool turned = in && !(la.zero_str || fx::is_zero(A));
        int quad = 0;
        if (turned) fx::sincos_series(A, C.half_pi9, tid & 1, series[tid], quad);
        __syncwarp();
        if (in) {  // the even thread takes the x extremes, the odd one the y extremes
            Fix<9> hc = C.half9, hs;  // halves of cos and sin (an untilted square's are 1/2 and 0)
            fx::set_zero(hs);
            if (turned) {
                Fix<9> sn, cs;
                fx::sincos_quadrant(series[tid | 1], series[tid & ~1], quad, sn, cs);
                hc = fx::mul(C.half9, cs, 0);
                hs = fx::mul(C.half9, sn, 0);
            }
            // corners: x + a, x - b, x - a, x + b and y + b, y + a, y - b, y - a
            const Fix<9> a = fx::sub<9, true>(hc, hs), b = fx::add<9, true>(hs, hc);
            const int ax = tid & 1;
            const Fix<9> Z = fx::sub<9, true>(fx::parse<9>(text, lits[3 * (s0 + i) + ax], 0), org[ax]);
            double cx[4], cy[4];
            fcorners(sq[i], cx, cy);
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {  // only corners that can be the extreme
                const double z = ax ? cy[c] : cx[c];
                const bool lo = z <= gext[2 * ax] + 1e-8, hi = z >= gext[2 * ax + 1] - 1e-8;
                if (!lo && !hi) continue;
                Fix<9> off = (c & 1) == ax ? a : b;
                if (ax ? c >= 2 : (c == 1 || c == 2)) off = fx::neg(off);
                const Fix<9> v = fx::add<9, true>(Z, off);
                if (lo && (!have[0] || fx::cmp<9, true>(v, ex[0]) < 0)) {
                    ex[0] = v;
                    have[0] = true;
                }
                if (hi && (!have[1] || fx::cmp<9, true>(v, ex[1]) > 0)) {
                    ex[1] = v;
                    have[1] = true;
                }
            }
        }
        __syncwarp();
    }
    for (int k = 0; k < 4; ++k) {
        Fix<9> v = ex[k & 1];
        const bool got = warp_extreme(v, have[k & 1] && (tid & 1) == k / 2, (k & 1) == 0);
        if (lane == 0) {
            ext_have[warp][k] = got;
            if (got) ext[warp][k] = v;
        }
    }
    __syncthreads();  // the candidates are read
    // 3. sort the AABBs by their padded min x, ties by square id
    for (int i = tid; i < NP; i += T) {
        key[i] = i < n ? bx0[i] : 1e300;
        idx[i] = (int16_t)i;
    }
    __syncthreads();
    if (warp == 0) {
        Fix<9> e[4];
        for (int k = 0; k < 4; ++k) {
            const bool own = lane < W && ext_have[lane][k];
            e[k] = ext[own ? lane : 0][k];
            warp_extreme(e[k], own, (k & 1) == 0);
        }
        if (lane == 0) {
            const Fix<9> sx = fx::sub(e[1], e[0]), sy = fx::sub(e[3], e[2]);
            out[pk].side = fx::cmp(sx, sy) >= 0 ? sx : sy;
        }
    }
    int np = 1;
    while (np < n) np <<= 1;
    for (int k = 2; k <= np; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = tid; i < np; i += T) {
                const int l = i ^ j;
                if (l > i) {
                    const bool up = (i & k) == 0;
                    const double ki = key[i], kl = key[l];
                    const int16_t ii = idx[i], il = idx[l];
                    const bool gt = ki > kl || (ki == kl && ii > il);
                    if (gt == up) {
                        key[i] = kl; key[l] = ki;
                        idx[i] = il; idx[l] = ii;
                    }
                }
            }
            __syncthreads();
        }
    }

    // 4. sort and sweep with the pair decision
    for (int ii = tid; ii < n; ii += T) {
        const int i = idx[ii];
        const double ix1 = bx1[i], iy0 = by0[i], iy1 = by1[i], ix0 = bx0[i];
        for (int jj = ii + 1; jj < n; ++jj) {
            const int j = idx[jj];
            if (bx0[j] > ix1) break;
            if (ix1 < bx0[j] || bx1[j] < ix0 || iy1 < by0[j] || by1[j] < iy0) continue;
            const int u = min(i, j), v = max(i, j);
            const int r = decide_pair(sq, ps, u, v, text, lits + 3 * s0);
            if (r == -1) {
                atomicMin(&s_fkey, ((unsigned long long)ii << 32) | (unsigned long long)jj);
            } else if (r == -2) {
                atomicOr(&out[pk].flags, kCertOverlap);
            } else if (r == 2) {
                atomicAdd(&s_undecided, 1u);
                const uint32_t slot = atomicAdd(pair_count, 1u);
                if (slot < pair_cap) pairs[slot] = Pair{pk, (int16_t)u, (int16_t)v};
                else atomicOr(&out[pk].flags, kPairOverflow);
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        out[pk].err_key = kNoKey;
        out[pk].fkey = s_fkey;
        out[pk].undecided = s_undecided;
        if (s_fkey != kNoPair) {
            const int a = idx[(int)(s_fkey >> 32)], c = idx[(int)(s_fkey & 0xffffffffu)];
            out[pk].fu = min(a, c);
            out[pk].fv = max(a, c);
        }
    }
}

// ------------------------------------------------------------ interval stages
template <int F>
struct IvSq {
    bool flat;
    Iv<F> c, s, x0, x1, y0, y1;
    Iv<F> px[4], py[4];
};

template <int F>
__device__ __forceinline__ const Iv<F>& half_pi_iv();
template <>
__device__ __forceinline__ const Iv<7>& half_pi_iv<7>() { return c_consts.half_pi7; }
template <>
__device__ __forceinline__ const Iv<15>& half_pi_iv<15>() { return c_consts.half_pi15; }
template <>
__device__ __forceinline__ const Iv<58>& half_pi_iv<58>() { return c_consts.half_pi58; }
template <int F>
__device__ __forceinline__ const Iv<F>& half_iv();
template <>
__device__ __forceinline__ const Iv<7>& half_iv<7>() { return c_consts.half7; }
template <>
__device__ __forceinline__ const Iv<15>& half_iv<15>() { return c_consts.half15; }
template <>
__device__ __forceinline__ const Iv<58>& half_iv<58>() { return c_consts.half58; }

// ensure_sq_iv (certifier.cpp:600-635)
template <int F>
__device__ __noinline__ void make_ivsq(const char* text, const Lit* L3, const Iv<F>& ox, const Iv<F>& oy, IvSq<F>& e) {
    const Iv<F>& h = half_iv<F>();
    const Iv<F> x = fx::isub(fx::parse_iv<F>(text, L3[0]), ox);
    const Iv<F> y = fx::isub(fx::parse_iv<F>(text, L3[1]), oy);
    fx::sincos_iv(fx::parse_iv<F>(text, L3[2]), half_pi_iv<F>(), e.s, e.c);
    e.flat = fx::is_zero(e.s.lo) && fx::is_zero(e.s.hi);
    if (e.flat) {
        e.x0 = fx::isub(x, h);
        e.x1 = fx::iadd(x, h);
        e.y0 = fx::isub(y, h);
        e.y1 = fx::iadd(y, h);
    }
    const Iv<F> hc = fx::imul(h, e.c), hs = fx::imul(h, e.s), nh = fx::ineg(h);
    const Iv<F> ux = fx::isub(hc, hs), uy = fx::iadd(hs, hc);
    const Iv<F> vx = fx::isub(fx::imul(nh, e.c), hs), vy = fx::iadd(fx::imul(nh, e.s), hc);
    e.px[0] = fx::iadd(x, ux); e.py[0] = fx::iadd(y, uy);
    e.px[1] = fx::iadd(x, vx); e.py[1] = fx::iadd(y, vy);
    e.px[2] = fx::isub(x, ux); e.py[2] = fx::isub(y, uy);
    e.px[3] = fx::isub(x, vx); e.py[3] = fx::isub(y, vy);
}

// The interval SAT test runs for nearly every undecided pair: its comparisons,
// additions and subtractions are inlined at 7 limbs (fx::kInlineLimbs), the
// products stay out of line.
template <int F>
__device__ __forceinline__ Fix<F> fmin_(const Fix<F>& a, const Fix<F>& b) { return fx::cmp<F, true>(a, b) < 0 ? a : b; }
template <int F>
__device__ __forceinline__ Fix<F> fmax_(const Fix<F>& a, const Fix<F>& b) { return fx::cmp<F, true>(a, b) > 0 ? a : b; }

// sat_check_interval_cached (certifier.cpp:638-703)
template <int F>
__device__ __noinline__ int iv_sat(const IvSq<F>& p, const IvSq<F>& q) {
    Fix<F> z;
    fx::set_zero(z);
    if (p.flat && q.flat) {
        const Iv<F> ox = fx::isub<F, true>(Iv<F>{fmin_(p.x1.lo, q.x1.lo), fmin_(p.x1.hi, q.x1.hi)},
                                  Iv<F>{fmax_(p.x0.lo, q.x0.lo), fmax_(p.x0.hi, q.x0.hi)});
        if (fx::cmp<F, true>(ox.hi, z) <= 0) return 1;
        const Iv<F> oy = fx::isub<F, true>(Iv<F>{fmin_(p.y1.lo, q.y1.lo), fmin_(p.y1.hi, q.y1.hi)},
                                  Iv<F>{fmax_(p.y0.lo, q.y0.lo), fmax_(p.y0.hi, q.y0.hi)});
        if (fx::cmp<F, true>(oy.hi, z) <= 0) return 1;
        if (fx::cmp<F, true>(ox.lo, z) <= 0 || fx::cmp<F, true>(oy.lo, z) <= 0) return 0;
        return -1;
    }
    bool open = false;
    for (int a = 0; a < 4; ++a) {
        const IvSq<F>& o = a < 2 ? p : q;
        const Iv<F> ax = (a & 1) ? fx::ineg(o.s) : o.c;
        const Iv<F>& ay = (a & 1) ? o.c : o.s;
        Iv<F> mn1, mx1, mn2, mx2;
        for (int k = 0; k < 4; ++k) {
            const Iv<F> u = fx::iadd<F, true>(fx::imul(ax, p.px[k]), fx::imul(ay, p.py[k]));
            const Iv<F> v = fx::iadd<F, true>(fx::imul(ax, q.px[k]), fx::imul(ay, q.py[k]));
            if (k == 0) {
                mn1 = mx1 = u;
                mn2 = mx2 = v;
                continue;
            }
            mn1.lo = fmin_(u.lo, mn1.lo); mn1.hi = fmin_(u.hi, mn1.hi);
            mx1.lo = fmax_(u.lo, mx1.lo); mx1.hi = fmax_(u.hi, mx1.hi);
            mn2.lo = fmin_(v.lo, mn2.lo); mn2.hi = fmin_(v.hi, mn2.hi);
            mx2.lo = fmax_(v.lo, mx2.lo); mx2.hi = fmax_(v.hi, mx2.hi);
        }
        const Iv<F> ov = fx::isub<F, true>(Iv<F>{fmin_(mx1.lo, mx2.lo), fmin_(mx1.hi, mx2.hi)},
                                  Iv<F>{fmax_(mn1.lo, mn2.lo), fmax_(mn1.hi, mn2.hi)});
        if (fx::cmp<F, true>(ov.hi, z) <= 0) return 1;
        if (fx::cmp<F, true>(ov.lo, z) <= 0) open = true;
    }
    return open ? 0 : -1;
}

template <int F>
__global__ void __launch_bounds__(128) cert_stage_kernel(
    const Pair* __restrict__ in, const uint32_t* __restrict__ in_count, uint32_t in_cap,
    Pair* __restrict__ next, uint32_t* __restrict__ next_count, uint32_t next_cap,
    const int64_t* __restrict__ pk_sq0, const Lit* __restrict__ lits, const char* __restrict__ text,
    PkOut* __restrict__ out) {
    const uint32_t total = min(*in_count, in_cap);
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const Pair pr = in[t];
        PkOut& po = out[pr.pk];
        if (po.fkey != kNoPair || (po.flags & kCertOverlap)) continue;
        const int64_t s0 = pk_sq0[pr.pk];
        const Iv<F> ox = fx::parse_iv<F>(text, lits[3 * s0]);
        const Iv<F> oy = fx::parse_iv<F>(text, lits[3 * s0 + 1]);
        IvSq<F> A, Bq;
        make_ivsq<F>(text, lits + 3 * (s0 + pr.u), ox, oy, A);
        make_ivsq<F>(text, lits + 3 * (s0 + pr.v), ox, oy, Bq);
        const int r = iv_sat<F>(A, Bq);
        if (r < 0) {
            atomicOr(&po.flags, kCertOverlap);
        } else if (r == 0) {
            if (next == nullptr) {
                atomicOr(&po.flags, kUndecidable);
            } else {
                const uint32_t slot = atomicAdd(next_count, 1u);
                if (slot < next_cap) next[slot] = pr;
                else atomicOr(&po.flags, kPairOverflow);
            }
        }
    }
}

// ------------------------------------------------------------ cached stages
// The same interval test with every square's interval corners computed once
// per stage, as the reference caches them per square (ensure_sq_iv,
// certifier.cpp:600-635): a square sits in about four undecided pairs of a
// contact-heavy packing, and its parse + Taylor sin/cos is the expensive part.
//   mark   claims a cache slot for each square of a live pair (one claim per
//          square: slot_of[] holds -1, then -2 while claimed, then the slot);
//   build  one thread per claimed square writes its IvSq<F> to the cache in
//          HBM;
//   pair   one thread per pair runs iv_sat on references into the cache.
// Flags only ever get set, so a pair the mark kernel skipped (its packing
// already decided) is skipped by the pair kernel too.
struct SqRef {
    int32_t sq;  // global square index (packing's first square + id)
    int32_t pk;
};

__device__ __forceinline__ bool pair_live(const PkOut& po) {
    return po.fkey == kNoPair && !(po.flags & kCertOverlap);
}

__global__ void __launch_bounds__(256) cert_mark_kernel(const Pair* __restrict__ in, const uint32_t* __restrict__ in_count,
                                                       uint32_t in_cap, const int64_t* __restrict__ pk_sq0,
                                                       int32_t* __restrict__ slot_of, SqRef* __restrict__ list,
                                                       uint32_t* __restrict__ list_count, uint32_t list_cap,
                                                       PkOut* __restrict__ out) {
    const uint32_t total = min(*in_count, in_cap);
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const Pair pr = in[t];
        if (!pair_live(out[pr.pk])) continue;
        const int64_t s0 = pk_sq0[pr.pk];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int32_t g = (int32_t)(s0 + (k ? pr.v : pr.u));
            if (atomicCAS(&slot_of[g], -1, -2) == -1) {
                const uint32_t slot = atomicAdd(list_count, 1u);
                if (slot < list_cap) {
                    list[slot] = SqRef{g, pr.pk};
                    slot_of[g] = (int32_t)slot;
                } else {
                    atomicOr(&out[pr.pk].flags, kPairOverflow);
                }
            }
        }
    }
}

template <int F>
__global__ void __launch_bounds__(128) cert_build_kernel(const SqRef* __restrict__ list,
                                                        const uint32_t* __restrict__ list_count, uint32_t list_cap,
                                                        const int64_t* __restrict__ pk_sq0,
                                                        const Lit* __restrict__ lits, const char* __restrict__ text,
                                                        IvSq<F>* __restrict__ cache) {
    const uint32_t total = min(*list_count, list_cap);
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const SqRef r = list[t];
        const int64_t s0 = pk_sq0[r.pk];
        const Iv<F> ox = fx::parse_iv<F>(text, lits[3 * s0]);
        const Iv<F> oy = fx::parse_iv<F>(text, lits[3 * s0 + 1]);
        make_ivsq<F>(text, lits + 3 * (int64_t)r.sq, ox, oy, cache[t]);
    }
}

template <int F>
__global__ void __launch_bounds__(128) cert_pair_kernel(const Pair* __restrict__ in,
                                                       const uint32_t* __restrict__ in_count, uint32_t in_cap,
                                                       Pair* __restrict__ next, uint32_t* __restrict__ next_count,
                                                       uint32_t next_cap, const int64_t* __restrict__ pk_sq0,
                                                       const int32_t* __restrict__ slot_of,
                                                       const IvSq<F>* __restrict__ cache, PkOut* __restrict__ out) {
    const uint32_t total = min(*in_count, in_cap);
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const Pair pr = in[t];
        PkOut& po = out[pr.pk];
        if (!pair_live(po)) continue;
        const int64_t s0 = pk_sq0[pr.pk];
        const int32_t a = slot_of[s0 + pr.u], b = slot_of[s0 + pr.v];
        if (a < 0 || b < 0) {  // no cache entry (the slot list overflowed): report, never guess
            atomicOr(&po.flags, kPairOverflow);
            continue;
        }
        const int r = iv_sat<F>(cache[a], cache[b]);
        if (r < 0) {
            atomicOr(&po.flags, kCertOverlap);
        } else if (r == 0) {
            if (next == nullptr) {
                atomicOr(&po.flags, kUndecidable);
            } else {
                const uint32_t slot = atomicAdd(next_count, 1u);
                if (slot < next_cap) next[slot] = pr;
                else atomicOr(&po.flags, kPairOverflow);
            }
        }
    }
}

// ------------------------------------------------------------ host side
// Constants (600-digit pi/2, 2 pi) are analysed without the 100-character
// literal limit that applies to submitted coordinates.
static int host_lit(const char* s, Lit& L) {
    if (!analyze(s, (int)std::strlen(s), 0, L, 1 << 20)) {
        set_error("internal: constant literal does not parse");
        return SQS_EINVAL;
    }
    L.dyadic = dyadic(s, L);
    return SQS_OK;
}

// Literal texts of this size range are staged in pinned memory for the
// upload (larger ones are uploaded from the caller's memory, rather than
// pinning gigabytes of host memory).
constexpr size_t kPinnedTextMin = (size_t)4 << 20;
constexpr size_t kPinnedTextMax = (size_t)1 << 30;

static int upload_consts(int device) {
    static std::atomic<bool> done[64];
    static std::mutex mu;  // several host threads may certify at once
    if (done[device & 63]) return SQS_OK;
    std::lock_guard<std::mutex> lk(mu);
    if (done[device & 63]) return SQS_OK;
    Consts c;
    Lit hp, tp, h;
    if (int r = host_lit(kHalfPi, hp)) return r;
    if (int r = host_lit(kTwoPi, tp)) return r;
    if (int r = host_lit("0.5", h)) return r;
    c.half_pi9 = fx::parse<9>(kHalfPi, hp, 0);
    c.two_pi9 = fx::parse<9>(kTwoPi, tp, 0);
    c.half9 = fx::parse<9>("0.5", h, 0);
    c.half_pi7 = fx::parse_iv<7>(kHalfPi, hp);
    c.half7 = fx::parse_iv<7>("0.5", h);
    c.half_pi15 = fx::parse_iv<15>(kHalfPi, hp);
    c.half15 = fx::parse_iv<15>("0.5", h);
    c.half_pi58 = fx::parse_iv<58>(kHalfPi, hp);
    c.half58 = fx::parse_iv<58>("0.5", h);
    SQS_CUDA(cudaMemcpyToSymbol(c_consts, &c, sizeof c));
    done[device & 63] = true;
    return SQS_OK;
}

// The side rounded half-to-even at 50 decimals (format_50_decimals,
// certifier.cpp:60-104), written into dst (cap >= 80 holds every side here).
static void fifty_into(const Fix<9>& v, char* dst, size_t cap) {
    const uint64_t B = 1000000000ULL;
    uint64_t low = v.d[6] % 10000ULL, top = v.d[6] / 10000ULL;
    const bool tail = v.d[7] || v.d[8] || v.d[9];
    const bool up = low > 5000ULL || (low == 5000ULL && (tail || (top & 1ULL)));
    uint64_t o[7] = {v.d[0], v.d[1], v.d[2], v.d[3], v.d[4], v.d[5], top};
    if (up && ++o[6] >= 100000ULL) {
        o[6] -= 100000ULL;
        int i = 5;
        for (; i >= 1; --i) {
            if (++o[i] < B) break;
            o[i] -= B;
        }
        if (i < 1) o[0] += 1;
    }
    bool allz = true;
    for (uint64_t w : o) allz &= w == 0;
    char buf[96];
    char* c = buf;
    if (v.neg && !allz) *c++ = '-';
    c = std::to_chars(c, c + 20, o[0]).ptr;
    *c++ = '.';
    for (int i = 1; i <= 6; ++i) {  // 9 digits a limb, the last 5
        const int nd = i == 6 ? 5 : 9;
        uint64_t w = o[i];
        for (int k = nd - 1; k >= 0; --k, w /= 10) c[k] = (char)('0' + w % 10);
        c += nd;
    }
    *c = 0;
    std::snprintf(dst, cap, "%s", buf);
}

static double grid_score(int n) { return std::ceil(std::sqrt((double)n)) / std::sqrt((double)n) - 1.0; }

// The pandas float round trip of one value (roundtrip_float_str,
// certifier.cpp:914-929): the shortest of %.15g, %.16g, %.17g that reads back
// as v, with ".0" appended to a plain integer; returns its length (< 40).
static size_t roundtrip_into(double v, char out[40]) {
    for (int p = 15; p <= 17; ++p) {
        if (std::isfinite(v)) {  // to_chars and from_chars are printf and strtod in the C locale, several times faster
            char* e = std::to_chars(out, out + 39, v, std::chars_format::general, p).ptr;
            *e = 0;
            double back = 0.0;
            std::from_chars(out, e, back);
            if (back == v) break;
        } else {
            std::snprintf(out, 40, "%.*g", p, v);
            if (std::strtod(out, nullptr) == v) break;
        }
    }
    size_t len = std::strlen(out);
    if (std::strpbrk(out, ".eE") == nullptr) {
        std::memcpy(out + len, ".0", 3);
        len += 2;
    }
    return len;
}

static std::string roundtrip(const char* s, size_t len) {
    std::string in(s, len);
    char buf[40];
    const size_t k = roundtrip_into(std::strtod(in.c_str(), nullptr), buf);
    return std::string(buf, k);
}

static void put(char* dst, size_t cap, const std::string& s) {
    size_t k = std::min(cap - 1, s.size());
    std::memcpy(dst, s.data(), k);
    dst[k] = 0;
}

// FSq, AABB, sort key, PairSq and sort index of NMAX squares.
constexpr size_t packing_smem(int nmax) { return (size_t)nmax * (sizeof(FSq) + 7 * sizeof(double) + 4 + 3 * 2 + 1); }

template <int T, int NMAX>
static int launch_packing(sqs_ctx* ctx, cudaStream_t st, int count, const int32_t* bucket, const int32_t* pk_n,
                          const int64_t* pk_sq0, const char* text, const SqText* raw, Lit* lits, PkOut* out, Pair* pairs, uint32_t* pair_count,
                          uint32_t cap) {
    if (count == 0) return SQS_OK;
    const size_t smem = packing_smem(NMAX);
    static std::atomic<bool> attr[64];  // set-up once per device (idempotent if repeated)
    if (!attr[ctx->device & 63]) {
        SQS_CUDA(cudaFuncSetAttribute(cert_packing_kernel<T, NMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        attr[ctx->device & 63] = true;
    }
    cert_packing_kernel<T, NMAX><<<count, T, smem, st>>>(count, bucket, pk_n, pk_sq0, text, raw, lits, out, pairs,
                                                          pair_count, cap);
    SQS_CUDA(cudaGetLastError());
    ctx->launches += 1;
    return SQS_OK;
}

// The packings of the three size classes, side by side on the context's
// streams, the largest first: one after another each class left the GPU
// part empty at its end (1,500 packings: 1.95 ms of kernels in a row,
// 1.2 ms side by side).
static int launch_buckets(sqs_ctx* ctx, int c0, int c1, int c2, const int32_t* b0, const int32_t* b1,
                          const int32_t* b2, const int32_t* pk_n, const int64_t* pk_sq0, const char* text,
                          const SqText* raw, Lit* lits, PkOut* out, Pair* pairs, uint32_t* pair_count, uint32_t cap) {
    const int classes = (c0 > 0) + (c1 > 0) + (c2 > 0);
    cudaStream_t s0 = ctx->stream, s1 = ctx->stream;
    if (classes > 1) {
        SQS_CUDA(cudaEventRecord(ctx->fork, ctx->stream));
        s0 = ctx->aux[0];
        s1 = ctx->aux[1];
        for (int a = 0; a < 2; ++a) SQS_CUDA(cudaStreamWaitEvent(ctx->aux[a], ctx->fork, 0));
    }
    int rc = launch_packing<256, 1024>(ctx, ctx->stream, c2, b2, pk_n, pk_sq0, text, raw, lits, out, pairs,
                                       pair_count, cap);
    if (!rc)
        rc = launch_packing<128, 256>(ctx, s1, c1, b1, pk_n, pk_sq0, text, raw, lits, out, pairs, pair_count, cap);
    if (!rc)
        rc = launch_packing<64, 64>(ctx, s0, c0, b0, pk_n, pk_sq0, text, raw, lits, out, pairs, pair_count, cap);
    if (classes > 1) {  // join the side streams, also after a failed launch
        for (int a = 0; a < 2; ++a) {
            SQS_CUDA(cudaEventRecord(ctx->join[a], ctx->aux[a]));
            SQS_CUDA(cudaStreamWaitEvent(ctx->stream, ctx->join[a], 0));
        }
    }
    return rc;
}

template <int F>
static int launch_stage(sqs_ctx* ctx, const Pair* in, const uint32_t* in_count, uint32_t in_cap, Pair* next,
                        uint32_t* next_count, uint32_t next_cap, const int64_t* pk_sq0, const Lit* lits,
                        const char* text, PkOut* out, int blocks) {
    cert_stage_kernel<F><<<blocks, 128, 0, ctx->stream>>>(in, in_count, in_cap, next, next_count, next_cap,
                                                         pk_sq0, lits, text, out);
    SQS_CUDA(cudaGetLastError());
    ctx->launches += 1;
    return SQS_OK;
}

static unsigned grid_for(sqs_ctx* ctx, uint32_t items, unsigned threads) {
    const uint64_t want = ((uint64_t)items + threads - 1) / threads;
    const uint64_t cap = (uint64_t)ctx->sm_count * 8;
    return (unsigned)std::max<uint64_t>(1, std::min(want, cap));
}

// One escalation stage with the per-square cache.  Reads back the stage's
// pair count (a stage without pairs launches nothing) and the number of
// claimed squares (the cache is sized to exactly those).
template <int F>
static int cached_stage(sqs_ctx* ctx, const Pair* in, const uint32_t* in_count, uint32_t cap, Pair* next,
                        uint32_t* next_count, const int64_t* d_s0, const Lit* d_lits, const char* d_text,
                        PkOut* d_out, int32_t* slot_of, SqRef* list, uint32_t* list_count, int64_t S) {
    uint32_t h_in = 0;
    SQS_CUDA(cudaMemcpyAsync(&h_in, in_count, 4, cudaMemcpyDeviceToHost, ctx->stream));
    SQS_CUDA(cudaStreamSynchronize(ctx->stream));
    h_in = std::min(h_in, cap);
    if (h_in == 0) return SQS_OK;
    const uint32_t list_cap = (uint32_t)std::min<int64_t>(S, 2ll * h_in);
    SQS_CUDA(cudaMemsetAsync(slot_of, 0xff, (size_t)S * sizeof(int32_t), ctx->stream));
    SQS_CUDA(cudaMemsetAsync(list_count, 0, sizeof(uint32_t), ctx->stream));
    cert_mark_kernel<<<grid_for(ctx, h_in, 256), 256, 0, ctx->stream>>>(in, in_count, cap, d_s0, slot_of, list,
                                                                         list_count, list_cap, d_out);
    SQS_CUDA(cudaGetLastError());
    ctx->launches += 1;
    uint32_t h_sq = 0;
    SQS_CUDA(cudaMemcpyAsync(&h_sq, list_count, 4, cudaMemcpyDeviceToHost, ctx->stream));
    SQS_CUDA(cudaStreamSynchronize(ctx->stream));
    h_sq = std::min(h_sq, list_cap);
    IvSq<F>* cache = nullptr;
    if (h_sq > 0) {
        if (int r = ctx->d_cert.reserve((size_t)h_sq * sizeof(IvSq<F>))) return r;
        cache = (IvSq<F>*)ctx->d_cert.p;
        cert_build_kernel<F><<<grid_for(ctx, h_sq, 128), 128, 0, ctx->stream>>>(list, list_count, list_cap, d_s0,
                                                                                 d_lits, d_text, cache);
        SQS_CUDA(cudaGetLastError());
        ctx->launches += 1;
    }
    cert_pair_kernel<F><<<grid_for(ctx, h_in, 128), 128, 0, ctx->stream>>>(
        in, in_count, cap, next, next_count, next ? cap : 0, d_s0, slot_of, cache, d_out);
    SQS_CUDA(cudaGetLastError());
    ctx->launches += 1;
    return SQS_OK;
}

}  // namespace cert
}  // namespace sqs

using namespace sqs;
using namespace sqs::cert;

extern "C" int sqs_certify_batch(sqs_ctx* ctx, int count, const int32_t* n_of, const int64_t* row_start,
                                 const int32_t* square_id, const char* text, const int64_t* lit_off, int flags,
                                 sqs_verdict* out) {
    if (int r = enter(ctx)) return r;
    SQS_REQUIRE(count >= 0, "count %d < 0", count);
    if (count == 0) return SQS_OK;
    SQS_REQUIRE(n_of && row_start && text && lit_off && out, "null host pointer");
    if (int r = upload_consts(ctx->device)) return r;

    // 1. the envelope of every packing (serial, cheap): verdict defaults, row
    //    counts, and the square offsets of those that may certify
    std::vector<int32_t> pk_n((size_t)count, 0);
    std::vector<int64_t> pk_sq0((size_t)count, 0);
    std::vector<char> live((size_t)count, 0);
    const bool do_rt = (flags & SQS_CERT_ROUNDTRIP) != 0;
    int64_t S = 0;
    for (int p = 0; p < count; ++p) {
        const int n = n_of[p];
        sqs_verdict& v = out[p];
        std::memset(&v, 0, sizeof v);
        v.n = n;
        SQS_REQUIRE(n >= 1 && n <= kMaxN, "packing %d: n=%d out of 1..%d", p, n, kMaxN);
        v.score = grid_score(n);
        const int64_t r0 = row_start[p], r1 = row_start[p + 1];
        SQS_REQUIRE(r1 >= r0, "packing %d: row_start not monotone", p);
        if (r1 - r0 != n) {
            const std::string N = std::to_string(n);
            put(v.reason, sizeof v.reason, "n=" + N + ": expected " + N + " rows, got " + std::to_string(r1 - r0));
            continue;
        }
        live[(size_t)p] = 1;
        pk_n[(size_t)p] = n;
        pk_sq0[(size_t)p] = S;
        S += n;
    }
    SQS_REQUIRE(S < (1ll << 30), "%lld squares in one call (limit 2^30)", (long long)S);
    // 2. square ids and literal slices (round-tripped when asked), host
    //    threads over contiguous ranges of packings with equal square counts
    // Literal slice tables, written straight into the context's pinned
    // staging: no zero fill, no page faults after the first call, and an
    // upload at the full host-link rate.  Every slot of a live packing is
    // written below; slots of packings found invalid are never read.
    // One 16-byte record a square (its three literals lie back to back).
    if (int r = ctx->h_cert.reserve((size_t)S * sizeof(SqText) + 16)) return r;
    SqText* const raw = (SqText*)ctx->h_cert.p;
    const int nt = count >= 64 ? (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency())) : 1;
    std::vector<int> p_lo((size_t)nt + 1, count);
    {
        int t = 0;
        p_lo[0] = 0;
        for (int p = 0; p < count && t + 1 < nt; ++p)
            if (pk_sq0[(size_t)p] >= (S * (t + 1)) / nt) p_lo[(size_t)++t] = p;
        for (++t; t <= nt; ++t) p_lo[(size_t)t] = count;
    }
    std::vector<std::string> rt((size_t)nt);  // round-tripped text of each thread's packings
    std::vector<int64_t> bad_row((size_t)nt, -1), far_row((size_t)nt, -1);
    // A large literal text is staged in pinned memory too, each thread copying
    // the span of its own packings (the first from offset 0), so that it
    // uploads at the full host-link rate.
    SQS_REQUIRE(lit_off[3 * row_start[count]] >= 0, "literal offsets end below 0");
    const size_t text_bytes = (size_t)lit_off[3 * row_start[count]];
    char* h_text = nullptr;
    if (!do_rt && text_bytes >= kPinnedTextMin && text_bytes <= kPinnedTextMax) {
        if (int r = ctx->h_text.reserve(text_bytes)) return r;
        h_text = (char*)ctx->h_text.p;
    }
    auto slice = [&](int t) {
        if (h_text) {
            const int64_t a = t == 0 ? 0 : lit_off[3 * row_start[p_lo[(size_t)t]]];
            const int64_t b = t + 1 == nt ? (int64_t)text_bytes : lit_off[3 * row_start[p_lo[(size_t)t + 1]]];
            if (b > a && a >= 0 && (size_t)b <= text_bytes) std::memcpy(h_text + a, text + a, (size_t)(b - a));
        }
        std::vector<int64_t> row_of;
        for (int p = p_lo[(size_t)t]; p < p_lo[(size_t)t + 1]; ++p) {
            if (!live[(size_t)p]) continue;
            const int n = pk_n[(size_t)p];
            const int64_t r0 = row_start[p];
            row_of.assign((size_t)n, -1);
            bool bad = false;
            for (int64_t r = r0; r < r0 + n && !bad; ++r) {
                const int sid = square_id ? square_id[r] : (int)(r - r0);
                if (sid < 0 || sid >= n || row_of[(size_t)sid] >= 0) bad = true;
                else row_of[(size_t)sid] = r;
            }
            if (bad) {
                live[(size_t)p] = 0;
                put(out[p].reason, sizeof out[p].reason,
                    "n=" + std::to_string(n) + ": square_ids should be 0.." + std::to_string(n - 1));
                continue;
            }
            for (int i = 0; i < n; ++i) {
                const int64_t r = row_of[(size_t)i];
                SqText& q = raw[pk_sq0[(size_t)p] + i];
                q.off = (uint32_t)(do_rt ? (int64_t)rt[(size_t)t].size() : lit_off[3 * r]);
                if (!do_rt && lit_off[3 * r + 2] > kOffMax) far_row[(size_t)t] = r;
                for (int k = 0; k < 3; ++k) {
                    const int64_t a = lit_off[3 * r + k], b = lit_off[3 * r + k + 1];
                    if (a < 0 || b < a || (size_t)b > text_bytes) {
                        bad_row[(size_t)t] = r;
                        return;
                    }
                    if (do_rt) {
                        const std::string s2 = roundtrip(text + a, (size_t)(b - a));
                        q.len[k] = (uint32_t)s2.size();
                        rt[(size_t)t] += s2;
                    } else {
                        q.len[k] = (uint32_t)std::min<int64_t>(b - a, UINT32_MAX);
                    }
                }
            }
        }
    };
    if (nt == 1) {
        slice(0);
    } else {
        std::vector<std::thread> pool;
        for (int t = 0; t < nt; ++t) pool.emplace_back(slice, t);
        for (auto& th : pool) th.join();
    }
    for (int t = 0; t < nt; ++t)
        SQS_REQUIRE(bad_row[(size_t)t] < 0, "literal offsets not monotone, or outside the text, at row %lld",
                    (long long)bad_row[(size_t)t]);
    for (int t = 0; t < nt; ++t)
        SQS_REQUIRE(far_row[(size_t)t] < 0, "literals of row %lld lie past 4 GiB of text (split the call)",
                    (long long)far_row[(size_t)t]);
    std::string rt_text;  // round-tripped literals, when requested
    if (do_rt) {
        size_t base = 0, rt_bytes = 0;
        for (const std::string& part : rt) rt_bytes += part.size();
        SQS_REQUIRE((int64_t)rt_bytes <= kOffMax, "round-tripped literals past 4 GiB of text (split the call)");
        for (int t = 0; t < nt; ++t) {
            if (base)
                for (int p = p_lo[(size_t)t]; p < p_lo[(size_t)t + 1]; ++p) {
                    if (!live[(size_t)p]) continue;
                    for (int64_t q = pk_sq0[(size_t)p]; q < pk_sq0[(size_t)p] + pk_n[(size_t)p]; ++q)
                        raw[q].off += (uint32_t)base;
                }
            base += rt[(size_t)t].size();
        }
        rt_text.reserve(base);
        for (int t = 0; t < nt; ++t) rt_text += rt[(size_t)t];
    }
    const char* blob = do_rt ? rt_text.data() : (h_text ? h_text : text);
    size_t blob_bytes = do_rt ? rt_text.size() : (size_t)lit_off[3 * row_start[count]];
    if (blob_bytes == 0) blob_bytes = 1;
    // buckets by n
    std::vector<int32_t> bk[3];
    for (int p = 0; p < count; ++p) {
        if (!live[(size_t)p]) continue;
        const int n = pk_n[(size_t)p];
        bk[n <= 64 ? 0 : (n <= 256 ? 1 : 2)].push_back(p);
    }
    const uint32_t cap = (uint32_t)std::min<int64_t>(16 * S + 4096, 1ll << 31);
    // device buffers (one staging allocation per call; reused when large enough)
    struct Seg { size_t off, bytes; };
    size_t tot = 0;
    auto seg = [&](size_t bytes) { Seg s{tot, bytes}; tot += (bytes + 255) & ~(size_t)255; return s; };
    const Seg g_text = seg(blob_bytes), g_raw = seg((size_t)S * sizeof(SqText) + 16);
    const Seg g_n = seg((size_t)count * 4), g_s0 = seg((size_t)count * 8);
    const Seg g_b0 = seg(bk[0].size() * 4 + 4), g_b1 = seg(bk[1].size() * 4 + 4), g_b2 = seg(bk[2].size() * 4 + 4);
    const Seg g_lits = seg((size_t)(3 * S + 3) * sizeof(Lit)), g_out = seg((size_t)count * sizeof(PkOut));
    const Seg g_pa = seg((size_t)cap * sizeof(Pair)), g_pb = seg((size_t)cap * sizeof(Pair)), g_cnt = seg(64);
    const Seg g_slot = seg((size_t)S * sizeof(int32_t) + 4), g_list = seg((size_t)S * sizeof(SqRef) + 8);
    if (int r = ctx->d_misc.reserve(tot)) return r;
    char* D = (char*)ctx->d_misc.p;
    auto up = [&](const Seg& s, const void* h, size_t bytes) -> int {
        if (bytes) SQS_CUDA(cudaMemcpyAsync(D + s.off, h, bytes, cudaMemcpyHostToDevice, ctx->stream));
        return SQS_OK;
    };
    if (int r = up(g_text, blob, do_rt ? rt_text.size() : (size_t)lit_off[3 * row_start[count]])) return r;
    if (int r = up(g_raw, raw, (size_t)S * sizeof(SqText))) return r;
    if (int r = up(g_n, pk_n.data(), (size_t)count * 4)) return r;
    if (int r = up(g_s0, pk_sq0.data(), (size_t)count * 8)) return r;
    if (int r = up(g_b0, bk[0].data(), bk[0].size() * 4)) return r;
    if (int r = up(g_b1, bk[1].data(), bk[1].size() * 4)) return r;
    if (int r = up(g_b2, bk[2].data(), bk[2].size() * 4)) return r;
    SQS_CUDA(cudaMemsetAsync(D + g_out.off, 0, g_out.bytes, ctx->stream));
    SQS_CUDA(cudaMemsetAsync(D + g_cnt.off, 0, 64, ctx->stream));
    PkOut* d_out = (PkOut*)(D + g_out.off);
    Pair* pa = (Pair*)(D + g_pa.off);
    Pair* pb = (Pair*)(D + g_pb.off);
    uint32_t* cnt = (uint32_t*)(D + g_cnt.off);
    const char* d_text = D + g_text.off;
    const SqText* d_raw = (const SqText*)(D + g_raw.off);
    const int32_t* d_n = (const int32_t*)(D + g_n.off);
    const int64_t* d_s0 = (const int64_t*)(D + g_s0.off);
    Lit* d_lits = (Lit*)(D + g_lits.off);
    if (int r = launch_buckets(ctx, (int)bk[0].size(), (int)bk[1].size(), (int)bk[2].size(),
                               (const int32_t*)(D + g_b0.off), (const int32_t*)(D + g_b1.off),
                               (const int32_t*)(D + g_b2.off), d_n, d_s0, d_text, d_raw, d_lits, d_out, pa, cnt, cap))
        return r;
    int32_t* slot_of = (int32_t*)(D + g_slot.off);
    SqRef* list = (SqRef*)(D + g_list.off);
    // the records and the number of open pairs; most batches have none left
    std::vector<PkOut> h((size_t)count);
    uint32_t open = 0;
    auto read_back = [&](uint32_t* c) -> int {
        SQS_CUDA(cudaMemcpyAsync(h.data(), d_out, (size_t)count * sizeof(PkOut), cudaMemcpyDeviceToHost, ctx->stream));
        if (c) SQS_CUDA(cudaMemcpyAsync(&open, c, 4, cudaMemcpyDeviceToHost, ctx->stream));
        SQS_CUDA(cudaStreamSynchronize(ctx->stream));
        return SQS_OK;
    };
    if (int r = read_back(cnt)) return r;
    if (open) {  // the 7-, 15- and 58-limb stages pa -> pb -> pa
        if (int r = cached_stage<7>(ctx, pa, cnt, cap, pb, cnt + 1, d_s0, d_lits, d_text, d_out, slot_of, list, cnt + 3, S))
            return r;
        if (int r = cached_stage<15>(ctx, pb, cnt + 1, cap, pa, cnt + 2, d_s0, d_lits, d_text, d_out, slot_of, list,
                                     cnt + 3, S))
            return r;
        if (int r = cached_stage<58>(ctx, pa, cnt + 2, cap, nullptr, nullptr, d_s0, d_lits, d_text, d_out, slot_of,
                                     list, cnt + 3, S))
            return r;
        if (int r = read_back(nullptr)) return r;
    }
    for (int p = 0; p < count; ++p) {
        if (!live[(size_t)p]) continue;
        sqs_verdict& v = out[p];
        const PkOut& o = h[(size_t)p];
        const int n = pk_n[(size_t)p];
        if (o.flags & kPairOverflow) {
            set_error("packing %d: undecided-pair list overflowed", p);
            return SQS_ENOMEM;
        }
        if (o.err_key != kNoKey) {
            static const char* what[4] = {"cannot parse coordinates", "value out of range for a double",
                                          "coordinate out of bounds", "angle out of bounds"};
            put(v.reason, sizeof v.reason,
                "n=" + std::to_string(n) + ", square " + std::to_string(o.err_key / 4) + ": " + what[o.err_key % 4]);
            continue;
        }
        if (o.fkey != kNoPair) {
            put(v.reason, sizeof v.reason,
                "infeasible: Squares " + std::to_string(o.fu) + " and " + std::to_string(o.fv) +
                    " overlap (float check)");
            continue;
        }
        if (o.flags & kCertOverlap) {
            put(v.reason, sizeof v.reason, "infeasible: Squares overlap (certified)");
            continue;
        }
        if (o.flags & kUndecidable) {
            put(v.reason, sizeof v.reason, "infeasible: Overlap undecidable at max precision");
            continue;
        }
        const double sf = fx::approx(o.side), lb = std::sqrt((double)n);
        if (sf < lb - 1e-7) {
            put(v.reason, sizeof v.reason, "infeasible: L is below area lower bound");
            continue;
        }
        v.ok = 1;
        put(v.reason, sizeof v.reason, "ok");
        fifty_into(o.side, v.L, sizeof v.L);
        v.score = std::max(0.0, sf / lb - 1.0);
    }
    return SQS_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free certification: the same kernels, with every device buffer
// carved from one file-scope array and every host buffer static.  For callers
// that must not allocate device memory at run time -- a host that owns all
// GPU memory through its own pool, a real-time loop that forbids allocation
// after start-up -- at the price of fixed limits and of a process-wide
// buffer that concurrent calls share.
namespace sqs {
namespace cert {

constexpr int kStaticMaxSquares = 16384;
constexpr int kStaticMaxPackings = 4096;
constexpr size_t kStaticMaxText = 2u << 20;               // literal bytes per call
constexpr uint32_t kStaticPairCap = 16u * kStaticMaxSquares + 4096u;

constexpr size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }
constexpr size_t kSoText = 0;
constexpr size_t kSoOff = kSoText + al256(kStaticMaxText);
constexpr size_t kSoN = kSoOff + al256(sizeof(SqText) * kStaticMaxSquares);
constexpr size_t kSoS0 = kSoN + al256(sizeof(int32_t) * kStaticMaxPackings);
constexpr size_t kSoBk = kSoS0 + al256(sizeof(int64_t) * kStaticMaxPackings);
constexpr size_t kSoLits = kSoBk + al256(sizeof(int32_t) * kStaticMaxPackings);
constexpr size_t kSoOut = kSoLits + al256(sizeof(Lit) * 3 * kStaticMaxSquares);
constexpr size_t kSoPa = kSoOut + al256(sizeof(PkOut) * kStaticMaxPackings);
constexpr size_t kSoPb = kSoPa + al256(sizeof(Pair) * kStaticPairCap);
constexpr size_t kSoCnt = kSoPb + al256(sizeof(Pair) * kStaticPairCap);
constexpr size_t kStaticScratchBytes = kSoCnt + 256;  // about 7.5 MiB

// The scratch every call of sqs_certify_batch_static shares.  In host code
// this name is only a stand-in: the device address comes from
// cudaGetSymbolAddress, taken once per device.
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];
static void* s_scratch_addr[64] = {nullptr};
static std::atomic<bool> s_ready[64];
static std::mutex s_setup_mu;
// Set while a call runs: the scratch and the host staging below are shared
// by every call in the process, so a call that would overlap another is
// refused instead of racing with it.
static std::atomic_flag s_busy = ATOMIC_FLAG_INIT;

// Host staging (static, not heap): literal slices in square-id order, packing
// tables, round-tripped literals, the per-packing records read back.
static SqText s_raw[kStaticMaxSquares];
static int32_t s_pk_n[kStaticMaxPackings];
static int64_t s_pk_sq0[kStaticMaxPackings];
static int32_t s_bucket[kStaticMaxPackings];
static unsigned char s_live[kStaticMaxPackings];
static int64_t s_row_of[kMaxN];
static char s_rt_text[kStaticMaxText];
static char s_lit_tmp[4096];
static PkOut s_out[kStaticMaxPackings];

// Per-device set-up of the allocation-free path, once, with that device
// current: the device address of the static array (cudaGetSymbolAddress;
// under lazy module loading this is also what loads the module holding the
// array), the certifier's constants, and one launch of each stage kernel
// with nothing to do, which loads the kernels and lets the driver size the
// local memory their stacks need.  Everything a later call uses is then in
// place, so later calls allocate nothing.
template <int T, int NMAX>
static int packing_attr() {
    const size_t smem = packing_smem(NMAX);
    SQS_CUDA(cudaFuncSetAttribute(cert_packing_kernel<T, NMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return SQS_OK;
}

static int static_setup(sqs_ctx* ctx) {
    const int dev = ctx->device & 63;
    if (s_ready[dev]) return SQS_OK;
    std::lock_guard<std::mutex> lk(s_setup_mu);
    if (s_ready[dev]) return SQS_OK;
    void* p = nullptr;
    SQS_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
    if (int r = upload_consts(ctx->device)) return r;
    if (int r = packing_attr<64, 64>()) return r;
    if (int r = packing_attr<128, 256>()) return r;
    if (int r = packing_attr<256, 1024>()) return r;
    char* D = (char*)p;
    Pair* pa = (Pair*)(D + kSoPa);
    uint32_t* cnt = (uint32_t*)(D + kSoCnt);
    SQS_CUDA(cudaMemsetAsync(cnt, 0, 64, ctx->stream));
    const int64_t* d_s0 = (const int64_t*)(D + kSoS0);
    const Lit* d_lits = (const Lit*)(D + kSoLits);
    PkOut* d_out = (PkOut*)(D + kSoOut);
    if (int r = launch_stage<7>(ctx, pa, cnt, 0, nullptr, nullptr, 0, d_s0, d_lits, D, d_out, 1)) return r;
    if (int r = launch_stage<15>(ctx, pa, cnt, 0, nullptr, nullptr, 0, d_s0, d_lits, D, d_out, 1)) return r;
    if (int r = launch_stage<58>(ctx, pa, cnt, 0, nullptr, nullptr, 0, d_s0, d_lits, D, d_out, 1)) return r;
    SQS_CUDA(cudaStreamSynchronize(ctx->stream));
    s_scratch_addr[dev] = p;
    s_ready[dev] = true;
    return SQS_OK;
}

namespace {
struct BusyGuard {
    bool held;
    BusyGuard() : held(!s_busy.test_and_set(std::memory_order_acquire)) {}
    ~BusyGuard() {
        if (held) s_busy.clear(std::memory_order_release);
    }
};
}  // namespace

}  // namespace cert
}  // namespace sqs

extern "C" int sqs_certify_batch_static(sqs_ctx* ctx, int count, const int32_t* n_of, const int64_t* row_start,
                                        const int32_t* square_id, const char* text, const int64_t* lit_off,
                                        int flags, sqs_verdict* out) {
    if (int r = enter(ctx)) return r;
    BusyGuard busy;
    if (!busy.held) {
        set_error("sqs_certify_batch_static: another call is in progress (all calls share one static scratch "
                  "array and must not overlap)");
        return SQS_EBUSY;
    }
    SQS_REQUIRE(count >= 0 && count <= kStaticMaxPackings, "count %d out of 0..%d (static certifier limit)", count,
                kStaticMaxPackings);
    // the first call on a device (count == 0 does only this) sets the path up
    if (int r = static_setup(ctx)) return r;
    if (count == 0) return SQS_OK;
    SQS_REQUIRE(n_of && row_start && text && lit_off && out, "null host pointer");
    const int dev = ctx->device & 63;
    const bool do_rt = (flags & SQS_CERT_ROUNDTRIP) != 0;
    // envelope checks and literal slices, as sqs_certify_batch does them
    const int64_t text_end = lit_off[3 * row_start[count]];
    SQS_REQUIRE(text_end >= 0, "literal offsets end below 0");
    SQS_REQUIRE(do_rt || text_end <= (int64_t)kStaticMaxText, "literals exceed %zu bytes (static certifier limit)",
                kStaticMaxText);
    int64_t S = 0;
    size_t rt_used = 0;
    for (int p = 0; p < count; ++p) {
        const int n = n_of[p];
        sqs_verdict& v = out[p];
        std::memset(&v, 0, sizeof v);
        v.n = n;
        s_live[p] = 0;
        SQS_REQUIRE(n >= 1 && n <= kMaxN, "packing %d: n=%d out of 1..%d", p, n, kMaxN);
        v.score = grid_score(n);
        const int64_t r0 = row_start[p], r1 = row_start[p + 1];
        SQS_REQUIRE(r1 >= r0, "packing %d: row_start not monotone", p);
        if (r1 - r0 != n) {
            std::snprintf(v.reason, sizeof v.reason, "n=%d: expected %d rows, got %lld", n, n, (long long)(r1 - r0));
            continue;
        }
        for (int i = 0; i < n; ++i) s_row_of[i] = -1;
        bool bad = false;
        for (int64_t r = r0; r < r1 && !bad; ++r) {
            const int sid = square_id ? square_id[r] : (int)(r - r0);
            if (sid < 0 || sid >= n || s_row_of[sid] >= 0) bad = true;
            else s_row_of[sid] = r;
        }
        if (bad) {
            std::snprintf(v.reason, sizeof v.reason, "n=%d: square_ids should be 0..%d", n, n - 1);
            continue;
        }
        SQS_REQUIRE(S + n <= kStaticMaxSquares, "more than %d squares in one static-certifier call",
                    kStaticMaxSquares);
        s_live[p] = 1;
        s_pk_n[p] = n;
        s_pk_sq0[p] = S;
        for (int i = 0; i < n; ++i) {
            const int64_t r = s_row_of[i];
            SqText& q = s_raw[S + i];
            q.off = (uint32_t)(do_rt ? (int64_t)rt_used : lit_off[3 * r]);
            for (int k = 0; k < 3; ++k) {
                const int64_t a = lit_off[3 * r + k], b = lit_off[3 * r + k + 1];
                SQS_REQUIRE(a >= 0 && b >= a && b <= text_end, "literal offsets not monotone, or outside the text, at row %lld",
                            (long long)r);
                if (do_rt) {
                    SQS_REQUIRE((size_t)(b - a) < sizeof(s_lit_tmp), "literal longer than %zu bytes",
                                sizeof(s_lit_tmp) - 1);
                    std::memcpy(s_lit_tmp, text + a, (size_t)(b - a));
                    s_lit_tmp[b - a] = 0;
                    char buf[40];
                    const size_t len = roundtrip_into(std::strtod(s_lit_tmp, nullptr), buf);
                    SQS_REQUIRE(rt_used + len <= kStaticMaxText, "literals exceed %zu bytes", kStaticMaxText);
                    std::memcpy(s_rt_text + rt_used, buf, len);
                    q.len[k] = (uint32_t)len;
                    rt_used += len;
                } else {
                    q.len[k] = (uint32_t)(b - a);
                }
            }
        }
        S += n;
    }
    const size_t text_bytes = do_rt ? rt_used : (size_t)text_end;
    int nb[3] = {0, 0, 0};
    for (int p = 0; p < count; ++p)
        if (s_live[p]) ++nb[s_pk_n[p] <= 64 ? 0 : (s_pk_n[p] <= 256 ? 1 : 2)];
    int fill[3] = {0, nb[0], nb[0] + nb[1]};
    for (int p = 0; p < count; ++p) {
        if (!s_live[p]) continue;
        const int b = s_pk_n[p] <= 64 ? 0 : (s_pk_n[p] <= 256 ? 1 : 2);
        s_bucket[fill[b]++] = p;
    }
    char* D = (char*)s_scratch_addr[dev];
    cudaStream_t st = ctx->stream;
    if (text_bytes)
        SQS_CUDA(cudaMemcpyAsync(D + kSoText, do_rt ? s_rt_text : text, text_bytes, cudaMemcpyHostToDevice, st));
    SQS_CUDA(cudaMemcpyAsync(D + kSoOff, s_raw, sizeof(SqText) * (size_t)S, cudaMemcpyHostToDevice, st));
    SQS_CUDA(cudaMemcpyAsync(D + kSoN, s_pk_n, sizeof(int32_t) * (size_t)count, cudaMemcpyHostToDevice, st));
    SQS_CUDA(cudaMemcpyAsync(D + kSoS0, s_pk_sq0, sizeof(int64_t) * (size_t)count, cudaMemcpyHostToDevice, st));
    SQS_CUDA(cudaMemcpyAsync(D + kSoBk, s_bucket, sizeof(int32_t) * (size_t)(nb[0] + nb[1] + nb[2]),
                             cudaMemcpyHostToDevice, st));
    // the shared scratch keeps the previous call's contents: clear what starts at zero
    SQS_CUDA(cudaMemsetAsync(D + kSoOut, 0, sizeof(PkOut) * (size_t)count, st));
    SQS_CUDA(cudaMemsetAsync(D + kSoCnt, 0, 64, st));
    const char* d_text = D + kSoText;
    const SqText* d_raw = (const SqText*)(D + kSoOff);
    const int32_t* d_n = (const int32_t*)(D + kSoN);
    const int64_t* d_s0 = (const int64_t*)(D + kSoS0);
    const int32_t* d_bk = (const int32_t*)(D + kSoBk);
    Lit* d_lits = (Lit*)(D + kSoLits);
    PkOut* d_out = (PkOut*)(D + kSoOut);
    Pair* pa = (Pair*)(D + kSoPa);
    Pair* pb = (Pair*)(D + kSoPb);
    uint32_t* cnt = (uint32_t*)(D + kSoCnt);
    const uint32_t cap = kStaticPairCap;
    if (int r = launch_buckets(ctx, nb[0], nb[1], nb[2], d_bk, d_bk + nb[0], d_bk + nb[0] + nb[1], d_n, d_s0, d_text,
                               d_raw, d_lits, d_out, pa, cnt, cap))
        return r;
    const int blocks = ctx->sm_count * 8;
    if (int r = launch_stage<7>(ctx, pa, cnt, cap, pb, cnt + 1, cap, d_s0, d_lits, d_text, d_out, blocks)) return r;
    if (int r = launch_stage<15>(ctx, pb, cnt + 1, cap, pa, cnt + 2, cap, d_s0, d_lits, d_text, d_out, blocks))
        return r;
    if (int r = launch_stage<58>(ctx, pa, cnt + 2, cap, nullptr, nullptr, 0, d_s0, d_lits, d_text, d_out, blocks))
        return r;
    SQS_CUDA(cudaMemcpyAsync(s_out, d_out, sizeof(PkOut) * (size_t)count, cudaMemcpyDeviceToHost, st));
    SQS_CUDA(cudaStreamSynchronize(st));
    static const char* what[4] = {"cannot parse coordinates", "value out of range for a double",
                                  "coordinate out of bounds", "angle out of bounds"};
    for (int p = 0; p < count; ++p) {
        if (!s_live[p]) continue;
        sqs_verdict& v = out[p];
        const PkOut& o = s_out[p];
        const int n = s_pk_n[p];
        if (o.flags & kPairOverflow) {
            set_error("packing %d: undecided-pair list overflowed", p);
            return SQS_ENOMEM;
        }
        if (o.err_key != kNoKey) {
            std::snprintf(v.reason, sizeof v.reason, "n=%d, square %u: %s", n, o.err_key / 4, what[o.err_key % 4]);
            continue;
        }
        if (o.fkey != kNoPair) {
            std::snprintf(v.reason, sizeof v.reason, "infeasible: Squares %d and %d overlap (float check)", o.fu, o.fv);
            continue;
        }
        if (o.flags & kCertOverlap) {
            std::snprintf(v.reason, sizeof v.reason, "infeasible: Squares overlap (certified)");
            continue;
        }
        if (o.flags & kUndecidable) {
            std::snprintf(v.reason, sizeof v.reason, "infeasible: Overlap undecidable at max precision");
            continue;
        }
        const double sf = fx::approx(o.side), lb = std::sqrt((double)n);
        if (sf < lb - 1e-7) {
            std::snprintf(v.reason, sizeof v.reason, "infeasible: L is below area lower bound");
            continue;
        }
        v.ok = 1;
        std::snprintf(v.reason, sizeof v.reason, "ok");
        fifty_into(o.side, v.L, sizeof v.L);
        v.score = std::max(0.0, sf / lb - 1.0);
    }
    return SQS_OK;
}
