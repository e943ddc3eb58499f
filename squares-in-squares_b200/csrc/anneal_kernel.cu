// Batched parallel-tempering simulated annealing of unit squares in a
// shrinking square container: one thread-block cluster per job, one warp per
// replica, every replica's squares and cell list in shared memory.
//
// Reference semantics it re-designs (cuda/seeded.cu): the energy model
// (pair_cached/boundary/total_cached :41-162), single-square Metropolis
// moves (:501-546), replica exchange within a temperature ladder
// (swap_replicas :791-817), the FP64 dilation-certified side of a candidate
// best state (device_certified_side :175-226) and the host's shrink of the
// container after every improvement (:919-938).  What is new:
//   * FP32 moves and energies, with dE of a single-square move taken over the
//     3x3 cell neighbourhood (O(1) per proposal instead of O(n));
//   * lanes of the replica's warp split the neighbour candidates, a butterfly
//     reduction leaves the same dE on every lane, so every lane takes the same
//     Metropolis decision without a broadcast;
//   * counter-based Philox keyed by (job seed, replica, proposal index): a
//     job's trajectory does not depend on the batch, slot or CTA running it;
//   * replica exchange swaps rungs (temperature indices), not states, and the
//     whole ladder (up to 64 rungs) may span a cluster of CTAs, exchanged over
//     distributed shared memory;
//   * the shrink decision is taken on the device at every exchange point
//     (no per-epoch device-to-host round trip).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <tuple>
#include <mutex>
#include <map>

#include <cmath>

#include "anneal.cuh"
#include "common.cuh"
#include "philox.cuh"
#include "sat_pair.cuh"

namespace cg = cooperative_groups;

namespace sqs {
namespace ann {

constexpr float kHalfPiF = 1.57079632679489662f;

// cos/sin of a replica's angle, wherever the state's trig is (re)computed:
// CUDA's full-accuracy sincosf, the same function everywhere so a state's
// (cos, sin) never depends on where it was computed (a sliced run reloads what
// an unsliced one kept).  Against the hardware approximation it costs about 3%
// of the proposal rate and cuts the FP32 energies' absolute error against the
// FP64 oracle about eightfold (measured on the batched and served samples), to
// well inside the 1e-5 floor.  The FP64 certified side recomputes trig from
// the angle itself.
__device__ __forceinline__ void state_trig(float a, float* s, float* c) { sincosf(a, s, c); }

// An angle into [0, pi/2), in one rounding wherever it is compiled in.
__device__ __forceinline__ float wrap_quarter_f(float a) {
    a = __fmaf_rn(-kHalfPiF, floorf(__fmul_rn(a, 1.0f / kHalfPiF)), a);
    return (a >= 0.f && a < kHalfPiF) ? a : 0.f;
}

struct Rep {  // one replica's shared-memory view
    float4* sq;        // (x, y, cos a, sin a)
    float* ang;        // a in [0, pi/2)
    uint8_t* cnt;      // squares per cell
    uint16_t* slot;    // cell c: slot[c * kCellK + k]
};

__device__ __forceinline__ Rep rep_view(unsigned char* base, int n, int Gmax) {
    Rep r;
    r.sq = reinterpret_cast<float4*>(base);
    r.ang = reinterpret_cast<float*>(r.sq + n);
    r.cnt = reinterpret_cast<uint8_t*>(r.ang + n);
    r.slot = reinterpret_cast<uint16_t*>(r.cnt + ((Gmax * Gmax + 3) & ~3));
    return r;
}

struct Grid {
    int G;
    float inv;  // G / L
    __device__ __forceinline__ int cx(float x) const {
        int c = (int)floorf(x * inv);
        return c < 0 ? 0 : (c >= G ? G - 1 : c);
    }
};

__device__ __forceinline__ Grid make_grid(float L, int Gmax, float cell) {
    Grid g;
    int G = (int)(L / cell);
    g.G = G < 1 ? 1 : (G > Gmax ? Gmax : G);
    g.inv = (float)g.G / L;
    return g;
}

__device__ __forceinline__ float wall_e(float x, float y, float c, float s, float L) {
    return wall_energy(x, y, c, s, L);
}

// Build the cell list of one replica (warp).  Returns false on overflow (a
// cell asked for more than kCellK slots); the list is then incomplete but
// every count is clamped to kCellK and the slots below it are all written
// (ranks 0 .. kCellK - 1 were handed out), so no later scan can leave the
// replica's arrays.  Slots at or past a cell's count are never read.
__device__ bool build_cells(const Rep& R, int n, const Grid& g, int lane) {
    const int ncell = g.G * g.G;
    for (int c = 4 * lane; c < ncell; c += 128) *reinterpret_cast<uint32_t*>(R.cnt + c) = 0u;
    __syncwarp();
    bool ok = true;
    for (int i = lane; i < n; i += 32) {
        const float4 p = R.sq[i];
        const int c = g.cx(p.y) * g.G + g.cx(p.x);
        const unsigned k = atomicAdd(reinterpret_cast<unsigned*>(R.cnt + (c & ~3)), 1u << (8 * (c & 3)));
        const unsigned slot_k = (k >> (8 * (c & 3))) & 0xffu;
        if (slot_k < (unsigned)kCellK) R.slot[c * kCellK + slot_k] = (uint16_t)i;
        else ok = false;
    }
    __syncwarp();
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
        for (int c = lane; c < ncell; c += 32)
            if (R.cnt[c] > kCellK) R.cnt[c] = (uint8_t)kCellK;
        __syncwarp();
    }
    return ok;
}

// Visit the squares of the 3x3 cell block around (cx, cy): calls fn(j) for
// every candidate t = lane, lane + kStride, ... (kStride lanes share the
// block: the whole warp, or a part of it).  The three counts of a block row
// are neighbouring bytes: two aligned word loads and a funnel shift fetch
// them (the word past the counts is the slots'), and one multiplication turns
// them into running sums, a byte each.  Slot t of the block is then found by
// two compares for its row and two for its cell.  Against nine guarded byte
// loads, a nine-step sum and an eight-step search this halves the instructions
// around a candidate.
template <int kStride, typename Fn>
__device__ __forceinline__ void for_block(const Rep& R, const Grid& g, int cx, int cy, int lane, Fn&& fn) {
    const unsigned mask = cx == g.G - 1 ? 0x00ffffu : 0xffffffu;
    const int xs = cx > 0 ? cx - 1 : 0;
    unsigned p[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const int y = cy + r - 1;
        unsigned w = 0u;
        if ((unsigned)y < (unsigned)g.G) {
            const int a = y * g.G + xs;
            const uint32_t* q = reinterpret_cast<const uint32_t*>(R.cnt + (a & ~3));
            w = __funnelshift_r(q[0], q[1], 8 * (a & 3));
            w = (cx > 0 ? w : w << 8) & mask;
        }
        p[r] = w * 0x010101u;  // bytes: c0, c0 + c1, c0 + c1 + c2
    }
    const int t0 = (p[0] >> 16) & 0xff, t1 = t0 + (int)((p[1] >> 16) & 0xff), run = t1 + (int)((p[2] >> 16) & 0xff);
    const int cell0 = (cy - 1) * g.G + cx - 1;
    for (int t = lane; t < run; t += kStride) {
        const bool r1 = t >= t0, r2 = t >= t1;
        const unsigned q = r2 ? p[2] : (r1 ? p[1] : p[0]);
        const int u = t - (r2 ? t1 : (r1 ? t0 : 0));
        const int row = cell0 + (r2 ? 2 * g.G : (r1 ? g.G : 0));
        const int c0 = q & 0xff, c1 = (q >> 8) & 0xff;
        const bool k1 = u >= c0, k2 = u >= c1;
        const int cell = row + (int)k1 + (int)k2;
        fn((int)R.slot[cell * kCellK + u - (k2 ? c1 : (k1 ? c0 : 0))]);
    }
}

// Warp sum of the fixed-point energy change of one proposal: each lane's
// term is split as hi * 2^20 + lo (0 <= lo < 2^20) and both parts are summed
// with 32-bit warp reductions.  Exact while every lane's term is below 2^46
// in magnitude: a proposal's lane holds a few pair terms of at most
// 1.5 * 2^40 each (and lane 0 the wall change), far inside that.
__device__ __forceinline__ long long warp_sum_dq(long long v) {
    const unsigned lo = (unsigned)(v & 0xFFFFF);
    const int hi = (int)(v >> 20);
    const unsigned slo = __reduce_add_sync(0xffffffffu, lo);
    const int shi = __reduce_add_sync(0xffffffffu, hi);
    return (long long)shi * 1048576ll + (long long)slo;
}

__device__ __forceinline__ long long qe(float e) { return __float2ll_rn(e * kEScale); }

// Change of square Q's pair term when a square moves from P to (nx, ny) with
// (cos, sin) = (nc, ns), in kEScale units.  Both terms are evaluated and each
// is kept only inside the cut-off: the same values as testing first, without
// a branch around them (a warp's lanes almost always disagree on the test).
__device__ __forceinline__ long long pair_delta(float4 Q, float nx, float ny, float nc, float ns, float4 P) {
    const float ex = Q.x - nx, ey = Q.y - ny, fx = Q.x - P.x, fy = Q.y - P.y;
    const long long en = qe(sat_pair_energy(ex, ey, nc, ns, Q.z, Q.w));
    const long long eo = qe(sat_pair_energy(fx, fy, P.z, P.w, Q.z, Q.w));
    return (ex * ex + ey * ey < kPairCut2 ? en : 0) - (fx * fx + fy * fy < kPairCut2 ? eo : 0);
}

// Exact 64-bit warp sum in three warp reductions: the value's 26 low bits,
// the next 26 and the signed rest each sum within 32 bits.
__device__ __forceinline__ long long warp_sum_ll(long long v) {
    const unsigned s0 = __reduce_add_sync(0xffffffffu, (unsigned)v & 0x3ffffffu);
    const unsigned s1 = __reduce_add_sync(0xffffffffu, (unsigned)(v >> 26) & 0x3ffffffu);
    const int s2 = __reduce_add_sync(0xffffffffu, (int)(v >> 52));
    return (long long)(((unsigned long long)(long long)s2 << 52) + ((unsigned long long)s1 << 26) + s0);
}

__device__ __forceinline__ double warp_max_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ double warp_min_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Half of a square's 3 x 3 block: k = 0 its own cell, 1 the cell to the east,
// 2..4 the row above.  Over all squares these visit each unordered pair of
// neighbours once (in the own cell, from the lower index) when the lists are
// current, that is every square is listed in the cell its centre lies in.
__device__ __forceinline__ void half_block(int k, int& dx, int& dy) {
    dx = k == 0 ? 0 : (k == 1 ? 1 : k - 3);
    dy = k >= 2;
}

// Full energy of one replica (walls + each neighbour pair once), fixed
// point, on current lists.  Work item w is square w / 5 against cell w % 5 of
// its half block, a lane each: a warp takes 5 n / 32 short rounds.  One
// square at a time with the warp on its whole block left most lanes without
// a candidate and took n rounds of a nine-count prefix each; a collective
// move spends most of its time here.  With the certified side split the same
// way, the slots no longer cleared and the undo copies in shared memory, a
// search of n = 50 with 64 chains (40 epochs x 64) went from 101.8 to 65.4 ms.
__device__ long long full_energy(const Rep& R, int n, const Grid& g, float L, int lane) {
    long long e = 0;
    for (int w = lane; w < 5 * n; w += 32) {
        const int i = w / 5, c = w - 5 * i;
        const float4 P = R.sq[i];
        if (c == 0) e += qe(wall_e(P.x, P.y, P.z, P.w, L));
        int dx, dy;
        half_block(c, dx, dy);
        const int x = g.cx(P.x) + dx, y = g.cx(P.y) + dy;
        if (x < 0 || x >= g.G || y >= g.G) continue;
        const int cell = y * g.G + x, m = R.cnt[cell];
        for (int k = 0; k < m; ++k) {
            const int j = R.slot[cell * kCellK + k];
            if (c == 0 && j <= i) continue;
            const float4 Q = R.sq[j];
            const float ex = Q.x - P.x, ey = Q.y - P.y;
            if (ex * ex + ey * ey < kPairCut2) e += qe(sat_pair_energy(ex, ey, P.z, P.w, Q.z, Q.w));
        }
    }
    return warp_sum_ll(e);
}

// FP64 dilation-certified side of a replica (device_certified_side,
// seeded.cu:175-226): the smallest centre dilation lambda that opens a
// tau = 2.6e-8 gap along the best axis of every close pair, rejection above
// 1.008, side of the bounding box of the dilated squares.  Products are kept
// unfused so the result rounds like the host oracle's.
__device__ double cert_side(const Rep& R, int n, const Grid& g, int lane, double2* trig, double& lam_out, double& x0_out,
                            double& y0_out) {
    const double tau = 2.6e-8;
    double lam = 1.0;
    for (int i = lane; i < n; i += 32) {
        double s, c;
        sincos((double)R.ang[i], &s, &c);
        trig[i] = make_double2(c, s);
    }
    __syncwarp();
    // a lane per (square, cell of its half block): the required dilation of a
    // pair is the same from either side, and the largest one needs no order
    for (int w = lane; w < 5 * n; w += 32) {
        const int i = w / 5, c = w - 5 * i;
        const float4 P = R.sq[i];
        int hx, hy;
        half_block(c, hx, hy);
        const int x = g.cx(P.x) + hx, y = g.cx(P.y) + hy;
        if (x < 0 || x >= g.G || y >= g.G) continue;
        const int cell = y * g.G + x, m = R.cnt[cell];
        const double xi = P.x, yi = P.y, ci = trig[i].x, si = trig[i].y;
        for (int k = 0; k < m; ++k) {
            const int j = R.slot[cell * kCellK + k];
            if (c == 0 && j <= i) continue;
            const double dx = __dsub_rn(xi, (double)R.sq[j].x), dyv = __dsub_rn(yi, (double)R.sq[j].y);
            if (__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dyv, dyv)) >= 2.05) continue;
            const double cj = trig[j].x, sj = trig[j].y;
            const double c12 = fabs(__dadd_rn(__dmul_rn(ci, cj), __dmul_rn(si, sj)));
            const double s12 = fabs(__dadd_rn(__dmul_rn(-si, cj), __dmul_rn(ci, sj)));
            const double r = __dadd_rn(0.5, __dmul_rn(0.5, __dadd_rn(c12, s12)));
            const double v1 = fabs(__dadd_rn(__dmul_rn(dx, ci), __dmul_rn(dyv, si)));
            const double v2 = fabs(__dadd_rn(__dmul_rn(-dx, si), __dmul_rn(dyv, ci)));
            const double v3 = fabs(__dadd_rn(__dmul_rn(dx, cj), __dmul_rn(dyv, sj)));
            const double v4 = fabs(__dadd_rn(__dmul_rn(-dx, sj), __dmul_rn(dyv, cj)));
            const double vmax = fmax(fmax(v1, v2), fmax(v3, v4));
            const double req = vmax > 1e-12 ? __ddiv_rn(__dadd_rn(r, tau), vmax) : 1e9;
            lam = fmax(lam, req);
        }
    }
    lam = warp_max_d(lam);
    lam_out = lam;
    if (lam > 1.008) return 1e9;
    double bx0 = 1e9, bx1 = -1e9, by0 = 1e9, by1 = -1e9;
    for (int i = lane; i < n; i += 32) {
        const float4 P = R.sq[i];
        const double x = __dmul_rn((double)P.x, lam), y = __dmul_rn((double)P.y, lam);
        const double r = __dmul_rn(0.5, __dadd_rn(fabs(trig[i].x), fabs(trig[i].y)));
        bx0 = fmin(bx0, __dsub_rn(x, r));
        bx1 = fmax(bx1, __dadd_rn(x, r));
        by0 = fmin(by0, __dsub_rn(y, r));
        by1 = fmax(by1, __dadd_rn(y, r));
    }
    bx0 = warp_min_d(bx0);
    bx1 = warp_max_d(bx1);
    by0 = warp_min_d(by0);
    by1 = warp_max_d(by1);
    x0_out = bx0;
    y0_out = by0;
    return fmax(__dsub_rn(bx1, bx0), __dsub_rn(by1, by0));
}

// ---- Cooperative forms: a group of warps works on one replica, one warp
// (WarpGrp) or several on a named barrier (BarGrp).  Results do not depend on
// the group: every sum below is an integer sum and slot order within a cell
// list changes no energy, gradient or decision.  A group sum publishes one
// partial a warp and takes one barrier; each kind of sum has its own slots,
// and two sums of one kind always have another barrier between them.
struct WarpGrp {
    int lane;
    __device__ __forceinline__ int t() const { return lane; }
    __device__ __forceinline__ int nt() const { return 32; }
    __device__ __forceinline__ void sync() const { __syncwarp(); }
    __device__ __forceinline__ bool sync_or(bool p) const {
        __syncwarp();
        return __any_sync(0xffffffffu, p);
    }
    __device__ __forceinline__ long long sum(long long v) const {
        __syncwarp();
        return warp_sum_ll(v);
    }
    __device__ __forceinline__ void sum2(long long& a, long long& b) const {
        a = warp_sum_ll(a);
        b = warp_sum_ll(b);
    }
    // group maximum of m and group OR of f; orders the group's memory like sync()
    __device__ __forceinline__ void max_or(unsigned& m, bool& f) const {
        m = __reduce_max_sync(0xffffffffu, m);
        f = __any_sync(0xffffffffu, f);
        __syncwarp();
    }
};
constexpr int kGrpSlots = 4;  // two dot products, the energy sum, maximum and flag
// `nw` consecutive warps of the CTA (nw >= 2) on named barrier `id` (1..15).
// The barrier is the non-aligned form: after a lane-strided loop nothing
// promises that a warp reaches it converged.
struct BarGrp {
    int id, nw, t0;  // barrier, warps, first thread of the group
    long long* red;  // kGrpSlots slots per warp of the group
    __device__ __forceinline__ int t() const { return (int)threadIdx.x - t0; }
    __device__ __forceinline__ int nt() const { return 32 * nw; }
    __device__ __forceinline__ void sync() const {
        asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(32 * nw) : "memory");
    }
    __device__ __forceinline__ bool sync_or(bool p) const {
        unsigned r;
        asm volatile(
            "{\n\t.reg .pred ip, op;\n\tsetp.ne.u32 ip, %1, 0;\n\tbarrier.red.or.pred op, %2, %3, ip;\n\t"
            "selp.u32 %0, 1, 0, op;\n\t}"
            : "=r"(r)
            : "r"((unsigned)p), "r"(id), "r"(32 * nw)
            : "memory");
        return r != 0;
    }
    __device__ __forceinline__ long long slot_sum(int k) const {
        const int lane = threadIdx.x & 31;
        return warp_sum_ll(lane < nw ? red[kGrpSlots * lane + k] : 0);
    }
    __device__ __forceinline__ long long sum(long long v) const {
        v = warp_sum_ll(v);
        if ((threadIdx.x & 31) == 0) red[kGrpSlots * (t() >> 5) + 2] = v;
        sync();
        return slot_sum(2);
    }
    __device__ __forceinline__ void sum2(long long& a, long long& b) const {
        a = warp_sum_ll(a);
        b = warp_sum_ll(b);
        if ((threadIdx.x & 31) == 0) {
            long long* r = red + kGrpSlots * (t() >> 5);
            r[0] = a;
            r[1] = b;
        }
        sync();
        a = slot_sum(0);
        b = slot_sum(1);
    }
    __device__ __forceinline__ void max_or(unsigned& m, bool& f) const {
        m = __reduce_max_sync(0xffffffffu, m);
        f = __any_sync(0xffffffffu, f);
        const int lane = threadIdx.x & 31;
        if (lane == 0) red[kGrpSlots * (t() >> 5) + 3] = (long long)(((unsigned long long)f << 32) | m);
        sync();
        const unsigned long long v = lane < nw ? (unsigned long long)red[kGrpSlots * lane + 3] : 0ull;
        m = __reduce_max_sync(0xffffffffu, (unsigned)v);
        f = __any_sync(0xffffffffu, (v >> 32) != 0);
    }
};

template <class Grp>
__device__ bool build_cells_grp(const Grp& gp, const Rep& R, int n, const Grid& g) {
    const int ncell = g.G * g.G, tid = gp.t(), nt = gp.nt();
    for (int c = 4 * tid; c < ncell; c += 4 * nt) *reinterpret_cast<uint32_t*>(R.cnt + c) = 0u;
    gp.sync();
    bool ok = true;
    for (int i = tid; i < n; i += nt) {
        const float4 p = R.sq[i];
        const int c = g.cx(p.y) * g.G + g.cx(p.x);
        const unsigned k = atomicAdd(reinterpret_cast<unsigned*>(R.cnt + (c & ~3)), 1u << (8 * (c & 3)));
        const unsigned slot_k = (k >> (8 * (c & 3))) & 0xffu;
        if (slot_k < (unsigned)kCellK) R.slot[c * kCellK + slot_k] = (uint16_t)i;
        else ok = false;
    }
    const bool bad = gp.sync_or(!ok);
    if (bad) {
        for (int c = tid; c < ncell; c += nt)
            if (R.cnt[c] > kCellK) R.cnt[c] = (uint8_t)kCellK;
        gp.sync();
    }
    return !bad;
}

// Full fixed-point energy of a trial state on the lists of the state it
// moved from.  Work item w is square w / 9 against the squares listed in cell
// w % 9 of its 3 x 3 block, each pair counted from its lower index (the half
// block of full_energy needs current lists).
template <class Grp>
__device__ long long full_energy_grp(const Grp& gp, const Rep& R, int n, const Grid& g, float L) {
    long long e = 0;
    for (int w = gp.t(); w < 9 * n; w += gp.nt()) {
        const int i = w / 9, c = w - 9 * i;
        const float4 P = R.sq[i];
        if (c == 0) e += qe(wall_e(P.x, P.y, P.z, P.w, L));
        const int x = g.cx(P.x) + c % 3 - 1, y = g.cx(P.y) + c / 3 - 1;
        if (x < 0 || x >= g.G || y < 0 || y >= g.G) continue;
        const int cell = y * g.G + x, m = R.cnt[cell];
        for (int k = 0; k < m; ++k) {
            const int j = R.slot[cell * kCellK + k];
            if (j <= i) continue;
            const float4 Q = R.sq[j];
            const float dx = Q.x - P.x, dy2 = Q.y - P.y;
            if (dx * dx + dy2 * dy2 < kPairCut2) e += qe(sat_pair_energy(dx, dy2, P.z, P.w, Q.z, Q.w));
        }
    }
    return gp.sum(e);
}

// Quench gradient sums: 32-bit integers in units of 2^-20.  A square's 3 x 3
// block lists at most 9 x 12 partners, each term below 5.2 (and the wall
// term below 1), so a sum stays below 6e8 < 2^31; integer atomics make the
// sums independent of the order of the terms.
constexpr float kQScale = 1048576.0f;
__device__ __forceinline__ int qg(float v) { return __float2int_rn(v * kQScale); }

// Line-search pair list.  A trial moves every centre coordinate by at most
// kListStep from the saved state; then a pair within the cut-off at the trial
// was at most 1.4142 + 2 kListStep < 1.59 (the smallest cell side) apart per
// axis at the saved state, so it sits in the saved 3 x 3 cell blocks, and at
// most sqrt(kPairCut2) + 2 sqrt(2) kListStep = 1.6546 apart: the pairs of
// those blocks closer than sqrt(kListCut2) = 1.6583 hold every pair with a
// non-zero trial energy, and the list's energy equals the full one exactly.
constexpr float kListStep = 0.085f, kListCut2 = 2.75f;

// Energy of a warp's replica over its pair list.  Two pairs a lane at once:
// the chains of loads and FP32 operations overlap.
__device__ long long list_energy(const Rep& R, int n, float L, const uint32_t* pl, int cnt, int lane) {
    long long e = 0;
    for (int i = lane; i < n; i += 32) {
        const float4 P = R.sq[i];
        e += qe(wall_e(P.x, P.y, P.z, P.w, L));
    }
    for (int k = lane; k < cnt; k += 64) {
        float v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const bool in = k + 32 * u < cnt;
            const uint32_t pr = pl[in ? k + 32 * u : k];
            const float4 P = R.sq[pr & 0xffffu], Q = R.sq[pr >> 16];
            const float dx = Q.x - P.x, dy = Q.y - P.y;
            const float pe = sat_pair_energy(dx, dy, P.z, P.w, Q.z, Q.w);
            v[u] = in && dx * dx + dy * dy < kPairCut2 ? pe : 0.f;
        }
        e += qe(v[0]) + qe(v[1]);
    }
    return warp_sum_ll(e);
}

// A thread's share of the energy over the pair list, and the gradient summed
// into tg (walls, and both sides of every overlapping pair); two pairs a
// thread at once as above.
template <class Grp>
__device__ __forceinline__ long long list_eval(const Grp& gp, const Rep& R, int n, float L, const uint32_t* pl, int cnt,
                                               int4* tg) {
    long long e = 0;
    // walls from the last thread down: the first ones have a second pair
    for (int i = gp.nt() - 1 - gp.t(); i < n; i += gp.nt()) {
        const float4 P = R.sq[i];
        e += qe(wall_e(P.x, P.y, P.z, P.w, L));
        float wx = 0.f, wy = 0.f, wa = 0.f;
        wall_energy_grad(P.x, P.y, P.z, P.w, L, wx, wy, wa);
        const int ax = qg(wx), ay = qg(wy), aa = qg(wa);
        if (ax | ay | aa) {
            atomicAdd(&tg[i].x, ax);
            atomicAdd(&tg[i].y, ay);
            atomicAdd(&tg[i].z, aa);
        }
    }
    for (int k = gp.t(); k < cnt; k += 2 * gp.nt()) {
        uint32_t pr[2];
        float4 P[2], Q[2];
        PairAxes ax[2];
        bool hit[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const bool in = k + u * gp.nt() < cnt;
            pr[u] = pl[in ? k + u * gp.nt() : k];
            P[u] = R.sq[pr[u] & 0xffffu];
            Q[u] = R.sq[pr[u] >> 16];
            const float dx = Q[u].x - P[u].x, dy = Q[u].y - P[u].y;
            ax[u] = sat_axes(dx, dy, P[u].z, P[u].w, Q[u].z, Q[u].w);
            hit[u] = in && dx * dx + dy * dy < kPairCut2 && ax[u].gap < 0.f;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (hit[u]) {
                PairGrad pg;  // q's side equals the pair taken from q, bit for bit
                sat_grad(ax[u], P[u].z, P[u].w, Q[u].z, Q[u].w, pg);
                e += qe(pg.e);
                int4* a = tg + (pr[u] & 0xffffu);
                int4* b = tg + (pr[u] >> 16);
                atomicAdd(&a->x, qg(pg.px));
                atomicAdd(&a->y, qg(pg.py));
                atomicAdd(&a->z, qg(pg.pa));
                atomicAdd(&b->x, qg(pg.qx));
                atomicAdd(&b->y, qg(pg.qy));
                atomicAdd(&b->z, qg(pg.qa));
            }
        }
    }
    return e;
}

__device__ __forceinline__ int clamp_q24(int v) { return max(-(1 << 24), min(1 << 24, v)); }

// The checkpoint quench of one replica (the coldest, or each one under
// SQS_JOB_QUENCH_ALL) by a group of threads: the reference's conjugate-gradient
// polish (seeded.cu:621-715) on the overlap energy.  Each iteration takes the
// gradient, a Polak-Ribiere direction d = -g + beta d (beta = max(0, (g -
// g_old).g / g_old.g), 0 on the first iteration and every 25th), and a
// backtracking line search of up to 5 trials from the carried step (x 0.45
// per trial).  An accepted trial sets the step to min(0.15, 1.25 alpha); when
// no trial improves, the direction is dropped and the step halves (at least
// 1e-7) -- the polish goes on from the same state, whose gradient is kept.
// It ends at zero energy, at a zero gradient, after `iters` iterations, or,
// with a stall limit (not kQuenchNoStall), after `stall_limit` accepted steps
// in a row that each gained less than 0.1% or at a line search without a gain.
// Gradients and their dot products are integer sums, so the result does not
// depend on the group's width.
//
// A step is a chain of short phases with a group barrier after each, so the
// barriers are what it costs: an accepted first trial takes three (dot
// products; direction, trial state, largest component and cell changes at
// once; energy and gradient of the trial).  Square i belongs to thread i mod nt throughout, so what
// only its owner reads (direction, saved state, old gradient) needs none, and
// the cell lists are rebuilt only when a square of the accepted trial has
// left its cell.  Scratch: kQuenchScr n float4 (gradient sums of this and of
// the previous iteration, direction, saved state, pair list: two counters and
// up to 8 n - 2 pairs).
template <class Grp>
__device__ long long quench_grp(const Grp& gp, const Rep& R, int n, const Grid& g, float L, int iters, int stall_limit,
                                float4* scr, long long E) {
    int4* acc = reinterpret_cast<int4*>(scr);       // gradient sums at the current state
    int4* gold = reinterpret_cast<int4*>(scr + n);  // at the state before, then at the trial
    float4* dir = scr + 2 * n;                      // search direction
    float4* saved = scr + 3 * n;                    // state before the line search
    uint32_t* plist = reinterpret_cast<uint32_t*>(scr + 4 * n);  // [cur] count, [cur ^ 1] zero, pairs
    const int pcap = 8 * n - 2;
    float step = 0.04f;
    int stall = 0;  // consecutive accepted steps that gained less than 0.1%
    float drift = 1e30f;  // bound on any centre's per-axis move since the pair list was built (none yet)
    int cur = 0;          // the pair list's counter
    bool fresh = true;    // the state moved since its gradient was taken
    bool have = false;    // acc holds the gradient of the state
    bool away = false;    // the replica holds a rejected trial, not the saved state
    long long s_gg = 0, s_oo = 0;
    for (int i = gp.t(); i < n; i += gp.nt()) {
        acc[i] = make_int4(0, 0, 0, 0);
        gold[i] = make_int4(0, 0, 0, 0);
        dir[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        saved[i] = make_float4(R.sq[i].x, R.sq[i].y, R.ang[i], 0.f);
    }
    if (gp.t() == 0) plist[0] = plist[1] = 0u;
    gp.sync();
    auto restore = [&]() {  // the owner's squares back to the saved state
        for (int i = gp.t(); i < n; i += gp.nt()) {
            const float4 o = saved[i];
            float sn, cs;
            state_trig(o.z, &sn, &cs);
            R.sq[i] = make_float4(o.x, o.y, cs, sn);
            R.ang[i] = o.z;
        }
        gp.sync();
    };
    for (int it = 0; it < iters && E > 0; ++it) {
        float beta = 0.f;
        if (fresh) {
            // A trial taken over the pair list brought its gradient along; a
            // state reached by the cell scan (the first, or one past the list's
            // reach) gets its gradient here, and a new list with it.
            if (!have) {
                // work item w: square w / 9 against cell w % 9 of its block; it also
                // lists the block's pairs (i < j) closer than sqrt(kListCut2)
                cur ^= 1;
                for (int w = gp.t(); w < 9 * n; w += gp.nt()) {
                    const int i = w / 9, c = w - 9 * i;
                    const float4 P = R.sq[i];
                    int ax = 0, ay = 0, aa = 0;
                    if (c == 0) {
                        float wx = 0.f, wy = 0.f, wa = 0.f;
                        wall_energy_grad(P.x, P.y, P.z, P.w, L, wx, wy, wa);
                        ax = qg(wx);
                        ay = qg(wy);
                        aa = qg(wa);
                    }
                    const int x = g.cx(P.x) + c % 3 - 1, y = g.cx(P.y) + c / 3 - 1;
                    if (x >= 0 && x < g.G && y >= 0 && y < g.G) {
                        const int cell = y * g.G + x, m = R.cnt[cell];
                        for (int k = 0; k < m; ++k) {
                            const int j = R.slot[cell * kCellK + k];
                            if (j == i) continue;
                            const float4 Q = R.sq[j];
                            const float ex = Q.x - P.x, ey = Q.y - P.y;
                            const float d2 = ex * ex + ey * ey;
                            if (j > i && d2 < kListCut2) {
                                const uint32_t slot = atomicAdd(&plist[cur], 1u);
                                if (slot < (uint32_t)pcap) plist[2 + slot] = (uint32_t)i | ((uint32_t)j << 16);
                            }
                            if (d2 >= kPairCut2) continue;
                            PairGrad pg;
                            if (sat_pair_grad(ex, ey, P.z, P.w, Q.z, Q.w, pg)) {
                                ax += qg(pg.px);
                                ay += qg(pg.py);
                                aa += qg(pg.pa);
                            }
                        }
                    }
                    if (ax | ay | aa) {
                        atomicAdd(&acc[i].x, ax);
                        atomicAdd(&acc[i].y, ay);
                        atomicAdd(&acc[i].z, aa);
                    }
                }
                gp.sync();
                drift = plist[cur] <= (uint32_t)pcap ? 0.f : 1e30f;  // an overflowed list is not used
            }
            // Polak-Ribiere: g.g and g_old.g as exact integer sums of
            // components clamped to 2^24 (a gradient of 16; only beta sees the
            // clamp): 3 n <= 3000 terms below 2^48 each fit 64 bits.
            // g_old.g_old is the g.g of the state before.
            long long s_og = 0;
            s_gg = 0;
            for (int i = gp.t(); i < n; i += gp.nt()) {
                const int4 a = acc[i], o = gold[i];
                const int gx = clamp_q24(a.x), gy = clamp_q24(a.y), ga = clamp_q24(a.z);
                const int ox = clamp_q24(o.x), oy = clamp_q24(o.y), oa = clamp_q24(o.z);
                s_og += (long long)gx * ox + (long long)gy * oy + (long long)ga * oa;
                s_gg += (long long)gx * gx + (long long)gy * gy + (long long)ga * ga;
            }
            gp.sum2(s_gg, s_og);
            const long long s_dg = s_gg - s_og;
            beta = (it == 0 || s_oo == 0 || it % 25 == 0 || s_dg <= 0) ? 0.f : (float)((double)s_dg / (double)s_oo);
        }
        if (s_gg == 0 && beta == 0.f) break;  // no direction left at the sums' resolution
        const int npairs = (int)plist[cur];
        float dmax = 0.f;
        // Trial steps move every coordinate by at most 0.1, so each partner
        // within the pair cut-off of a moved square still sits in one of the
        // 3 x 3 cells around it on the lists built for the saved state
        // (1.4142 + 0.1 < 1.59 <= cell side): trial energies use those lists.
        // A trial that keeps every centre within kListStep per axis of where
        // the pair list was built sums the list instead (the same energy,
        // without the cell scan).
        float alpha = step;
        bool moved = false;
        for (int tries = 0; tries < 5 && !moved; ++tries) {
            unsigned dbits = 0u;  // largest |d.x|, |d.y| (bits of non-negative floats order as integers)
            bool left = false;    // a square left its cell
            for (int i = gp.t(); i < n; i += gp.nt()) {
                float4 d = dir[i];
                if (tries == 0) {
                    const int4 a = acc[i];
                    d = make_float4(__fmaf_rn(beta, d.x, -(float)a.x * (1.0f / kQScale)),
                                    __fmaf_rn(beta, d.y, -(float)a.y * (1.0f / kQScale)),
                                    __fmaf_rn(beta, d.z, -(float)a.z * (1.0f / kQScale)), 0.f);
                    dir[i] = d;
                    dbits = max(dbits, __float_as_uint(fmaxf(fabsf(d.x), fabsf(d.y))));
                }
                gold[i] = make_int4(0, 0, 0, 0);  // consumed: the trial's gradient is summed here
                const float4 o = saved[i];
                const float sx = fminf(0.1f, fmaxf(-0.1f, alpha * d.x));
                const float sy = fminf(0.1f, fmaxf(-0.1f, alpha * d.y));
                const float a = wrap_quarter_f(o.z + fminf(0.1f, fmaxf(-0.1f, alpha * d.z)));
                float sn, cs;
                state_trig(a, &sn, &cs);
                const float nx = o.x + sx, ny = o.y + sy;
                R.sq[i] = make_float4(nx, ny, cs, sn);
                R.ang[i] = a;
                left |= g.cx(nx) != g.cx(o.x) || g.cx(ny) != g.cx(o.y);
            }
            if (tries == 0 && gp.t() == 0) plist[cur ^ 1] = 0u;
            gp.max_or(dbits, left);
            if (tries == 0) dmax = __uint_as_float(dbits);
            const bool by_list = npairs <= pcap && drift + alpha * dmax <= kListStep;
            const long long En = by_list ? gp.sum(list_eval(gp, R, n, L, plist + 2, npairs, gold))
                                         : full_energy_grp(gp, R, n, g, L);
            if (En < E && (!left || build_cells_grp(gp, R, n, g))) {
                stall = En > E - E / 1000 ? stall + 1 : 0;  // less than 0.1% gained
                E = En;
                step = fminf(0.15f, alpha * 1.25f);
                drift += fminf(0.1f, alpha * dmax);  // every centre moved at most this far per axis
                moved = true;
                have = by_list;
                for (int i = gp.t(); i < n; i += gp.nt())
                    saved[i] = make_float4(R.sq[i].x, R.sq[i].y, R.ang[i], 0.f);
            } else {
                if (En < E) {  // the better state overflows a cell: lists back to the saved state
                    restore();
                    build_cells_grp(gp, R, n, g);  // the saved state fitted
                }
                alpha *= 0.45f;
            }
        }
        fresh = moved;
        away = !moved;
        if (moved) {
            int4* const s = acc;
            acc = gold;
            gold = s;
            s_oo = s_gg;
        } else {  // direction dropped (beta is 0 next), the saved state's gradient kept
            step = fmaxf(1e-7f, step * 0.5f);
            if (stall_limit < kQuenchNoStall) break;  // the library's default quench ends here
        }
        if (stall >= stall_limit) break;
    }
    if (away) restore();  // the lists are those of the saved state
    return E;
}

// Quench of replica view R by warps 0 .. gw - 1 of a group that starts at
// thread t0 (all of them call this): one warp for 8 squares, at most gw.  More
// warps than that add barrier latency and no parallelism.  400 checkpoints of
// n = 10: 53.9 ms with 16 squares a warp, 51.8 with 8, 51.1 with 4; 16
// replicas of n = 60: 16.6, 16.1, 16.6; n = 50 with 64 chains, whose groups
// have 4 warps: 48.4 each.
constexpr int kQuenchSquares = 8;
__device__ __forceinline__ long long quench_group(int id, int gw, int t0, long long* red, const Rep& R, int n,
                                                  const Grid& g, float L, int iters, int stall_limit, float4* scr,
                                                  long long E) {
    const int nw = min(gw, (n + kQuenchSquares - 1) / kQuenchSquares), t = (int)threadIdx.x - t0;
    if (t >= 32 * nw) return E;
    if (nw == 1) return quench_grp(WarpGrp{t}, R, n, g, L, iters, stall_limit, scr, E);
    return quench_grp(BarGrp{id, nw, t0, red}, R, n, g, L, iters, stall_limit, scr, E);
}

// Pair list of a warp's replica for collective moves: every pair closer than
// sqrt(kListCut2) at the reference state, whose centres go to `ref`.  It holds
// every pair inside the cut-off while each centre stays within kListStep per
// axis of its reference (the quench's argument above).  Pairs are ranked by
// ballots, without atomics.  Returns the number of pairs (past `pcap` the list
// is incomplete and not to be used).  The cell lists must be current.
__device__ int build_pair_list(const Rep& R, int n, const Grid& g, int lane, float2* ref, uint32_t* pl, int pcap) {
    int cnt = 0;
    for (int i = lane; i < n; i += 32) ref[i] = make_float2(R.sq[i].x, R.sq[i].y);
    for (int w0 = 0; w0 < 5 * n; w0 += 32) {
        const int w = w0 + lane, i = w / 5, c = w - 5 * i;
        int m = 0, cell = 0;
        float4 P = make_float4(0.f, 0.f, 0.f, 0.f);
        if (w < 5 * n) {
            P = R.sq[i];
            int dx, dy;
            half_block(c, dx, dy);
            const int x = g.cx(P.x) + dx, y = g.cx(P.y) + dy;
            if (x >= 0 && x < g.G && y < g.G) {
                cell = y * g.G + x;
                m = R.cnt[cell];
            }
        }
        const int most = __reduce_max_sync(0xffffffffu, m);
        for (int k = 0; k < most; ++k) {
            int j = 0;
            bool take = false;
            if (k < m) {
                j = R.slot[cell * kCellK + k];
                const float ex = R.sq[j].x - P.x, ey = R.sq[j].y - P.y;
                take = (c != 0 || j > i) && ex * ex + ey * ey < kListCut2;
            }
            const unsigned b = __ballot_sync(0xffffffffu, take);
            const int at = cnt + __popc(b & ((1u << lane) - 1u));
            if (take && at < pcap) pl[at] = (uint32_t)i | ((uint32_t)j << 16);
            cnt += __popc(b);
        }
    }
    __syncwarp();
    return cnt;
}

// Collective proposal (one warp, one replica): the set of squares the mode
// selects around square `c` -- 1 its row (|dy| < 0.55), 2 its column
// (|dx| < 0.55), 3 the disc dx^2 + dy^2 < 2.5, 4 its orientation class
// (angles within 0.06 modulo pi/2), 5 its diagonal strips (|dx +- dy| < 0.85),
// 6 every tilted square (0.04 < a < 1.53) -- is translated by (tx, ty)
// (mode 6: by +-(tx, ty) alternating with the square index), rotated about
// the drawn square by `th` for modes 3 and 4, and every moved square turned by
// `th` (seeded.cu:547-613).  Centres stay in [0.5, L - 0.5].  The move is
// judged on the full fixed-point energy, over the replica's pair list: a scan
// of the cells takes a serial chain of loads per candidate (16,000 cycles a
// move at n = 50, against 3,900 over the list).  The list is built at the state
// under trial when there is none or a square has left its reach, and `npl`
// (its pairs; -1: none) is kept by the caller across proposals.  The cell
// lists are rebuilt only when a square changes cells.  A rejected move (or one
// that overflows a cell) is undone from `scr`, the replica's scratch block
// (n float4 undo copy, at 3 n the reference centres, from 4 n the pairs).
// Returns whether it was accepted; an overflow adds `count` to *ovf.
__device__ __forceinline__ bool collective_move(const Rep& rep, const Grid& g, int n, float L, int lane, int mode, int c,
                                             float tx, float ty, float th, float u, float invT, long long& E,
                                             float4* __restrict__ scr, int& npl, int count, int* ovf) {
    float4* save = scr;
    float2* ref = reinterpret_cast<float2*>(scr + 3 * n);
    uint32_t* pl = reinterpret_cast<uint32_t*>(scr + 4 * n);
    const int pcap = 8 * n;
    const float cx = rep.sq[c].x, cy = rep.sq[c].y, ca = rep.ang[c];
    float st, ct;
    state_trig(th, &st, &ct);
    __syncwarp();
    bool left = false;  // a square changes cells
    bool far = false;   // a square leaves the pair list's reach
    bool big = false;   // a square moves further than kListStep
    for (int s = lane; s < n; s += 32) {
        const float4 P = rep.sq[s];
        const float a = rep.ang[s];
        const float ex = P.x - cx, ey = P.y - cy, da = a - ca;
        const bool take = mode == 1   ? fabsf(ey) < 0.55f
                          : mode == 2 ? fabsf(ex) < 0.55f
                          : mode == 3 ? ex * ex + ey * ey < 2.5f
                          : mode == 4 ? (fabsf(da) < 0.06f || fabsf(da) > kHalfPiF - 0.06f)
                          : mode == 5 ? (fabsf(ex + ey) < 0.85f || fabsf(ex - ey) < 0.85f)
                                      : (a > 0.04f && a < 1.53f);
        save[s] = make_float4(P.x, P.y, a, take ? 1.f : 0.f);
        if (take) {
            float nx, ny;
            if (mode == 3 || mode == 4) {
                nx = cx + ct * ex - st * ey + tx;
                ny = cy + st * ex + ct * ey + ty;
            } else if (mode == 6) {
                const float sg = (s & 1) ? 1.f : -1.f;
                nx = P.x + sg * tx;
                ny = P.y + sg * ty;
            } else {
                nx = P.x + tx;
                ny = P.y + ty;
            }
            nx = fminf(L - 0.5f, fmaxf(0.5f, nx));
            ny = fminf(L - 0.5f, fmaxf(0.5f, ny));
            const float na = wrap_quarter_f(a + th);
            float sn, cs;
            state_trig(na, &sn, &cs);
            rep.sq[s] = make_float4(nx, ny, cs, sn);
            rep.ang[s] = na;
            left |= g.cx(nx) != g.cx(P.x) || g.cx(ny) != g.cx(P.y);
            big |= !(fabsf(nx - P.x) <= kListStep && fabsf(ny - P.y) <= kListStep);
            if (npl >= 0) far |= !(fabsf(nx - ref[s].x) <= kListStep && fabsf(ny - ref[s].y) <= kListStep);
        }
    }
    __syncwarp();
    left = __any_sync(0xffffffffu, left);
    const bool build = npl < 0 || __any_sync(0xffffffffu, far);
    const bool fits = !left || build_cells(rep, n, g, lane);
    bool acc = false;
    if (fits) {
        if (build) npl = build_pair_list(rep, n, g, lane, ref, pl, pcap);
        const long long En =
            npl <= pcap ? list_energy(rep, n, L, pl, npl, lane) : full_energy(rep, n, g, L, lane);
        if (npl > pcap) npl = -1;
        const long long dq = En - E;
        acc = dq <= 0 || u < __expf(-((float)dq * (1.0f / kEScale)) * invT);
        if (acc) E = En;
    } else {
        *ovf += count;
    }
    if (!acc) {
        for (int s = lane; s < n; s += 32) {
            const float4 o = save[s];
            if (o.w != 0.f) {
                float sn, cs;
                state_trig(o.z, &sn, &cs);
                rep.sq[s] = make_float4(o.x, o.y, cs, sn);
                rep.ang[s] = o.z;
            }
        }
        __syncwarp();
        if (left) build_cells(rep, n, g, lane);  // the saved state fitted
        // a list built at the trial serves the saved state if that is in its reach
        if (build && fits && __any_sync(0xffffffffu, big)) npl = -1;
    }
    return acc;
}

// Kick of an overlapped replica at an exchange round (seeded.cu:721-778):
// every square's energy (its wall term and its pairs); on odd rounds, when
// the worst square's energy exceeds 1e-5, that square moves to the probe of
// an 8 x 8 grid over [0.55, L - 0.55]^2 farthest from every other centre
// (jittered by up to 0.05, a fresh angle); then every square is jittered,
// by up to 0.08 / 0.18 rad where its energy exceeds 1e-6 and 0.008 / 0.015
// elsewhere.  Draws are Philox blocks keyed by (round, square, replica).
// Returns the new energy (the old one if a cell would overflow, the state
// then restored from `save`).
__device__ __forceinline__ long long kick_replica(const Rep& rep, const Grid& g, int n, float L, int lane, int r,
                                               int round, uint32_t k0, uint32_t k1, long long E,
                                               float4* __restrict__ save) {
    float wmax = -1.f;
    int worst = 0x7fffffff;
    for (int s = lane; s < n; s += 32) {
        const float4 P = rep.sq[s];
        float e = wall_e(P.x, P.y, P.z, P.w, L);
        const int cxs = g.cx(P.x), cys = g.cx(P.y);
        for (int dyc = -1; dyc <= 1; ++dyc) {
            for (int dxc = -1; dxc <= 1; ++dxc) {
                const int x = cxs + dxc, y = cys + dyc;
                if (x < 0 || x >= g.G || y < 0 || y >= g.G) continue;
                const int cell = y * g.G + x, m = rep.cnt[cell];
                for (int k = 0; k < m; ++k) {
                    const int j = rep.slot[cell * kCellK + k];
                    if (j == s) continue;
                    const float4 Q = rep.sq[j];
                    const float dx = Q.x - P.x, dy = Q.y - P.y;
                    if (dx * dx + dy * dy < kPairCut2) e += sat_pair_energy(dx, dy, P.z, P.w, Q.z, Q.w);
                }
            }
        }
        save[s] = make_float4(P.x, P.y, rep.ang[s], e);
        if (e > wmax) {
            wmax = e;
            worst = s;
        }
    }
    // warp arg-max (ties: the smaller index)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float om = __shfl_xor_sync(0xffffffffu, wmax, o);
        const int oi = __shfl_xor_sync(0xffffffffu, worst, o);
        if (om > wmax || (om == wmax && oi < worst)) {
            wmax = om;
            worst = oi;
        }
    }
    if ((round & 1) && wmax > 1e-5f && worst < n) {
        float bd = -1.f;
        int bp = 64;
        for (int p = lane; p < 64; p += 32) {
            const float vx = 0.55f + (L - 1.1f) * ((float)(p % 8) + 0.5f) / 8.f;
            const float vy = 0.55f + (L - 1.1f) * ((float)(p / 8) + 0.5f) / 8.f;
            float d2 = 1e9f;
            for (int j = 0; j < n; ++j) {
                if (j == worst) continue;
                const float dx = vx - rep.sq[j].x, dy = vy - rep.sq[j].y;
                d2 = fminf(d2, dx * dx + dy * dy);
            }
            if (d2 > bd) {
                bd = d2;
                bp = p;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float od = __shfl_xor_sync(0xffffffffu, bd, o);
            const int op = __shfl_xor_sync(0xffffffffu, bp, o);
            if (od > bd || (od == bd && op < bp)) {
                bd = od;
                bp = op;
            }
        }
        if (lane == 0) {
            const U4 q = philox4x32_10(U4{(uint32_t)round, 0xffffu, (uint32_t)r, 3u}, k0, k1);
            const float vx = 0.55f + (L - 1.1f) * ((float)(bp % 8) + 0.5f) / 8.f;
            const float vy = 0.55f + (L - 1.1f) * ((float)(bp / 8) + 0.5f) / 8.f;
            const float na = wrap_quarter_f(u01(q.z) * kHalfPiF);
            float sn, cs;
            state_trig(na, &sn, &cs);
            rep.sq[worst] = make_float4(fminf(L - 0.5f, fmaxf(0.5f, vx + 0.05f * (2.f * u01(q.x) - 1.f))),
                                        fminf(L - 0.5f, fmaxf(0.5f, vy + 0.05f * (2.f * u01(q.y) - 1.f))), cs, sn);
            rep.ang[worst] = na;
        }
        __syncwarp();
    }
    for (int s = lane; s < n; s += 32) {
        const float hot = save[s].w > 1e-6f;
        const float axy = hot ? 0.08f : 0.008f, aa = hot ? 0.18f : 0.015f;
        const U4 q = philox4x32_10(U4{(uint32_t)round, (uint32_t)s, (uint32_t)r, 2u}, k0, k1);
        const float4 P = rep.sq[s];
        const float na = wrap_quarter_f(rep.ang[s] + aa * (2.f * u01(q.z) - 1.f));
        float sn, cs;
        state_trig(na, &sn, &cs);
        rep.sq[s] = make_float4(fminf(L - 0.48f, fmaxf(0.48f, P.x + axy * (2.f * u01(q.x) - 1.f))),
                                fminf(L - 0.48f, fmaxf(0.48f, P.y + axy * (2.f * u01(q.y) - 1.f))), cs, sn);
        rep.ang[s] = na;
    }
    __syncwarp();
    if (build_cells(rep, n, g, lane)) return full_energy(rep, n, g, L, lane);
    for (int s = lane; s < n; s += 32) {
        const float4 o = save[s];
        float sn, cs;
        state_trig(o.z, &sn, &cs);
        rep.sq[s] = make_float4(o.x, o.y, cs, sn);
        rep.ang[s] = o.z;
    }
    __syncwarp();
    build_cells(rep, n, g, lane);
    return E;
}

// Rungs per ladder (a job's R rungs form `ladders` ladders of RL rungs; rung
// k is position k % RL of ladder k / RL, as the reference groups its chains
// into ladders of 8, seeded.cu:493, 791-817).
__device__ __forceinline__ int rungs_per_ladder(const JobDev& jd) { return jd.R / max(1, jd.ladders); }

// Ladder temperature of rung k: geometric from tmin (position 0) to tmax
// (position RL - 1), the reference's ladder T_b = tmin (tmax / tmin)^(b / 7)
// for RL = 8 (seeded.cu:493-494).
__device__ __forceinline__ float rung_temp(const JobDev& jd, int k) {
    const int RL = rungs_per_ladder(jd), pos = k % RL;
    const float lt = logf(jd.tmin), lh = logf(jd.tmax);
    return RL > 1 ? expf(lt + (lh - lt) * (float)pos / (float)(RL - 1)) : jd.tmin;
}

// Cooling factor of exchange round x under SQS_JOB_ADAPT: 0.002^((x mod 200)
// / 199), the reference's cool (seeded.cu:493); 1 otherwise.
__device__ __forceinline__ float cool_of(bool adaptive, int xround) {
    return adaptive ? powf(0.002f, (float)(xround % 200) / 199.f) : 1.f;
}

// Step scale of a replica on rung k under SQS_JOB_ADAPT: adaptation factor x
// (0.15 + 1.85 pos / (RL - 1)) x sqrt(cool), the reference's scale = adapt *
// baseMove * (.15 + 1.85 (b % 8) / 7) * sqrt(cool) (seeded.cu:506), in units
// of the job's sigma.
__device__ __forceinline__ float step_scale(const JobDev& jd, float adapt, int k, float cool) {
    const int RL = rungs_per_ladder(jd), pos = k % RL;
    return adapt * (RL > 1 ? 0.15f + 1.85f * (float)pos / (float)(RL - 1) : 1.f) * sqrtf(cool);
}

// Container side of rung k when the job's side is B: B itself, or under
// SQS_JOB_TARGETS the reference's target below the best,
// max(sqrt n + 1e-6, B (1 - shrink m(pos))) (seeded.cu:478-481, with the
// shrink relative to the side).
__device__ __forceinline__ float rung_side(const JobDev& jd, float B, int k) {
    if (!(jd.flags & kTargets)) return B;
    const int RL = rungs_per_ladder(jd);
    const float lb = sqrtf((float)jd.n) + 1e-6f;
    return fmaxf(lb, B * (1.f - jd.shrink * target_mult(k % RL, RL)));
}

struct CtaShared {
    JobDev jd;
    JobMut jm;
    float temps[kMaxR];
    long long wE[kMaxRl];      // this CTA's replica energies at a checkpoint
    double wL[kMaxRl];         // this CTA's candidate certified sides at a checkpoint
    double wlam[kMaxRl], wx0[kMaxRl], wy0[kMaxRl];
    float wside[kMaxRl];       // each replica's container side (per rung under SQS_JOB_TARGETS)
    int wbad[kMaxRl];          // cell-list overflow per warp
    int decision_win;          // global replica index of the new best (-1: none)
    int bad;                   // any overflow in the cluster
    int reset0;                // SQS_JOB_TARGETS: the gain resets every rung of ladder 0, not only heads
    float newL;
    long long red[kGrpSlots * kMaxRl];  // group sums: kGrpSlots values a warp
    long long qE;              // energy of the replica quenched by this CTA
    long long qEv[kMaxRl];     // each replica's energy before a group quench
    long long qEnew[kMaxRl];   // and after it
};

// MOVES: whether the move-set options (adaptation, collective moves, kicks)
// are compiled in; jobs without them run the leaner instance.
template <int V>
struct IntTag {
    static constexpr int value = V;
};

// A proposal's old and new cells, one byte per coordinate (grids are at most
// 64 / 1.59 < 256 wide).
__device__ __forceinline__ int pack_cells(int ox, int oy, int nx, int ny) {
    return ox | (oy << 8) | (nx << 16) | (ny << 24);
}
// Whether two cells (16 bits a coordinate) are the same or adjacent: each
// half of a + 0x8001 - b holds 0x8000 + difference + 1, without borrows, and
// the difference + 1 must be 0, 1 or 2.
__device__ __forceinline__ bool near_cells(unsigned a, unsigned b) {
    const unsigned d = (a + 0x80018001u - b) ^ 0x80008000u;
    return ((d & 0xfffcfffcu) | (d & (d >> 1) & 0x00010001u)) == 0u;
}
// Did the move of square mi (-1: none) between cells mc change what a
// proposal of square ik from cells ck read?
__device__ __forceinline__ bool touches(int mi, int mc, int ik, int ck) {
    const unsigned b = __byte_perm((unsigned)ck, 0u, 0x4140);
    const unsigned o = __byte_perm((unsigned)mc, 0u, 0x4140), n = __byte_perm((unsigned)mc, 0u, 0x4342);
    return mi >= 0 && (mi == ik || near_cells(o, b) || near_cells(n, b));
}

template <bool MOVES>
__global__ void __launch_bounds__(32 * kMaxRl) anneal_kernel(const int32_t* __restrict__ job_list,
                                                      const JobDev* __restrict__ jdev, JobMut* __restrict__ jmut,
                                                      float4* __restrict__ pos, double* __restrict__ best,
                                                      int slice_sweeps, int dyn_bytes) {
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ CtaShared S;
    extern __shared__ __align__(16) unsigned char dyn[];
    const int rank = (int)cluster.block_rank();
    const int job = job_list[blockIdx.x / cluster.num_blocks()];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) {
        S.jd = jdev[job];
        S.jm = jmut[job];
    }
    __syncthreads();
    const JobDev& jd = S.jd;
    if (S.jm.status != kRunning) return;  // identical in every CTA of the cluster
    const int n = jd.n, R = jd.R, Rl = jd.Rl;
    const int r = rank * Rl + w;  // global replica index of this warp
    const bool active = w < Rl;
    if (tid < R) S.temps[tid] = rung_temp(jd, tid);
    const int64_t rb = replica_smem_bytes(n, jd.Gmax);
    Rep rep = rep_view(dyn + (active ? w : 0) * rb, n, jd.Gmax);
    float L = S.jm.L;  // the job's side: every replica's, or under SQS_JOB_TARGETS the best the rung sides hang from
    Grid g = make_grid(L, jd.Gmax, jd.cell);
    // this replica's side (walls, move clamps, kicks, quench)
    float Lr = active ? rung_side(jd, L, S.jm.perm[r]) : L;
    if (active && lane == 0) S.wside[w] = Lr;
    const uint32_t k0 = (uint32_t)jd.seed, k1 = (uint32_t)(jd.seed >> 32);

    // load the replica
    if (active) {
        const float4* src = pos + jd.pos_off + (int64_t)r * n;
        for (int i = lane; i < n; i += 32) {
            const float4 p = src[i];
            float s, c;
            state_trig(p.z, &s, &c);
            rep.sq[i] = make_float4(p.x, p.y, c, s);
            rep.ang[i] = p.z;
        }
        __syncwarp();
        const bool ok = build_cells(rep, n, g, lane);
        if (lane == 0) S.wbad[w] = !ok;
    }
    __syncthreads();
    cluster.sync();
    if (tid == 0) {
        int bad = 0;
        for (int q = 0; q < (int)cluster.num_blocks(); ++q) {
            const CtaShared* o = cluster.map_shared_rank(&S, q);
            for (int k = 0; k < Rl; ++k) bad |= o->wbad[k];
        }
        S.bad = bad;
    }
    cluster.sync();
    if (S.bad) {
        if (rank == 0 && tid == 0) jmut[job].status = kErrCells;
        return;
    }
    long long E = 0;
    if (active) {
        E = S.jm.done == 0 ? full_energy(rep, n, g, Lr, lane) : S.jm.E[r];
    }
    // sums of a lane's share, added up at the end (Epart: at each checkpoint)
    unsigned accs = 0;
    int ovf = 0;
    long long Epart = 0;
    // move-set options: step adaptation with a cooling cycle of 200 exchange
    // rounds (temperatures x 0.002^(k/199), steps x its square root)
    const bool adaptive = MOVES && (jd.flags & kMoveAdapt) != 0;
    float adapt = (MOVES && active) ? S.jm.adapt[r] : 1.f;
    int win = (MOVES && active) ? S.jm.win[r] : 0;
    float cool = cool_of(adaptive, S.jm.xround);
    float invT = active ? 1.0f / (S.temps[S.jm.perm[r]] * cool) : 0.f;
    // this replica's scratch block (kQuenchScr n float4): in shared memory after
    // the replicas when the launch left room for every replica's, else in HBM;
    // between quenches it holds the undo copy of a collective move or kick and
    // the FP64 trig of the certified side
    const bool smem_scr = (int64_t)dyn_bytes >= (int64_t)Rl * (rb + (int64_t)sizeof(float4) * kQuenchScr * n);
    float4* scr_own = smem_scr ? reinterpret_cast<float4*>(dyn + (int64_t)Rl * rb) + (int64_t)(active ? w : 0) * kQuenchScr * n
                               : pos + jd.scr_off + (int64_t)r * kQuenchScr * n;

    // Proposals are numbered per replica across the whole job (a sweep is n
    // of them); checkpoints fall after every xprops proposals and at the end
    // of the budget; a slice ends after its sweeps' worth of proposals.
    const int64_t P_total = jd.props_total, xp = jd.xprops;
    int64_t p_at = S.jm.done;
    const int64_t p_end = min(P_total, p_at + (int64_t)(jd.slice > 0 ? jd.slice : slice_sweeps) * n);
    int npl = -1;  // pairs on the replica's pair list (collective moves; -1: none)
    while (p_at < p_end) {
        const int64_t next_cp = min(P_total, (p_at / xp + 1) * xp);
        const int64_t stop = min(next_cp, p_end);
        if (active) {
            const bool small = !MOVES && n <= 32;
            float4 own = make_float4(0.f, 0.f, 1.f, 0.f);
            int own_cell = -1;
            if (small && lane < n) {
                own = rep.sq[lane];
                own_cell = g.cx(own.y) * g.G + g.cx(own.x);
            }
            for (int64_t base = p_at; base < stop; base += 32) {
                // Lane l draws proposal base + l: two Philox blocks keyed by
                // (proposal index, replica, 0 / 1), Box-Muller for the centre
                // step and the angle step, the uniform of the Metropolis test.
                // Each proposal then broadcasts its draws.
                const int kn = (int)(stop - base < 32 ? stop - base : 32);
                int di = 0;
                float ddx = 0.f, ddy = 0.f, dda = 0.f, du = 0.f;
                if (lane < kn) {
                    const uint64_t ev = (uint64_t)(base + lane);
                    const U4 ra = philox4x32_10(U4{(uint32_t)ev, (uint32_t)(ev >> 32), (uint32_t)r, 0u}, k0, k1);
                    const U4 rb = philox4x32_10(U4{(uint32_t)ev, (uint32_t)(ev >> 32), (uint32_t)r, 1u}, k0, k1);
                    di = (int)(((uint64_t)ra.x * (uint64_t)n) >> 32);
                    if (adaptive) {
                        // the reference search's steps: uniform in +-sigma
                        // for each coordinate and the angle (seeded.cu:508-510)
                        ddx = jd.sigma_xy * (2.f * u01(ra.y) - 1.f);
                        ddy = jd.sigma_xy * (2.f * u01(ra.z) - 1.f);
                        dda = jd.sigma_a * (2.f * u01(ra.w) - 1.f);
                    } else {
                        const float rad1 = sqrtf(-2.f * __logf(u01(ra.y)));
                        float sn1, cs1;
                        __sincosf(6.2831853f * u01(ra.z), &sn1, &cs1);
                        const float rad2 = sqrtf(-2.f * __logf(u01(ra.w)));
                        const float n2 = rad2 * __cosf(6.2831853f * u01(rb.x));
                        ddx = jd.sigma_xy * rad1 * cs1;
                        ddy = jd.sigma_xy * rad1 * sn1;
                        dda = jd.sigma_a * n2;
                    }
                    du = u01(rb.y);
                    if (MOVES && (jd.flags & kMoveCollective)) di |= (int)(rb.z % 7u) << 16;  // move mode
                }
                // one lane moves square i to its new state and cell
                auto apply_move = [&](int i, float nx, float ny, float nc, float ns, float na, int oc, int ncell) {
                    rep.sq[i] = make_float4(nx, ny, nc, ns);
                    rep.ang[i] = na;
                    if (oc != ncell) {
                        const int m = rep.cnt[oc];
                        for (int t = 0; t < m; ++t) {
                            if (rep.slot[oc * kCellK + t] == (uint16_t)i) {
                                rep.slot[oc * kCellK + t] = rep.slot[oc * kCellK + m - 1];
                                break;
                            }
                        }
                        rep.cnt[oc] = (uint8_t)(m - 1);
                        rep.slot[ncell * kCellK + rep.cnt[ncell]] = (uint16_t)i;
                        rep.cnt[ncell] = (uint8_t)(rep.cnt[ncell] + 1);
                    }
                };
                // A lane's own proposal against the current state: the trial
                // position and trig, the wall energy's change, and the old and
                // new cells.  It depends on the proposal's square alone, so
                // without move-set options (whose step scale follows the
                // acceptance before) all 32 are formed at once, a lane each,
                // and a proposal only broadcasts its own; `stale` marks a lane
                // whose square has moved since, which forms its trial again
                // when its turn comes.  A group of four proposals used to form
                // its trials with eight lanes each repeating the work.
                float tx = 0.f, ty = 0.f, tc = 1.f, ts = 0.f, ta = 0.f;
                long long tw = 0;
                int tcells = 0;
                bool stale = false;
                auto form_trial = [&](float dx, float dy, float da) {
                    const int i = di & 0xffff;
                    const float4 P = rep.sq[i];
                    // keep centres in [0.5, Lr - 0.5] without ever moving a square
                    // further than the clamped step (it may start outside)
                    tx = fminf(fmaxf(P.x, Lr - 0.5f), fmaxf(fminf(P.x, 0.5f), P.x + dx));
                    ty = fminf(fmaxf(P.y, Lr - 0.5f), fmaxf(fminf(P.y, 0.5f), P.y + dy));
                    ta = wrap_quarter_f(__fadd_rn(rep.ang[i], da));
                    state_trig(ta, &ts, &tc);
                    tw = qe(wall_e(tx, ty, tc, ts, Lr)) - qe(wall_e(P.x, P.y, P.z, P.w, Lr));
                    tcells = pack_cells(g.cx(P.x), g.cx(P.y), g.cx(tx), g.cx(ty));
                };
                auto form_plain = [&]() {
                    form_trial(fminf(kMaxStep, fmaxf(-kMaxStep, ddx)), fminf(kMaxStep, fmaxf(-kMaxStep, ddy)), dda);
                };
                if (!MOVES) form_plain();
                // proposal q of this batch, evaluated by the whole warp
                auto single = [&](int q) {
                    const int dpk = __shfl_sync(0xffffffffu, di, q);
                    const int i = dpk & 0xffff, mode = dpk >> 16;
                    const float u_acc = __shfl_sync(0xffffffffu, du, q);
                    const uint64_t pidx = (uint64_t)(base + q);
                    bool acc;
                    float dx = 0.f, dy = 0.f, da = 0.f;
                    if (MOVES) {
                        float sc = 1.f;  // step scale (adaptive moves)
                        if (adaptive) {
                            sc = step_scale(jd, adapt, S.jm.perm[r], cool);
                            if ((pidx & 15u) == 0) sc *= 3.5f;
                        }
                        dx = fminf(kMaxStep, fmaxf(-kMaxStep, __shfl_sync(0xffffffffu, ddx, q) * sc));
                        dy = fminf(kMaxStep, fmaxf(-kMaxStep, __shfl_sync(0xffffffffu, ddy, q) * sc));
                        da = __shfl_sync(0xffffffffu, dda, q) * sc;
                    }
                    if (MOVES && mode != 0) {
                        acc = collective_move(rep, g, n, Lr, lane, mode, i, dx, dy, da, u_acc, invT, E, scr_own, npl,
                                              lane == 0, &ovf);
                        if (lane == 0) accs += acc;
                    } else {
                        if (MOVES) {
                            if (lane == q) form_trial(dx, dy, da);
                        } else if (__shfl_sync(0xffffffffu, (int)stale, q)) {
                            if (stale) form_plain();
                            stale = false;
                        }
                        const float nx = __shfl_sync(0xffffffffu, tx, q), ny = __shfl_sync(0xffffffffu, ty, q);
                        const float nc = __shfl_sync(0xffffffffu, tc, q), ns = __shfl_sync(0xffffffffu, ts, q);
                        const int cells = __shfl_sync(0xffffffffu, tcells, q);
                        const int ocx = cells & 0xff, ocy = (cells >> 8) & 0xff, ncx = (cells >> 16) & 0xff,
                                  ncy = (int)((unsigned)cells >> 24);
                        const float4 P = rep.sq[i];
                        long long dq = lane == q ? tw : 0;
                        for_block<32>(rep, g, ocx, ocy, lane, [&](int j) {
                            const long long d = pair_delta(rep.sq[j], nx, ny, nc, ns, P);
                            dq += j != i ? d : 0;
                        });
                        dq = warp_sum_dq(dq);
                        const float de = (float)dq * (1.0f / kEScale);
                        acc = dq <= 0 || u_acc < __expf(-de * invT);
                        const int oc = ocy * g.G + ocx, ncell = ncy * g.G + ncx;
                        if (acc && oc != ncell && rep.cnt[ncell] >= kCellK) {
                            acc = false;
                            if (lane == 0) ++ovf;
                        }
                        if (acc) {
                            if (lane == 0) ++accs;
                            if (MOVES) E += dq;
                            else if (lane == 0) Epart += dq;
                            if (lane == q) apply_move(i, tx, ty, tc, ts, ta, oc, ncell);
                            stale |= (di & 0xffff) == i;
                            if (MOVES && npl >= 0) {  // out of the pair list's reach?
                                const float2 o = reinterpret_cast<const float2*>(scr_own + 3 * n)[i];
                                if (!(fabsf(nx - o.x) <= kListStep && fabsf(ny - o.y) <= kListStep)) npl = -1;
                            }
                        }
                    }
                    if (adaptive) {  // every 16 proposals: steer toward 25% acceptance
                        win += acc;
                        if (((pidx + 1u) & 15u) == 0) {
                            adapt = fmaxf(0.1f, fminf(4.0f, adapt * expf(((float)win / 16.f - 0.25f) * 0.5f)));
                            win = 0;
                        }
                    }
                    __syncwarp();
                };
                // Proposals q .. q + M - 1 evaluated at once, one per group of
                // 32 / M lanes, all against the current state.  A proposal's
                // result stands unless an earlier move of the group that was
                // accepted touched what it read: the same square, or an old or
                // new cell of that move inside its 3x3 block (cells are wider
                // than a step, so a move changes a square's cell by at most one;
                // every other read -- counts and slots of the block, squares in
                // it, the count of its target cell -- lies in that block).  The
                // proposals before the first that was touched are settled: their
                // accepted moves lie in distinct cells, and each proposal's own
                // lane applies its move at the same time; the next group starts
                // at the touched one.  Energies are exact and order-free, so the
                // trajectory is the one-at-a-time trajectory, bit for bit.
                // Energy, acceptances and overflows are summed a lane each and
                // added up after the batch.  Returns the proposals settled.
                auto group = [&](int q, auto mtag) -> int {
                    constexpr int M = decltype(mtag)::value, W = 32 / M;
                    const int grp = lane / W, gl = lane % W;
                    const int qs = q + grp;
                    if (__any_sync(0xffffffffu, stale && lane >= q && lane < q + M)) {
                        if (stale) form_plain();
                        stale = false;
                    }
                    const int i = __shfl_sync(0xffffffffu, di, qs);
                    const float nx = __shfl_sync(0xffffffffu, tx, qs), ny = __shfl_sync(0xffffffffu, ty, qs);
                    const float nc = __shfl_sync(0xffffffffu, tc, qs), ns = __shfl_sync(0xffffffffu, ts, qs);
                    const int cells = __shfl_sync(0xffffffffu, tcells, qs);
                    const float u_acc = __shfl_sync(0xffffffffu, du, qs);
                    const int ocx = cells & 0xff, ocy = (cells >> 8) & 0xff, ncx = (cells >> 16) & 0xff,
                              ncy = (int)((unsigned)cells >> 24);
                    const float4 P = rep.sq[i];
                    long long dq = 0;
                    for_block<W>(rep, g, ocx, ocy, gl, [&](int j) {
                        const long long d = pair_delta(rep.sq[j], nx, ny, nc, ns, P);
                        dq += j != i ? d : 0;
                    });
                    // exact sum over the group's lanes: hi * 2^20 + lo parts
                    // (a lane's term is below 2^46, so both parts stay in 32 bits)
                    int hi = (int)(dq >> 20);
                    unsigned lo = (unsigned)(dq & 0xFFFFF);
#pragma unroll
                    for (int off = W / 2; off > 0; off >>= 1) {
                        hi += __shfl_xor_sync(0xffffffffu, hi, off);
                        lo += __shfl_xor_sync(0xffffffffu, lo, off);
                    }
                    const unsigned wlo = __shfl_sync(0xffffffffu, (unsigned)(unsigned long long)tw, qs);
                    const int whi = __shfl_sync(0xffffffffu, (int)(tw >> 32), qs);
                    const long long mine = (long long)hi * 1048576ll + (long long)lo +
                                           (long long)(((unsigned long long)(unsigned)whi << 32) | wlo);
                    const float de = (float)mine * (1.0f / kEScale);
                    bool acc = mine <= 0 || u_acc < __expf(-de * invT), full = false;
                    if (acc && ((cells ^ (cells >> 16)) & 0xffff)) {  // a new cell: has it room?
                        full = rep.cnt[ncy * g.G + ncx] >= kCellK;
                        acc = !full;
                    }
                    unsigned am = __ballot_sync(0xffffffffu, acc && gl == 0);
                    if (am == 0u) {  // nothing moves
                        ovf += full && gl == 0;
                        __syncwarp();
                        return M;
                    }
                    // does an accepted move of an earlier proposal touch this one?
                    const int mv_i = acc ? i : -1;
                    bool hit = false;
#pragma unroll
                    for (int d = 1; d < M; ++d) {
                        const int oi = __shfl_up_sync(0xffffffffu, mv_i, d * W);
                        const int ocl = __shfl_up_sync(0xffffffffu, cells, d * W);
                        hit |= grp >= d && touches(oi, ocl, i, cells);
                    }
                    const unsigned hm = __ballot_sync(0xffffffffu, hit);
                    const int take = hm ? (__ffs(hm) - 1) / W : M;  // (the first proposal is never touched)
                    if (gl == 0 && grp < take) {
                        if (acc) {
                            Epart += mine;
                            ++accs;
                        }
                        ovf += full;
                    }
                    if (take < M) am &= (1u << (take * W)) - 1u;
                    if (lane >= q && lane < q + take && (am >> ((lane - q) * W) & 1u))
                        apply_move(di, tx, ty, tc, ts, ta, ((tcells >> 8) & 0xff) * g.G + (tcells & 0xff),
                                   (int)((unsigned)tcells >> 24) * g.G + ((tcells >> 16) & 0xff));
#pragma unroll
                    for (int k = 0; k < M; ++k) stale |= (am >> (k * W) & 1u) && di == __shfl_sync(0xffffffffu, i, k * W);
                    __syncwarp();
                    return take;
                };
                // A replica of up to 32 squares without move-set options holds
                // square `lane` in registers and tests a proposal against every
                // other square, a lane each, cell lists aside: pairs outside the
                // cut-off add zero, so the change is the same, and the chain of
                // dependent loads (counts, slot, square) is gone.  A cell's
                // count, for the capacity rule, is a ballot.
                auto tiny = [&](int q) {
                    const int i = __shfl_sync(0xffffffffu, di, q);
                    if (__shfl_sync(0xffffffffu, (int)stale, q)) {
                        if (stale) form_plain();
                        stale = false;
                    }
                    const float nx = __shfl_sync(0xffffffffu, tx, q), ny = __shfl_sync(0xffffffffu, ty, q);
                    const float nc = __shfl_sync(0xffffffffu, tc, q), ns = __shfl_sync(0xffffffffu, ts, q);
                    const float u_acc = __shfl_sync(0xffffffffu, du, q);
                    const float4 P = rep.sq[i];
                    const long long d = pair_delta(own, nx, ny, nc, ns, P);
                    const long long dq = warp_sum_dq((lane != i && lane < n ? d : 0) + (lane == q ? tw : 0));
                    const bool acc = dq <= 0 || u_acc < __expf(-((float)dq * (1.0f / kEScale)) * invT);
                    if (!acc) return;
                    if (n > kCellK) {
                        const int cells = __shfl_sync(0xffffffffu, tcells, q);
                        const int ncell = (int)((unsigned)cells >> 24) * g.G + ((cells >> 16) & 0xff);
                        const int there = __popc(__ballot_sync(0xffffffffu, own_cell == ncell));
                        if (ncell != ((cells >> 8) & 0xff) * g.G + (cells & 0xff) && there >= kCellK) {
                            if (lane == 0) ++ovf;
                            return;
                        }
                        if (lane == i) own_cell = ncell;
                    }
                    if (lane == 0) {
                        ++accs;
                        Epart += dq;
                    }
                    if (lane == i) own = make_float4(nx, ny, nc, ns);
                    if (lane == q) {
                        rep.sq[i] = make_float4(nx, ny, nc, ns);
                        rep.ang[i] = ta;
                    }
                    stale |= di == i;
                    __syncwarp();
                };
                // groups need room: on small grids most proposals would be
                // evaluated twice (fours from G = 6 on against 8: 16 replicas of
                // n = 120 take 14.2 against 15.1 ms, n = 60 is the same); the
                // move-set instance keeps one at a time (its step scale follows
                // the acceptance of the previous move)
                const bool fours = !MOVES && g.G >= 6, twos = !MOVES && g.G >= 4;
                for (int q = 0; q < kn;) {
                    if (small) {
                        tiny(q);
                        ++q;
                    } else if (fours && q + 3 < kn) {
                        q += group(q, IntTag<4>{});
                    } else if (twos && q + 1 < kn) {
                        q += group(q, IntTag<2>{});
                    } else {
                        single(q);
                        ++q;
                    }
                }
                if (accs >= kCountFlush) {
                    atomicAdd(reinterpret_cast<unsigned long long*>(&jmut[job].accepted), (unsigned long long)accs);
                    accs = 0;
                }
            }
            if (small) build_cells(rep, n, g, lane);  // every cell within its capacity
            if (!MOVES) {
                E += warp_sum_ll(Epart);
                Epart = 0;
            }
        }
        p_at = stop;
        // ---- checkpoint: best-state search, shrink, replica exchange.  Only
        // after every xprops proposals (and at the end of the budget), so a
        // job's trajectory does not depend on how it is sliced.
        if (p_at != next_cp) break;  // the slice ends between checkpoints
        const bool xpoint = p_at % xp == 0;
        npl = -1;
        if (MOVES && (jd.flags & kMoveQuenchAll) && jd.quench_iters > 0) {
            // every replica at once, each by its own group of gw warps (the
            // launch gives each replica gw = blockDim / (32 Rl) warps); the
            // scratch (kQuenchScr n float4 a replica) in shared memory after
            // the replicas when the launch left room for all of them, else
            // the replica's own block of the job's scratch in HBM
            const int gw = (int)(blockDim.x >> 5) / Rl, q = w / gw;
            float4* qw = smem_scr ? reinterpret_cast<float4*>(dyn + (int64_t)Rl * rb) + (int64_t)q * kQuenchScr * n
                                  : pos + jd.scr_off + ((int64_t)rank * Rl + q) * kQuenchScr * n;
            if (gw == 1) {
                if (active) E = quench_grp(WarpGrp{lane}, rep, n, g, Lr, jd.quench_iters, jd.quench_stall, qw, E);
            } else {
                if (active && lane == 0) S.qEv[w] = E;
                __syncthreads();
                if (q < Rl) {
                    const Rep cr = rep_view(dyn + q * rb, n, jd.Gmax);
                    const long long e0 = S.qEv[q];
                    __syncwarp();
                    const long long e = quench_group(1 + q, gw, q * gw * 32, S.red + kGrpSlots * q * gw, cr, n, g,
                                                     S.wside[q], jd.quench_iters, jd.quench_stall, qw, e0);
                    if (tid == q * gw * 32) S.qEnew[q] = e;
                }
                __syncthreads();
                if (active) E = S.qEnew[w];
            }
            __syncthreads();
        } else {
            // the replica on the coldest rung, by warps of the CTA that holds it;
            // its scratch in shared memory after the replicas when the launch left
            // room, else its first replica's block of the job's scratch (the other
            // CTAs' replicas may be using theirs)
            float4* qs = (int64_t)dyn_bytes >= (int64_t)Rl * rb + (int64_t)sizeof(float4) * kQuenchScr * n
                             ? reinterpret_cast<float4*>(dyn + (int64_t)Rl * rb)
                             : pos + jd.scr_off + (int64_t)rank * Rl * kQuenchScr * n;
            int cold = 0;
            for (int q = 0; q < R; ++q)
                if (S.jm.perm[q] == 0) cold = q;
            if (jd.quench_iters > 0 && cold / Rl == rank) {
                if (w == cold % Rl && lane == 0) S.qE = E;
                __syncthreads();
                const Rep cr = rep_view(dyn + (cold % Rl) * rb, n, jd.Gmax);
                const long long e = quench_group(1, (int)(blockDim.x >> 5), 0, S.red, cr, n, g, S.wside[cold % Rl],
                                                 jd.quench_iters, jd.quench_stall, qs, S.qE);
                if (tid == 0) S.qEnew[0] = e;
                __syncthreads();
                if (w == cold % Rl) E = S.qEnew[0];
            }
        }
        if (active) {
            double Lc = 1e30, lam = 0, x0 = 0, y0 = 0;
            // any state whose overlaps a dilation of at most 0.8% removes is a
            // certified candidate (penetrations of depth d cost about d^2 each,
            // so the energy gate skips states that cannot pass); under
            // SQS_JOB_CERT_ALL every replica is measured, as the reference
            // search measures every chain after its polish (seeded.cu:716)
            if (E < qe(1e-4f) || (jd.flags & kCertAll))
                Lc = cert_side(rep, n, g, lane, reinterpret_cast<double2*>(scr_own), lam, x0, y0);
            if (lane == 0) {
                S.wE[w] = E;
                S.wL[w] = Lc;
                S.wlam[w] = lam;
                S.wx0[w] = x0;
                S.wy0[w] = y0;
            }
        }
        __syncthreads();
        cluster.sync();
        if (tid == 0) {
            // every CTA takes the same decisions from the same gathered values
            long long Eall[kMaxR];
            // under SQS_JOB_TARGETS only a side below the initial one counts, as
            // the reference's chain bests start at the seed's side (seeded.cu:883)
            const double best0 = (jd.flags & kTargets) ? fmin(S.jm.best_L, (double)jd.L0) : S.jm.best_L;
            double bestc = best0;
            int win = -1;
            for (int q = 0; q < (int)cluster.num_blocks(); ++q) {
                const CtaShared* o = cluster.map_shared_rank(&S, q);
                for (int k = 0; k < Rl; ++k) {
                    Eall[q * Rl + k] = o->wE[k];
                    if (o->wL[k] < bestc) {
                        bestc = o->wL[k];
                        win = q * Rl + k;
                    }
                }
            }
            S.decision_win = win;
            S.newL = L;
            S.reset0 = 0;
            const bool targets = (jd.flags & kTargets) != 0;
            if (win >= 0) {
                const double gain = best0 < 1e29 ? best0 - bestc : 0.0;
                S.jm.best_L = bestc;
                S.jm.improvements += 1;
                const float lb = sqrtf((float)n) + 1e-6f;
                // the job's side: the new best (the rung targets hang below it), or
                // the best shrunk by the job's factor
                float nl = targets ? (float)fmin((double)L, bestc)
                                   : (float)(fmin((double)L, bestc) * (1.0 - (double)jd.shrink));
                if (nl < lb) nl = lb;
                if (nl < L) {
                    S.newL = nl;
                    S.jm.shrinks += 1;
                }
                // a large gain resets every rung of ladder 0 to the new best (seeded.cu:929)
                S.reset0 = targets && gain > 5e-4;
            }
            // replica exchange between neighbouring rungs of each ladder, alternating
            // parity; under SQS_JOB_TARGETS only in rounds without a new best, as the
            // reference swaps only in epochs that did not improve (seeded.cu:939-941)
            if (xpoint && !(targets && win >= 0)) {
                int holder[kMaxR];
                for (int q = 0; q < R; ++q) holder[S.jm.perm[q]] = q;
                const int par = S.jm.xround & 1;
                const int RL = rungs_per_ladder(jd);
                for (int k = 0; k + 1 < R; ++k) {
                    const int pos = k % RL;
                    if ((pos & 1) != par || pos + 1 >= RL) continue;
                    const int a = holder[k], b = holder[k + 1];
                    const U4 u = philox4x32_10(U4{(uint32_t)S.jm.xround, (uint32_t)k, 0u, 0x7fffffffu}, k0, k1);
                    const float d = (1.0f / S.temps[k] - 1.0f / S.temps[k + 1]) *
                                    ((float)(Eall[a] - Eall[b]) * (1.0f / kEScale)) / cool;
                    S.jm.xatt += 1;
                    if (d >= 0.f || u01(u.x) < expf(d)) {
                        S.jm.xacc += 1;
                        S.jm.perm[a] = k + 1;
                        S.jm.perm[b] = k;
                        holder[k] = b;
                        holder[k + 1] = a;
                    }
                }
            }
            if (xpoint) S.jm.xround += 1;
        }
        cluster.sync();
        __syncthreads();
        if (adaptive) cool = cool_of(true, S.jm.xround);
        const bool targets = MOVES && (jd.flags & kTargets) != 0;
        if (active) {
            invT = 1.0f / (S.temps[S.jm.perm[r]] * cool);
            if (S.decision_win == r) {
                // new best: dilated, translated to the origin, angles in [0, pi/2)
                double* dst = best + jd.best_off;
                const double lam = S.wlam[w], x0 = S.wx0[w], y0 = S.wy0[w];
                for (int i = lane; i < n; i += 32) {
                    dst[3 * i] = __dsub_rn(__dmul_rn((double)rep.sq[i].x, lam), x0);
                    dst[3 * i + 1] = __dsub_rn(__dmul_rn((double)rep.sq[i].y, lam), y0);
                    dst[3 * i + 2] = (double)rep.ang[i];
                }
            }
        }
        if (targets && S.decision_win >= 0) {  // the new best is read by the ladder heads below
            __threadfence();
            __syncthreads();
            cluster.sync();
        }
        const bool regrid = S.newL < L;
        if (regrid || targets) {
            const float f = S.newL / L;
            if (regrid) {
                L = S.newL;
                g = make_grid(L, jd.Gmax, jd.cell);
            }
            if (active) {
                const int rung = S.jm.perm[r];
                const float Ln = rung_side(jd, L, rung);
                const int RL = rungs_per_ladder(jd);
                const bool reset = targets && S.decision_win >= 0 && (rung % RL == 0 || (S.reset0 && rung < RL));
                if (reset) {
                    // ladder head: the new best, scaled into its own side (seeded.cu:928-936)
                    const double* src = best + jd.best_off;
                    const double sc = (double)Ln / (double)L;
                    for (int i = lane; i < n; i += 32) {
                        const float a = (float)src[3 * i + 2];
                        float sn, cs;
                        state_trig(a, &sn, &cs);
                        rep.sq[i] = make_float4((float)(src[3 * i] * sc), (float)(src[3 * i + 1] * sc), cs, sn);
                        rep.ang[i] = a;
                    }
                } else if (regrid && !targets) {
                    for (int i = lane; i < n; i += 32) {
                        rep.sq[i].x *= f;
                        rep.sq[i].y *= f;
                    }
                }
                __syncwarp();
                if (reset || regrid) {
                    const bool ok = build_cells(rep, n, g, lane);
                    if (lane == 0) S.wbad[w] = !ok;
                }
                const bool changed = reset || regrid || Ln != Lr;
                Lr = Ln;
                if (lane == 0) S.wside[w] = Lr;
                if (changed) E = full_energy(rep, n, g, Lr, lane);
            }
            if (regrid || (targets && S.decision_win >= 0)) {
                __syncthreads();
                cluster.sync();
                if (tid == 0) {
                    int bad = 0;
                    for (int q = 0; q < (int)cluster.num_blocks(); ++q) {
                        const CtaShared* o = cluster.map_shared_rank(&S, q);
                        for (int k = 0; k < Rl; ++k) bad |= o->wbad[k];
                    }
                    S.bad = bad;
                }
                cluster.sync();
                if (S.bad) {
                    if (rank == 0 && tid == 0) jmut[job].status = kErrCells;
                    return;
                }
            }
            __syncthreads();
        }
        // overlapped replicas are kicked (the round just completed decides
        // whether the worst square is also moved)
        if (MOVES && active && (jd.flags & kMoveKick) && E > qe(1e-12f))
            E = kick_replica(rep, g, n, Lr, lane, r, S.jm.xround, k0, k1, E, scr_own);
    }

    // ---- write the slice back
    if (active) {
        const long long accs_all = warp_sum_ll((long long)accs);
        const int ovf_all = __reduce_add_sync(0xffffffffu, ovf);
        float4* dst = pos + jd.pos_off + (int64_t)r * n;
        for (int i = lane; i < n; i += 32) dst[i] = make_float4(rep.sq[i].x, rep.sq[i].y, rep.ang[i], 0.f);
        if (lane == 0) {
            jmut[job].E[r] = E;
            if (MOVES) {
                jmut[job].adapt[r] = adapt;
                jmut[job].win[r] = win;
            }
            atomicAdd(reinterpret_cast<unsigned long long*>(&jmut[job].proposals), (unsigned long long)(p_at - S.jm.done));
            atomicAdd(reinterpret_cast<unsigned long long*>(&jmut[job].accepted), (unsigned long long)accs_all);
            if (ovf_all) atomicAdd(&jmut[job].overflows, ovf_all);
        }
    }
    if (rank == 0 && tid == 0) {
        JobMut& m = jmut[job];
        m.L = L;
        m.done = p_end;
        m.xround = S.jm.xround;
        m.status = p_end >= P_total ? kFinished : kRunning;
        m.shrinks = S.jm.shrinks;
        m.improvements = S.jm.improvements;
        m.best_L = S.jm.best_L;
        m.xatt = S.jm.xatt;
        m.xacc = S.jm.xacc;
        for (int q = 0; q < R; ++q) m.perm[q] = S.jm.perm[q];
    }
}

// Replica states of a batch call from the start states it uploads: angles
// wrapped to [0, pi/2) in double first, init_replicas bit for bit (fmod is
// exact).  kInitCtas CTAs a job.  The call uploads one n x 3 start a job (or
// one a replica when the caller gives them) and nothing else: expanding and
// zeroing every job's whole region on the host, replicas and quench scratch
// (which nothing reads before it is written), and uploading that took 92 ms
// of the 144 ms of a call of 256 jobs of n 20..400 x 32 replicas (52 ms now).
constexpr int kInitCtas = 8;
__global__ void __launch_bounds__(256) init_states_kernel(const InitRec* __restrict__ rec,
                                                          const double* __restrict__ start, float4* __restrict__ pos) {
    const InitRec r = rec[blockIdx.x / kInitCtas];
    const int total = r.R * r.n;
    const double* src = start + r.src;
    float4* dst = pos + r.dst;
    const double q = 1.57079632679489661923;
    for (int k = (blockIdx.x % kInitCtas) * blockDim.x + threadIdx.x; k < total; k += kInitCtas * blockDim.x) {
        const double* p = src + 3 * (r.states > 1 ? k : k % r.n);
        double a = fmod(p[2], q);
        if (a < 0.0) a += q;
        dst[k] = make_float4((float)p[0], (float)p[1], (float)a, 0.f);
    }
}

int launch_init(cudaStream_t stream, int njobs, const InitRec* rec, const double* start, float4* pos) {
    if (njobs <= 0) return SQS_OK;
    init_states_kernel<<<(unsigned)njobs * kInitCtas, 256, 0, stream>>>(rec, start, pos);
    SQS_CUDA(cudaGetLastError());
    return SQS_OK;
}

// Final state of every replica, read back by sqs_anneal_batch_trace: one
// warp per (job, replica) loads the replica as the annealer left it, rebuilds
// its cell list on the job's grid and recomputes, with the annealer's own
// device functions, its fixed-point energy from scratch (equal, bit for bit,
// to the running energy the proposals kept when nothing drifts) and its FP64
// dilation-certified side, and reports the temperature and step scale its
// next proposal would use.
__global__ void __launch_bounds__(32) trace_kernel(const int2* __restrict__ items, const JobDev* __restrict__ jdev,
                                                   const JobMut* __restrict__ jmut, float4* __restrict__ pos,
                                                   TraceRec* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char dyn[];
    const int2 it = items[blockIdx.x];
    const JobDev& jd = jdev[it.x];
    const JobMut& jm = jmut[it.x];
    const int n = jd.n, r = it.y, lane = threadIdx.x;
    const Rep rep = rep_view(dyn, n, jd.Gmax);
    const Grid g = make_grid(jm.L, jd.Gmax, jd.cell);
    const float L = rung_side(jd, jm.L, jm.perm[r]);
    const float4* src = pos + jd.pos_off + (int64_t)r * n;
    for (int i = lane; i < n; i += 32) {
        const float4 p = src[i];
        float sn, cs;
        state_trig(p.z, &sn, &cs);
        rep.sq[i] = make_float4(p.x, p.y, cs, sn);
        rep.ang[i] = p.z;
    }
    __syncwarp();
    const bool ok = build_cells(rep, n, g, lane);
    const long long E = full_energy(rep, n, g, L, lane);
    double lam = 0, x0 = 0, y0 = 0;
    const double Lc = cert_side(rep, n, g, lane, reinterpret_cast<double2*>(pos + jd.scr_off + (int64_t)r * kQuenchScr * n), lam,
                                x0, y0);
    if (lane == 0) {
        const bool adaptive = (jd.flags & kMoveAdapt) != 0;
        const float cool = cool_of(adaptive, jm.xround);
        const int rung = jm.perm[r];
        TraceRec t;
        t.E_full = E;
        t.L_cert = Lc;
        t.lam = lam;
        t.temp = rung_temp(jd, rung) * cool;
        t.step = adaptive ? step_scale(jd, jm.adapt[r], rung, cool) : 1.f;
        t.side = L;
        t.rung = rung;
        t.cells_ok = ok ? 1 : 0;
        t.pad = 0;
        out[blockIdx.x] = t;
    }
}

int launch_trace(cudaStream_t stream, int items, const int2* list, const JobDev* jdev, const JobMut* jmut,
                 float4* pos, TraceRec* out, size_t smem) {
    static bool attr_done[64] = {false};
    int dev = 0;
    SQS_CUDA(cudaGetDevice(&dev));
    if (!attr_done[dev & 63]) {
        SQS_CUDA(cudaFuncSetAttribute(trace_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAnnealSmemLimit));
        attr_done[dev & 63] = true;
    }
    if (items <= 0) return SQS_OK;
    trace_kernel<<<items, 32, smem, stream>>>(list, jdev, jmut, pos, out);
    SQS_CUDA(cudaGetLastError());
    return SQS_OK;
}

// Kernel attributes (dynamic shared memory up to the opt-in limit,
// non-portable cluster sizes), once per device; call before any capture.
int prime_anneal() {
    static bool attr_done[64] = {false};
    int dev = 0;
    SQS_CUDA(cudaGetDevice(&dev));
    if (!attr_done[dev & 63]) {
        for (int v = 0; v < 2; ++v) {
            const void* fn = v ? (const void*)anneal_kernel<true> : (const void*)anneal_kernel<false>;
            cudaFuncAttributes fa;
            SQS_CUDA(cudaFuncGetAttributes(&fa, fn));
            SQS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          232448 - (int)fa.sharedSizeBytes));
            SQS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        }
        attr_done[dev & 63] = true;
    }
    return SQS_OK;
}

static cudaLaunchConfig_t anneal_config(int clusters, int cs, int Rl, size_t smem, cudaStream_t stream,
                                        cudaLaunchAttribute* attr, int gw = 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * cs), 1, 1);
    cfg.blockDim = dim3((unsigned)(Rl * 32 * gw), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Clusters of this shape (gw warps a replica) that can be resident at once
// (one wave), memoized per device and shape.
static int max_clusters_gw(int cs, int Rl, size_t smem, bool moves, int gw, int* out) {
    static std::mutex mu;
    static std::map<std::tuple<int, int, int, size_t, bool, int>, int> memo;
    int dev = 0;
    SQS_CUDA(cudaGetDevice(&dev));
    const auto key = std::make_tuple(dev, cs, Rl, smem, moves, gw);
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = memo.find(key);
        if (it != memo.end()) {
            *out = it->second;
            return SQS_OK;
        }
    }
    if (int r = prime_anneal()) return r;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = anneal_config(1, cs, Rl, smem, nullptr, attr, gw);
    int num = 0;
    if (moves) SQS_CUDA(cudaOccupancyMaxActiveClusters(&num, anneal_kernel<true>, &cfg));
    else SQS_CUDA(cudaOccupancyMaxActiveClusters(&num, anneal_kernel<false>, &cfg));
    std::lock_guard<std::mutex> lk(mu);
    memo[key] = num;
    *out = num;
    return SQS_OK;
}

int anneal_max_clusters(int cs, int Rl, size_t smem, bool moves, int* out) {
    return max_clusters_gw(cs, Rl, smem, moves, 1, out);
}

// Warps a replica for a launch of njobs clusters: the most, up to
// kMaxRl / Rl, that keep as many of the launch's clusters resident at once.
// The extra warps idle while their CTA anneals and join the checkpoint quench
// (same results: the quench's sums are integers), be it of every replica
// (SQS_JOB_QUENCH_ALL) or of the coldest: with 4 replicas a CTA the quench of
// n = 200 went from 4 to 13 warps and 100 sweeps from 12.5 to 11.4 ms.
static int quench_warps(int njobs, int cs, int Rl, size_t smem, bool moves) {
    if (Rl >= kMaxRl) return 1;
    int base = 0;
    if (max_clusters_gw(cs, Rl, smem, moves, 1, &base) != SQS_OK) return 1;
    const int need = std::min(njobs, base);
    for (int gw = kMaxRl / Rl; gw > 1; gw /= 2) {
        int m = 0;
        if (max_clusters_gw(cs, Rl, smem, moves, gw, &m) == SQS_OK && m >= need) return gw;
    }
    return 1;
}

int launch_anneal(cudaStream_t stream, int njobs, int cs, int Rl, size_t smem, bool moves, const int32_t* job_list,
                  const JobDev* jdev, JobMut* jmut, float4* pos, double* best, int slice) {
    if (int r = prime_anneal()) return r;
    cudaLaunchAttribute attr[1];
    const int gw = quench_warps(njobs, cs, Rl, smem, moves);
    const cudaLaunchConfig_t cfg = anneal_config(njobs, cs, Rl, smem, stream, attr, gw);
    if (moves) SQS_CUDA(cudaLaunchKernelEx(&cfg, anneal_kernel<true>, job_list, jdev, jmut, pos, best, slice, (int)smem));
    else SQS_CUDA(cudaLaunchKernelEx(&cfg, anneal_kernel<false>, job_list, jdev, jmut, pos, best, slice, (int)smem));
    return SQS_OK;
}

// Shared memory of a launch whose largest job needs rb bytes a replica and
// has n_max squares: the replicas, plus room for the checkpoint quench's
// scratch (kQuenchScr n float4 per quench) when that fits and keeps as many
// clusters resident -- the quench then runs on shared instead of global
// memory (same results).  Launches with the move-set options first try room
// for every replica's quench (SQS_JOB_QUENCH_ALL quenches them all at once),
// then for one.  `need` is how many clusters the launch must keep resident:
// a size is taken when it keeps min(need, the clusters the bare replicas
// allow) resident, so a launch of a few jobs always gets the room.
size_t anneal_smem(int cs, int Rl, int64_t rb, int n_max, bool moves, int need) {
    const size_t base = (size_t)(rb * Rl), q1 = sizeof(float4) * kQuenchScr * (size_t)n_max;
    const size_t one = base + q1, all = moves ? base + q1 * (size_t)Rl : one;
    static std::mutex mu;
    static std::map<std::tuple<int, int, int, size_t, size_t, bool, int>, size_t> memo;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return base;
    const auto key = std::make_tuple(dev, cs, Rl, base, all, moves, need);
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = memo.find(key);
        if (it != memo.end()) return it->second;
    }
    int a = 0;
    size_t pick = base;
    if (anneal_max_clusters(cs, Rl, base, moves, &a) == SQS_OK) {
        for (const size_t cand : {all, one}) {
            int b = 0;
            if (cand <= kAnnealSmemLimit && anneal_max_clusters(cs, Rl, cand, moves, &b) == SQS_OK &&
                b >= std::min(need, a)) {
                pick = cand;
                break;
            }
        }
    }
    std::lock_guard<std::mutex> lk(mu);
    memo[key] = pick;
    return pick;
}

}  // namespace ann
}  // namespace sqs
