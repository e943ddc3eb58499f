// FP32 cell-list SAT overlap + wall energy and gradient of many independent
// configurations: one CTA, or for n <= 256 one warp, per configuration.
//
// Per configuration:
//   1. load the n squares, cos/sin, wall term, cell on a G x G grid of cells
//      with side >= sqrt(2.000001) (so every interacting pair sits in the same
//      or adjacent cells), rank within the cell; a thread keeps its squares in
//      registers until the scatter;
//   2. exclusive scan of the cell counts, scatter to cell order;
//   3. broad phase: every square scans two contiguous ranges of the
//      cell-sorted array -- the rest of its own cell plus the east cell, and
//      the three cells of the row above -- which visits each unordered
//      neighbour pair exactly once, and keeps the hits of up to 32 candidates
//      as bits.  The set bits (a third of the candidates) are then appended
//      to a per-warp queue, one a lane a round, and every time 32 pairs are
//      queued the warp evaluates them (narrow phase at full SIMT width),
//      adding both squares' gradients with shared-memory integer atomics;
//   4. exact integer reduction of the energy, store of the gradient.
// Energies and gradients are integer sums, so results do not depend on the
// order in which pairs are found and the cells need no sorting.
// Reference: total_cached (seeded.cu:148-162) is the all-pairs O(n^2) form
// of the same energy; the legacy FP32 path's 16x16 cell grid of width 2
// (packing.cu:22-47) is the reference's own cell-list idea.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "sat_pair.cuh"

namespace sqs {

constexpr int kSatMaxN = 1024;
constexpr float kCellMin = 1.41422f;  // > sqrt(2.000001) = 1.4142139
constexpr int kQueue = 256, kCtaQueue = 128;  // pair queue entries of a warp: warp form, CTA form

// Pair energies are summed as integers in units of 2^-48.  A gap below zero is
// the difference of two floats of at least 1/2, or lies below -1/2 itself: a
// multiple of 2^-24 either way, so its square is a whole number of units and
// nothing is lost down to the smallest overlap (in units of 2^-40 a gap below
// 7e-7 vanished).  A term is below 1.46 * 2^48, and pairs go to the lanes in turn, at
// most 16,384 to one (half a million pairs, all taken by one warp), so a lane's
// sum stays below 2^63.  Wall terms have no bound (a square may lie anywhere), so
// they are summed in double, in thread order.
constexpr float kEnergyUnits = 281474976710656.0f;  // 2^48
__device__ __forceinline__ long long e_units(float e) { return __float2ll_rn(e * kEnergyUnits); }

// Exact sum past 64 bits: hi * 2^52 + lo with 0 <= lo < 2^52, one form for each
// value, so converting it does not depend on how the terms were dealt out.
struct EnergySum {
    long long hi, lo;
    __device__ __forceinline__ EnergySum(long long h, long long l) : hi(h + (l >> 52)), lo(l & ((1ll << 52) - 1)) {}
    __device__ __forceinline__ double value() const { return (double)hi * 0x1p4 + (double)lo * 0x1p-48; }
};

// Warp sum: the 26 low bits, the next 26 and the signed rest each sum within
// 32 bits.
__device__ __forceinline__ EnergySum warp_sum_units(long long v) {
    const unsigned s0 = __reduce_add_sync(0xffffffffu, (unsigned)v & 0x3ffffffu);
    const unsigned s1 = __reduce_add_sync(0xffffffffu, (unsigned)(v >> 26) & 0x3ffffffu);
    const int s2 = __reduce_add_sync(0xffffffffu, (int)(v >> 52));
    return EnergySum(s2, (long long)(((unsigned long long)s1 << 26) + s0));
}

// Nearest integer (ties to even) of |x| < 2^22 on the FMA pipe: x + 1.5 * 2^23
// lands in [2^23, 2^24), where one float ulp is 1, so its bit pattern minus
// that of 1.5 * 2^23 is the rounded integer.
constexpr float kMagic = 12582912.0f;
__device__ __forceinline__ int magic_int(float shifted) { return __float_as_int(shifted) - 0x4B400000; }

// Gradient accumulation with native 32-bit integer shared-memory atomics
// (shared-memory float atomics are several times slower): a contribution v
// is split into round(v * 2^12) and the signed rest in units of 2^-32, two
// integer sums that cannot overflow for n <= 1024 (|v| < 6 per pair) and that
// do not depend on the order of the additions.
struct GradFix {
    int* hi;  // [3n]
    int* lo;  // [3n]
    __device__ __forceinline__ void add(int k, float v) const {
        const float s = v * 4096.0f;
        const float h = s + kMagic;
        atomicAdd(hi + k, magic_int(h));
        atomicAdd(lo + k, magic_int(fmaf(s - (h - kMagic), 1048576.0f, kMagic)));
    }
    __device__ __forceinline__ float value(int k) const {
        return (float)(((double)hi[k] + (double)lo[k] * (1.0 / 1048576.0)) * (1.0 / 4096.0));
    }
};

__host__ __device__ inline int sat_grid_cap(int n) {
    // Cell grid side cap: about sqrt(2n) cells per side, at most 45 (L = 64).
    int g = (int)sqrtf(2.0f * (float)n);
    return g < 1 ? 1 : (g > 45 ? 45 : g);
}

__host__ __device__ inline size_t sat_smem_bytes(int n, int threads) {
    const int G = sat_grid_cap(n);
    size_t b = 0;
    b += (size_t)n * 16;                      // cell-sorted (x, y) and (c, s)
    b += (size_t)n * 24;                      // pair gradient accumulators (GradFix)
    b += (size_t)(threads / 32) * kCtaQueue * 4;  // warp pair queues
    b += ((size_t)(G * G + 1) * 2 + 3) & ~(size_t)3;  // cell counts / starts
    b += (size_t)n * 4;                       // sorted -> (original index, cell)
    b += 8 + (size_t)(threads / 32) * 32;     // reduction scratch
    return (b + 15) & ~(size_t)15;
}

// Broad phase of one warp's 32 squares p = base + lane over the cell-sorted
// centres: the two candidate ranges of each, 32 candidates at a time as hit
// bits; then every lane writes its hits at its place in the warp's queue (a
// prefix sum of the hit counts), and `flush(entry)` takes 32 queued pairs at a
// time off its end.  `qn`: queued pairs (below 32 on entry and exit).
//
// The test of a candidate is kept free of branches: a lane past its ranges
// reads on (at most 2 n + 4 centres from sxy, still the configuration's shared
// memory, whatever it holds) and its bits are masked at the end.  With a guard
// around each load a candidate took 21 instructions, half of the kernel's; at
// 4,096 x 200 41.1 us against 38.9 now, at 1,500 x 999 88.6 against 84.3.
template <bool COUNT, int CAP, class E, class Flush>
__device__ __forceinline__ void broad_phase(const float2* sxy, int p, float px, float py, int a1, int len1, int a2,
                                            int len, int lane, E* queue, int& qn, uint32_t& cand_loc, Flush&& flush) {
    constexpr int kShift = sizeof(E) * 4;  // an entry is p | q << kShift
    const int maxlen = __reduce_max_sync(0xffffffffu, len);
    for (int t0 = 0; t0 < maxlen; t0 += 32) {
        uint32_t hits = 0u, close = 0u;
        const float2* c1 = sxy + (a1 + t0);
        const float2* c2 = sxy + (a2 + t0);
        const int end = min(maxlen - t0, 32), n1 = len1 - t0;
        for (int k = 0; k < end; k += 4) {
            uint32_t m = 0u, mc = 0u;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float2 Q = (k + u < n1 ? c1 : c2)[k + u];
                const float dx = Q.x - px, dy = Q.y - py;
                const float d2 = dx * dx + dy * dy;
                if (d2 < kPairCut2) m |= 1u << u;
                if (COUNT && d2 < 2.0f) mc |= 1u << u;
            }
            hits |= m << k;
            if (COUNT) close |= mc << k;
        }
        const int mine_len = len - t0;
        const uint32_t valid = mine_len >= 32 ? 0xffffffffu : (mine_len > 0 ? (1u << mine_len) - 1u : 0u);
        hits &= valid;
        if (COUNT) cand_loc += __popc(close & valid);
        int left;  // hits of the warp not queued yet
        do {
            const int mine = __popc(hits);
            int incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            int at = qn + incl - mine;
            while (hits && at < CAP) {
                const int t = t0 + __ffs(hits) - 1;
                hits &= hits - 1u;
                queue[at++] = (E)((uint32_t)p | ((uint32_t)((t < len1 ? a1 : a2) + t) << kShift));
            }
            __syncwarp();
            left = max(qn + total - CAP, 0);
            for (qn = min(qn + total, CAP); qn >= 32; qn -= 32) flush((uint32_t)queue[qn - 32 + lane]);
            __syncwarp();
        } while (left > 0);
    }
}

// One CTA per configuration, a thread's squares (at most NPT) in registers from
// the load to the scatter.  n = 999 holds 52 KB of shared memory, so four CTAs
// of 256 threads share an SM.  The form before kept an original-order copy of
// the squares and the wall gradients there and summed energies in float, for
// which every cell was sorted: 76 KB, eight warps an SM, 243 us at 1,500 x 999
// against 88.6 (queues of 64 or 256 pairs a warp: 96 us, the one for its
// rounds, the other for a CTA less an SM; 512 threads: 97 us).
template <int T, int NPT>
__global__ void __launch_bounds__(T, T == 256 ? 4 : 1) sat_energy_kernel(int n, const float* __restrict__ xya,
                                                        const float* __restrict__ side,
                                                        float* __restrict__ energy,
                                                        float* __restrict__ grad,
                                                        uint32_t* __restrict__ cand) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int W = T / 32;
    const int cfg = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Gcap = sat_grid_cap(n);
    float2* sxy = reinterpret_cast<float2*>(smem);                  // cell-sorted centres
    float2* scs = sxy + n;                                          // cell-sorted cos/sin
    const GradFix gf{reinterpret_cast<int*>(scs + n), reinterpret_cast<int*>(scs + n) + 3 * n};
    uint32_t* queues = reinterpret_cast<uint32_t*>(gf.lo + 3 * n);
    uint16_t* cells = reinterpret_cast<uint16_t*>(queues + W * kCtaQueue);  // G*G + 1
    short2* sorted_meta = reinterpret_cast<short2*>(cells + ((Gcap * Gcap + 2) & ~1));  // (orig, cell)
    long long* red = reinterpret_cast<long long*>(((uintptr_t)(sorted_meta + n) + 7) & ~(uintptr_t)7);

    const float L = side[cfg];
    int G = (int)(L / kCellMin);
    G = G < 1 ? 1 : (G > Gcap ? Gcap : G);
    const float inv_cell = (float)G / L;
    const int ncell = G * G;

    for (int c = tid; c <= ncell; c += T) cells[c] = 0;
    for (int k = tid; k < 6 * n; k += T) gf.hi[k] = 0;
    __syncthreads();

    // 1. load, trig, walls, cell binning
    long long e_loc = 0;
    double e_wall = 0.0;
    const float* src = xya + (size_t)cfg * 3 * n;
    float sx[NPT], sy[NPT], sc[NPT], ss[NPT], wx[NPT], wy[NPT], wa[NPT];
    int cr[NPT];  // cell << 16 | rank
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
        const int i = tid + k * T;
        if (i < n) {
            const float x = src[3 * i], y = src[3 * i + 1], a = src[3 * i + 2];
            float s, c;
            sincosf(a, &s, &c);
            float gx = 0.f, gy = 0.f, ga = 0.f;
            e_wall += (double)wall_energy_grad(x, y, c, s, L, gx, gy, ga);
            wx[k] = gx;
            wy[k] = gy;
            wa[k] = ga;
            int cx = (int)floorf(x * inv_cell), cy = (int)floorf(y * inv_cell);
            cx = cx < 0 ? 0 : (cx >= G ? G - 1 : cx);
            cy = cy < 0 ? 0 : (cy >= G ? G - 1 : cy);
            const int cell = cy * G + cx;
            // per-cell counts in 16-bit halves of 32-bit words (native integer atomics)
            const unsigned old = atomicAdd(reinterpret_cast<unsigned*>(cells) + (cell >> 1), 1u << (16 * (cell & 1)));
            cr[k] = (cell << 16) | (int)((old >> (16 * (cell & 1))) & 0xffffu);
            sx[k] = x;
            sy[k] = y;
            sc[k] = c;
            ss[k] = s;
        }
    }
    __syncthreads();

    // 2. exclusive scan over ncell counts (one warp; ncell <= 2025)
    if (tid < 32) {
        const int per = (ncell + 31) / 32;
        const int lo = tid * per, hi = min(lo + per, ncell);
        int sum = 0;
        for (int c = lo; c < hi; ++c) sum += cells[c];
        int incl = sum;
        for (int o = 1; o < 32; o <<= 1) {
            int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (tid >= o) incl += v;
        }
        int run = incl - sum;
        for (int c = lo; c < hi; ++c) {
            int k = cells[c];
            cells[c] = (uint16_t)run;
            run += k;
        }
        if (tid == 31) cells[ncell] = (uint16_t)incl;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NPT; ++k) {
        const int i = tid + k * T;
        if (i < n) {
            const int cell = cr[k] >> 16, pos = cells[cell] + (cr[k] & 0xffff);
            sxy[pos] = make_float2(sx[k], sy[k]);
            scs[pos] = make_float2(sc[k], ss[k]);
            sorted_meta[pos] = make_short2((short)i, (short)cell);
        }
    }
    __syncthreads();

    // 3. broad phase into warp queues, narrow phase 32 pairs at a time
    uint32_t cand_loc = 0;
    uint32_t* queue = queues + warp * kCtaQueue;
    int qn = 0;  // warp-uniform queue length
    auto narrow = [&](uint32_t entry) {
        const int p = (int)(entry & 0xffffu), q = (int)(entry >> 16);
        const float2 P = sxy[p], Q = sxy[q], Pc = scs[p], Qc = scs[q];
        PairGrad g;
        if (sat_pair_grad(Q.x - P.x, Q.y - P.y, Pc.x, Pc.y, Qc.x, Qc.y, g)) {
            e_loc += e_units(g.e);
            const int i = sorted_meta[p].x, j = sorted_meta[q].x;
            gf.add(3 * i, g.px);
            gf.add(3 * i + 1, g.py);
            gf.add(3 * i + 2, g.pa);
            gf.add(3 * j, g.qx);
            gf.add(3 * j + 1, g.qy);
            gf.add(3 * j + 2, g.qa);
        }
    };
    for (int base = warp * 32; base < n; base += T) {
        const int p = base + lane;
        int a1 = 0, len1 = 0, a2 = 0, len = 0;
        float px = 0.f, py = 0.f;
        if (p < n) {
            const float2 P = sxy[p];
            px = P.x;
            py = P.y;
            const int cell = sorted_meta[p].y, cy = cell / G, cx = cell - cy * G;
            // own cell after p, then the east cell (same row, contiguous)
            a1 = p + 1;
            len1 = cells[cy * G + min(cx + 2, G)] - a1;
            // the row above: cells cx-1 .. cx+1
            int len2 = 0;
            if (cy + 1 < G) {
                a2 = cells[(cy + 1) * G + max(cx - 1, 0)];
                len2 = cells[(cy + 1) * G + min(cx + 2, G)] - a2;
            }
            len = len1 + len2;
            a2 -= len1;  // q = a2 + t for t >= len1
        }
        if (cand) broad_phase<true, kCtaQueue>(sxy, p, px, py, a1, len1, a2, len, lane, queue, qn, cand_loc, narrow);
        else broad_phase<false, kCtaQueue>(sxy, p, px, py, a1, len1, a2, len, lane, queue, qn, cand_loc, narrow);
    }
    __syncwarp();
    if (lane < qn) narrow(queue[lane]);
    __syncthreads();

    // 4. reductions and stores
    const EnergySum e_warp = warp_sum_units(e_loc);
    cand_loc = __reduce_add_sync(0xffffffffu, cand_loc);
    for (int o = 16; o > 0; o >>= 1) e_wall += __shfl_xor_sync(0xffffffffu, e_wall, o);
    if (lane == 0) {
        red[4 * warp] = e_warp.hi;
        red[4 * warp + 1] = e_warp.lo;
        red[4 * warp + 2] = cand_loc;
        red[4 * warp + 3] = __double_as_longlong(e_wall);
    }
    __syncthreads();
    if (tid == 0) {
        long long hi = 0, lo = 0, cc = 0;
        double walls = 0.0;
        for (int w = 0; w < W; ++w) {
            hi += red[4 * w];
            lo += red[4 * w + 1];
            cc += red[4 * w + 2];
            walls += __longlong_as_double(red[4 * w + 3]);
        }
        energy[cfg] = (float)(walls + EnergySum(hi, lo).value());
        if (cand) cand[cfg] = (uint32_t)cc;
    }
    if (grad) {
        float* dst = grad + (size_t)cfg * 3 * n;
#pragma unroll
        for (int k = 0; k < NPT; ++k) {
            const int i = tid + k * T;
            if (i < n) {
                dst[3 * i] = wx[k] + gf.value(3 * i);
                dst[3 * i + 1] = wy[k] + gf.value(3 * i + 1);
                dst[3 * i + 2] = wa[k] + gf.value(3 * i + 2);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Warp-per-configuration form for n <= 256: the same phases as above run by
// one warp without block barriers, several configurations per CTA.  A lane
// keeps its squares (NPL of them, the kernel is instantiated for each number)
// in registers from the load to the scatter, all loads are issued before any
// is used, and the cell grid is sized from n, so ~7.7 KB of shared memory per
// configuration lets a whole 4,096-configuration batch of n = 200 be resident
// in one wave.  Bound by issue slots (70% issuing at 4,096 x 200).  An instance
// sized for n = 17 takes 6.15 us a call of 48 against 8.2 for the largest's.
constexpr int kWarpMaxN = 256;

__host__ __device__ inline int warp_grid_cap(int n) {
    int g = (int)sqrtf((float)n) + 2;
    return g > 45 ? 45 : g;
}

__host__ __device__ inline size_t warp_smem_bytes(int n) {
    const int G = warp_grid_cap(n);
    // sorted (x, y) + (c, s), pair-gradient accumulators, original index (byte),
    // cell starts (uint16), pair queue
    size_t b = (size_t)n * 16 + (size_t)n * 12 + (((size_t)n + 3) & ~(size_t)3) +
               (((size_t)(G * G + 1) * 2 + 3) & ~(size_t)3) + kQueue * 2;
    return (b + 15) & ~(size_t)15;
}

// Pair-gradient sums of the warp kernel: one 32-bit integer per component in
// units of 2^-19.  A pair term is bounded by 2 r_max (|d| + 1/sqrt 2) =
// 2 * 1.2071 * 2.1213 < 5.13, so with n <= 256 (at most 255 partners) a sum
// stays below 2^31 units; every term is rounded once (error < 1e-6) and the
// sum is exact and order-free.
constexpr float kGScale = 524288.0f;

// round(v * kGScale) on the FMA pipe: |v| < 5.13 keeps v * 2^19 below 2^22.
__device__ __forceinline__ int gq_units(float v) { return magic_int(fmaf(v, kGScale, kMagic)); }

// 28 / W CTAs of W warps per SM (72 registers a thread at W = 4; the default
// is W = 2, measured 2% faster than 4 and 20% faster than 8): with the
// shared memory of n = 200 that keeps 4,096 configurations in one wave.
template <int W, bool COUNT, int NPL>
__global__ void __launch_bounds__(W * 32, 28 / W) sat_energy_warp_kernel(int configs, int n, const float* __restrict__ xya,
                                                                 const float* __restrict__ side,
                                                                 float* __restrict__ energy, float* __restrict__ grad,
                                                                 uint32_t* __restrict__ cand) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cfg = blockIdx.x * W + warp;
    if (cfg >= configs) return;
    const size_t wb = warp_smem_bytes(n);
    unsigned char* base = smem + (size_t)warp * wb;
    const int Gcap = warp_grid_cap(n);
    float2* sxy = reinterpret_cast<float2*>(base);            // cell-sorted centres
    float2* scs = sxy + n;                                     // cell-sorted cos/sin
    int* gq = reinterpret_cast<int*>(scs + n);                 // pair-gradient sums (kGScale units)
    uint8_t* orig = reinterpret_cast<uint8_t*>(gq + 3 * n);    // sorted -> original index
    uint16_t* cells = reinterpret_cast<uint16_t*>(orig + ((n + 3) & ~3));  // G*G + 1 starts
    uint16_t* queue = cells + (((Gcap * Gcap + 1) + 1) & ~1);  // p | q << 8

    const float L = side[cfg];
    int G = (int)(L / kCellMin);
    G = G < 1 ? 1 : (G > Gcap ? Gcap : G);
    const float inv_cell = (float)G / L;
    const int ncell = G * G;
    for (int c = lane; c <= ncell; c += 32) cells[c] = 0;
    float* gdst = grad ? grad + (size_t)cfg * 3 * n : nullptr;

    // 1. all loads first, then trig, walls and cell ranks
    const float* src = xya + (size_t)cfg * 3 * n;
    float px[NPL], py[NPL], pa[NPL];
#pragma unroll
    for (int k = 0; k < NPL; ++k) {
        const int i = lane + 32 * k;
        if (i < n) {
            px[k] = src[3 * i];
            py[k] = src[3 * i + 1];
            pa[k] = src[3 * i + 2];
        }
    }
    __syncwarp();
    long long e_loc = 0;  // exact, so the sum does not depend on the order of the pairs
    double e_wall = 0.0;
    // Wall gradients wait in registers for the pair sums; with many squares a
    // lane there is no room, and they go straight out and are read back.
    constexpr bool kKeepWalls = NPL <= 2;
    float wx[kKeepWalls ? NPL : 1], wy[kKeepWalls ? NPL : 1], wa[kKeepWalls ? NPL : 1];
    float pc[NPL], ps[NPL];
    int cr[NPL];  // cell << 16 | rank
#pragma unroll
    for (int k = 0; k < NPL; ++k) {
        const int i = lane + 32 * k;
        if (i < n) {
            sincosf(pa[k], &ps[k], &pc[k]);
            float gx = 0.f, gy = 0.f, ga = 0.f;
            e_wall += (double)wall_energy_grad(px[k], py[k], pc[k], ps[k], L, gx, gy, ga);
            // (kept apart from the pair sums: unbounded for squares far outside the box)
            if (kKeepWalls) {
                wx[k % (kKeepWalls ? NPL : 1)] = gx;
                wy[k % (kKeepWalls ? NPL : 1)] = gy;
                wa[k % (kKeepWalls ? NPL : 1)] = ga;
            } else if (gdst) {
                gdst[3 * i] = gx;
                gdst[3 * i + 1] = gy;
                gdst[3 * i + 2] = ga;
            }
            gq[3 * i] = gq[3 * i + 1] = gq[3 * i + 2] = 0;
            int cx = (int)floorf(px[k] * inv_cell), cy = (int)floorf(py[k] * inv_cell);
            cx = cx < 0 ? 0 : (cx >= G ? G - 1 : cx);
            cy = cy < 0 ? 0 : (cy >= G ? G - 1 : cy);
            const int cell = cy * G + cx;
            // per-cell counts in 16-bit halves of 32-bit words (native integer atomics)
            const unsigned old = atomicAdd(reinterpret_cast<unsigned*>(cells) + (cell >> 1), 1u << (16 * (cell & 1)));
            cr[k] = (cell << 16) | (int)((old >> (16 * (cell & 1))) & 0xffffu);
        }
    }
    __syncwarp();
    // 2. exclusive scan of the cell counts, scatter from registers
    {
        const int per = (ncell + 31) / 32;
        const int lo = lane * per, hi = min(lo + per, ncell);
        int sum = 0;
        for (int c = lo; c < hi; ++c) sum += cells[c];
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        int run = incl - sum;
        for (int c = lo; c < hi; ++c) {
            const int k = cells[c];
            cells[c] = run;
            run += k;
        }
        if (lane == 31) cells[ncell] = incl;
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < NPL; ++k) {
        const int i = lane + 32 * k;
        if (i < n) {
            const int cell = cr[k] >> 16;
            const int pos = cells[cell] + (cr[k] & 0xffff);
            sxy[pos] = make_float2(px[k], py[k]);
            scs[pos] = make_float2(pc[k], ps[k]);
            orig[pos] = (uint8_t)i;
        }
    }
    __syncwarp();

    // 3. broad phase into the warp queue, narrow phase 32 pairs at a time
    uint32_t cand_loc = 0;
    int qn = 0;
    auto narrow = [&](uint32_t entry) {
        const int p = (int)(entry & 0xffu), q = (int)(entry >> 8);
        const float2 P = sxy[p], Q = sxy[q], Pc = scs[p], Qc = scs[q];
        PairGrad g;
        if (sat_pair_grad(Q.x - P.x, Q.y - P.y, Pc.x, Pc.y, Qc.x, Qc.y, g)) {
            e_loc += e_units(g.e);
            const int i = orig[p], j = orig[q];
            atomicAdd(gq + 3 * i, gq_units(g.px));
            atomicAdd(gq + 3 * i + 1, gq_units(g.py));
            atomicAdd(gq + 3 * i + 2, gq_units(g.pa));
            atomicAdd(gq + 3 * j, gq_units(g.qx));
            atomicAdd(gq + 3 * j + 1, gq_units(g.qy));
            atomicAdd(gq + 3 * j + 2, gq_units(g.qa));
        }
    };
    for (int base0 = 0; base0 < n; base0 += 32) {
        const int p = base0 + lane;
        int a1 = 0, len1 = 0, a2 = 0, len = 0;
        float qx0 = 0.f, qy0 = 0.f;
        if (p < n) {
            const float2 P = sxy[p];
            qx0 = P.x;
            qy0 = P.y;
            int cx = (int)floorf(P.x * inv_cell), cy = (int)floorf(P.y * inv_cell);
            cx = cx < 0 ? 0 : (cx >= G ? G - 1 : cx);
            cy = cy < 0 ? 0 : (cy >= G ? G - 1 : cy);
            a1 = p + 1;
            len1 = cells[cy * G + min(cx + 2, G)] - a1;
            int len2 = 0;
            if (cy + 1 < G) {
                a2 = cells[(cy + 1) * G + max(cx - 1, 0)];
                len2 = cells[(cy + 1) * G + min(cx + 2, G)] - a2;
            }
            len = len1 + len2;
            a2 -= len1;  // q = a2 + t for t >= len1
        }
        broad_phase<COUNT, kQueue>(sxy, p, qx0, qy0, a1, len1, a2, len, lane, queue, qn, cand_loc, narrow);
    }
    __syncwarp();
    if (lane < qn) narrow(queue[lane]);
    __syncwarp();

    // 4. reductions and the gradient store
    const EnergySum e_sum = warp_sum_units(e_loc);
    if (COUNT) cand_loc = __reduce_add_sync(0xffffffffu, cand_loc);
    for (int o = 16; o > 0; o >>= 1) e_wall += __shfl_xor_sync(0xffffffffu, e_wall, o);
    if (lane == 0) {
        energy[cfg] = (float)(e_wall + e_sum.value());
        if (COUNT) cand[cfg] = cand_loc;
    }
    if (!gdst) return;
    if (kKeepWalls) {
#pragma unroll
        for (int k = 0; k < NPL; ++k) {
            const int i = lane + 32 * k;
            if (i < n) {
                gdst[3 * i] = wx[k % (kKeepWalls ? NPL : 1)] + (float)gq[3 * i] * (1.0f / kGScale);
                gdst[3 * i + 1] = wy[k % (kKeepWalls ? NPL : 1)] + (float)gq[3 * i + 1] * (1.0f / kGScale);
                gdst[3 * i + 2] = wa[k % (kKeepWalls ? NPL : 1)] + (float)gq[3 * i + 2] * (1.0f / kGScale);
            }
        }
    } else {
        for (int k = lane; k < 3 * n; k += 32) gdst[k] += (float)gq[k] * (1.0f / kGScale);
    }
}

template <int W, int NPL>
static int launch_warp_npl(sqs_ctx* ctx, cudaStream_t st, int configs, int n, const float* xya, const float* side,
                           float* energy, float* grad, uint32_t* cand) {
    const size_t smem = warp_smem_bytes(n) * W;
    static bool attr_set[64] = {false};
    const int dev = ctx->device & 63;
    if (!attr_set[dev]) {
        SQS_CUDA(cudaFuncSetAttribute(sat_energy_warp_kernel<W, true, NPL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      200 * 1024));
        SQS_CUDA(cudaFuncSetAttribute(sat_energy_warp_kernel<W, false, NPL>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr_set[dev] = true;
    }
    const unsigned blocks = (unsigned)((configs + W - 1) / W);
    if (cand)
        sat_energy_warp_kernel<W, true, NPL><<<blocks, W * 32, smem, st>>>(configs, n, xya, side, energy, grad, cand);
    else
        sat_energy_warp_kernel<W, false, NPL><<<blocks, W * 32, smem, st>>>(configs, n, xya, side, energy, grad,
                                                                            nullptr);
    SQS_CUDA(cudaGetLastError());
    ctx->launches += 1;
    return SQS_OK;
}

// W warps per CTA; the instance with the squares a lane has, rounded up (the
// widths other than the default keep one instance for every n).
template <int W>
static int launch_warp(sqs_ctx* ctx, cudaStream_t st, int configs, int n, const float* xya, const float* side,
                       float* energy, float* grad, uint32_t* cand) {
    if (W != 2) return launch_warp_npl<W, 8>(ctx, st, configs, n, xya, side, energy, grad, cand);
    switch ((n + 31) / 32) {
        case 1: return launch_warp_npl<2, 1>(ctx, st, configs, n, xya, side, energy, grad, cand);
        case 2: return launch_warp_npl<2, 2>(ctx, st, configs, n, xya, side, energy, grad, cand);
        case 3: return launch_warp_npl<2, 3>(ctx, st, configs, n, xya, side, energy, grad, cand);
        case 4: return launch_warp_npl<2, 4>(ctx, st, configs, n, xya, side, energy, grad, cand);
        case 5: return launch_warp_npl<2, 5>(ctx, st, configs, n, xya, side, energy, grad, cand);
        case 6: return launch_warp_npl<2, 6>(ctx, st, configs, n, xya, side, energy, grad, cand);
        case 7: return launch_warp_npl<2, 7>(ctx, st, configs, n, xya, side, energy, grad, cand);
        default: return launch_warp_npl<2, 8>(ctx, st, configs, n, xya, side, energy, grad, cand);
    }
}

// The CTA form at T threads, in the instance with the squares a thread has,
// rounded up to a power of two.  One instance for 1024 / T squares a thread at
// every n cost registers and unrolled rounds that small configurations have no
// use for (255 at 32 threads): 8,192 x 17 at 32 threads took 61.8 us against
// 14.7 now, 4,096 x 200 at 64 threads 90.6 against 53.3.
template <int T, int NPT = 1>
static int launch(sqs_ctx* ctx, cudaStream_t st, int configs, int n, const float* xya, const float* side,
                  float* energy, float* grad, uint32_t* cand) {
    if constexpr (T * NPT < kSatMaxN)
        if (n > T * NPT) return launch<T, 2 * NPT>(ctx, st, configs, n, xya, side, energy, grad, cand);
    const size_t smem = sat_smem_bytes(n, T);
    static bool attr_set[64] = {false};
    const int dev = ctx->device & 63;
    if (!attr_set[dev]) {
        SQS_CUDA(cudaFuncSetAttribute(sat_energy_kernel<T, NPT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      96 * 1024));
        attr_set[dev] = true;
    }
    sat_energy_kernel<T, NPT><<<configs, T, smem, st>>>(n, xya, side, energy, grad, cand);
    SQS_CUDA(cudaGetLastError());
    ctx->launches += 1;
    return SQS_OK;
}

static int sat_energy_launch_on(sqs_ctx* ctx, cudaStream_t st, int configs, int n, const float* xya,
                                const float* side, float* energy, float* grad, uint32_t* cand, int threads) {
    SQS_REQUIRE(configs >= 0 && configs <= (1 << 30), "configs %d out of range", configs);
    SQS_REQUIRE(n >= 1 && n <= kSatMaxN, "n %d out of 1..%d", n, kSatMaxN);
    SQS_REQUIRE(xya && side && energy, "null device pointer");
    if (configs == 0) return SQS_OK;
    if (threads == 0) threads = n <= kWarpMaxN ? -2 : 256;
    if (threads < 0) {  // warp-per-configuration kernel, -threads warps per CTA
        SQS_REQUIRE(n <= kWarpMaxN, "the warp-per-configuration kernel takes n <= %d", kWarpMaxN);
        switch (-threads) {
            case 2: return launch_warp<2>(ctx, st, configs, n, xya, side, energy, grad, cand);
            case 4: return launch_warp<4>(ctx, st, configs, n, xya, side, energy, grad, cand);
            case 8: return launch_warp<8>(ctx, st, configs, n, xya, side, energy, grad, cand);
            default: break;
        }
        SQS_REQUIRE(false, "threads %d: warps per CTA must be 2, 4 or 8", threads);
    }
    switch (threads) {
        case 32: return launch<32>(ctx, st, configs, n, xya, side, energy, grad, cand);
        case 64: return launch<64>(ctx, st, configs, n, xya, side, energy, grad, cand);
        case 128: return launch<128>(ctx, st, configs, n, xya, side, energy, grad, cand);
        case 256: return launch<256>(ctx, st, configs, n, xya, side, energy, grad, cand);
        default: break;
    }
    SQS_REQUIRE(false, "threads %d not in {32, 64, 128, 256}", threads);
}

int sat_energy_launch(sqs_ctx* ctx, int configs, int n, const float* xya, const float* side,
                      float* energy, float* grad, uint32_t* cand, int threads) {
    return sat_energy_launch_on(ctx, ctx->stream, configs, n, xya, side, energy, grad, cand, threads);
}

}  // namespace sqs

extern "C" int sqs_sat_energy(sqs_ctx* ctx, int configs, int n, const float* xya, const float* side,
                              float* energy, float* grad, uint32_t* cand, int threads) {
    if (int r = sqs::enter(ctx)) return r;
    return sqs::sat_energy_launch(ctx, configs, n, xya, side, energy, grad, cand, threads);
}

extern "C" int sqs_sat_energy_host(sqs_ctx* ctx, int configs, int n, const float* xya,
                                   const float* side, float* energy, float* grad, uint32_t* cand) {
    if (int r = sqs::enter(ctx)) return r;
    SQS_REQUIRE(configs >= 0 && n >= 1 && n <= sqs::kSatMaxN, "configs/n out of range");
    SQS_REQUIRE(xya && side && energy, "null host pointer");
    if (configs == 0) return SQS_OK;
    const size_t sb = (size_t)configs * n * 3 * sizeof(float);
    if (int r = ctx->d_in.reserve(sb)) return r;
    if (int r = ctx->d_side.reserve((size_t)configs * sizeof(float))) return r;
    if (int r = ctx->d_out.reserve((size_t)configs * sizeof(float))) return r;
    if (grad)
        if (int r = ctx->d_grad.reserve(sb)) return r;
    if (cand)
        if (int r = ctx->d_cand.reserve((size_t)configs * sizeof(uint32_t))) return r;
    // Chunks of the batch on the context's side streams: the upload of one
    // chunk, the kernel of the one before and the download of the one before
    // that overlap.  Four chunks measured best for 4,096 x 200 squares
    // (0.38 ms per call against 0.44 ms in one piece; 8 and 16 chunks cost
    // more in calls than they gain: the host link carried about 51 GB/s in
    // both directions together, so the transfers overlap only in part).
    const int chunks = configs >= 1024 ? std::min(4, configs / 256) : 1;
    float* d_in = (float*)ctx->d_in.p;
    float* d_side = (float*)ctx->d_side.p;
    float* d_out = (float*)ctx->d_out.p;
    float* d_grad = grad ? (float*)ctx->d_grad.p : nullptr;
    uint32_t* d_cand = cand ? (uint32_t*)ctx->d_cand.p : nullptr;
    const int na = chunks == 1 ? 0 : std::min(chunks, sqs_ctx::kAux);
    SQS_CUDA(cudaEventRecord(ctx->fork, ctx->stream));
    for (int a = 0; a < na; ++a) SQS_CUDA(cudaStreamWaitEvent(ctx->aux[a], ctx->fork, 0));
    int rc = SQS_OK;
    for (int c = 0; c < chunks && rc == SQS_OK; ++c) {
        cudaStream_t st = chunks == 1 ? ctx->stream : ctx->aux[c % sqs_ctx::kAux];
        const int64_t lo = (int64_t)configs * c / chunks, hi = (int64_t)configs * (c + 1) / chunks;
        const int cnt = (int)(hi - lo);
        const size_t e0 = (size_t)lo * n * 3, eb = (size_t)cnt * n * 3 * sizeof(float);
        SQS_CUDA(cudaMemcpyAsync(d_in + e0, xya + e0, eb, cudaMemcpyHostToDevice, st));
        SQS_CUDA(cudaMemcpyAsync(d_side + lo, side + lo, (size_t)cnt * sizeof(float), cudaMemcpyHostToDevice, st));
        rc = sqs::sat_energy_launch_on(ctx, st, cnt, n, d_in + e0, d_side + lo, d_out + lo,
                                       d_grad ? d_grad + e0 : nullptr, d_cand ? d_cand + lo : nullptr, 0);
        if (rc) break;
        SQS_CUDA(cudaMemcpyAsync(energy + lo, d_out + lo, (size_t)cnt * sizeof(float), cudaMemcpyDeviceToHost, st));
        if (grad) SQS_CUDA(cudaMemcpyAsync(grad + e0, d_grad + e0, eb, cudaMemcpyDeviceToHost, st));
        if (cand)
            SQS_CUDA(cudaMemcpyAsync(cand + lo, d_cand + lo, (size_t)cnt * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                     st));
    }
    // join every side stream, also after a failure
    for (int a = 0; a < na; ++a) {
        SQS_CUDA(cudaEventRecord(ctx->join[a], ctx->aux[a]));
        SQS_CUDA(cudaStreamWaitEvent(ctx->stream, ctx->join[a], 0));
    }
    if (rc) return rc;
    SQS_CUDA(cudaStreamSynchronize(ctx->stream));
    return SQS_OK;
}
