// FP64 gradient polish of every job's best state, one CTA per job.
//
// The reference polishes every chain after every epoch with PRP+ conjugate
// gradient and a 5-step backtracking search on the squared-penetration
// energy at the chain's target side (seeded.cu:621-713, gradient
// pair_cached_smooth :67-90 and the smooth wall derivative :640-645).  Here
// the polish runs once per job on its best FP64 state: compress the state by
// a factor (1 - delta) into a side L (1 - delta), descend the same energy
// with a backtracking line search until it vanishes, and keep the result if
// its dilation-certified side (device_certified_side, seeded.cu:175-226) is
// smaller; delta shrinks after every failure.  Every square's pairs are taken
// in ascending order of the partner, over a neighbour list found through a
// cell grid, so gradients need no atomics and all sums have a fixed order:
// the result is deterministic and equals the all-pairs loop's bit for bit.
//
// Bound by the FP64 pipe for large n (one CTA on one SM) and by the chain of
// dependent FP64 operations for small n.  A line-search trial brings the
// gradient of its state along, so an accepted step evaluates its state once
// instead of twice; lists and certified sides go through cells instead of all
// pairs; a trial takes two block barriers instead of six, and for small n
// several lanes share a square's partners.  64 packings of n 5..1000, half of
// them overlapped, 200 steps: 7.8 -> 3.2 ms a call (one B200).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>
#include <vector>

#include "anneal.cuh"
#include "common.cuh"

namespace sqs {
namespace ann {

// Threads of a CTA by its size class (see launch_widths): a narrow CTA takes
// packings of up to kWidthN squares and shares its SM with others.
constexpr int kSmallT = 128, kMidT = 256, kWideT = 512;
template <int PT>
constexpr int kWidthN = PT == kSmallT ? 64 : (PT == kMidT ? 256 : kMaxN);
template <int PT>
constexpr int kResident = PT == kSmallT ? 4 : (PT == kMidT ? 2 : 1);  // CTAs an SM the registers allow
template <int PT>
constexpr int kPer = (kWidthN<PT> + PT - 1) / PT;  // squares a thread
constexpr int kPS = 256;  // an energy's partial sums (see energy())

// Neighbour lists of the polish: every partner within sqrt(2.000001) + 0.25
// of a square when the list was built (at most kNbK, ascending), valid while
// no square has moved more than kNbMove since -- then every pair inside the
// pair cut-off is listed.  Energies over the list sum the same nonzero terms
// in the same order as the all-pairs loop, so they are bit-identical to it.
constexpr int kNbK = 24;
constexpr double kNbR2 = 2.7697;       // (sqrt(2.000001) + 0.25)^2 = 2.76961, rounded up
constexpr double kNbMove = 0.1249;     // below 0.125 by more than the bounds' rounding
// Cells of the grid that finds neighbours: wider than the list's radius
// (1.66424) and the certified side's (sqrt 2.05), at most kCG a side.
constexpr double kCellW = 1.6645, kCellMinW = 1.6643;
constexpr int kCG = 32;

constexpr int kTerms = 4;  // energy terms kept a square (see energy())
// An array in the CTA's dynamic shared memory by its byte offset: buffers that
// are passed around and swapped stay visibly shared, so every access is a
// shared-memory instruction (as pointers they became generic loads, a third
// of the kernel's stalls).
extern __shared__ __align__(16) unsigned char polish_dyn[];
template <class T>
struct Sh {
    int off;
    __device__ __forceinline__ T& operator[](int i) const { return reinterpret_cast<T*>(polish_dyn + off)[i]; }
    __device__ __forceinline__ Sh operator+(int i) const { return Sh{off + i * (int)sizeof(T)}; }
};

__device__ __forceinline__ double sgn_s(double x) { return fabs(x) > 1e-6 ? (x >= 0.0 ? 1.0 : -1.0) : 0.0; }

// Smooth-variant pair gradient for square p against q (pair_cached_smooth):
// returns gap^2 and adds d/dp into g.
__device__ __forceinline__ double pair_smooth(double px, double py, double c, double s, double qx, double qy,
                                              double d, double t, double& gx, double& gy, double& ga) {
    const double dx = qx - px, dy = qy - py;
    if (dx * dx + dy * dy >= 2.000001) return 0.0;
    const double cd = c * d + s * t, sd = s * d - c * t;
    const double rad = 0.5 + 0.5 * (fabs(cd) + fabs(sd));
    const double deriv = 0.5 * (-sgn_s(cd) * sd + sgn_s(sd) * cd);
    const double ux[4] = {c, -s, d, -t}, uy[4] = {s, c, t, d};
    double gap = -1e100, ggx = 0, ggy = 0, gga = 0;
    for (int k = 0; k < 4; ++k) {
        const double v = dx * ux[k] + dy * uy[k], z = fabs(v) - rad;
        if (z > gap) {
            gap = z;
            const double sv = v >= 0.0 ? 1.0 : -1.0;
            ggx = -sv * ux[k];
            ggy = -sv * uy[k];
            gga = -deriv + (k < 2 ? sv * (-dx * uy[k] + dy * ux[k]) : 0.0);
        }
    }
    if (gap >= 0.0) return 0.0;
    gx += 2.0 * gap * ggx;
    gy += 2.0 * gap * ggy;
    ga += 2.0 * gap * gga;
    return gap * gap;
}

__device__ __forceinline__ double wall_smooth(double x, double y, double c, double s, double L, double& gx,
                                              double& gy, double& ga) {
    const double r = 0.5 * (fabs(c) + fabs(s));
    const double dr = 0.5 * (-sgn_s(c) * s + sgn_s(s) * c);
    const double v[4] = {r - x, x + r - L, r - y, y + r - L};
    double e = 0.0;
    for (int k = 0; k < 4; ++k) {
        if (v[k] > 0.0) {
            e += v[k] * v[k];
            const double f = 2.0 * v[k];
            gx += f * (k == 0 ? -1.0 : k == 1 ? 1.0 : 0.0);
            gy += f * (k == 2 ? -1.0 : k == 3 ? 1.0 : 0.0);
            ga += f * dr;
        }
    }
    return e;
}

template <int PT>
__device__ double block_max(double v, Sh<double> red) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = red[0];
    for (int w = 1; w < PT / 32; ++w) t = fmax(t, red[w]);
    return t;
}

struct NbrList {
    Sh<uint16_t> idx;  // partners of square i: idx[i * kNbK + k], k < cnt[i]
    Sh<uint8_t> cnt;
};

// Squares by cell: order[start[c] .. start[c + 1]) lie in cell c = cy * G + cx
// of a G x G grid over [x0, x0 + side] x [y0, y0 + side].  A square outside
// counts into the nearest edge cell, which keeps any two squares closer than
// a cell's width in the same or adjacent cells.
struct Cells {
    Sh<uint16_t> order;
    Sh<int> start;  // kCG * kCG + 1
    double x0, y0, inv;
    int G;
    __device__ __forceinline__ int at(double x) const { return min(G - 1, max(0, __double2int_rd(x * inv))); }
    __device__ __forceinline__ int cx(const double3& p) const { return at(p.x - x0); }
    __device__ __forceinline__ int cy(const double3& p) const { return at(p.y - y0); }
};

// Sort the squares of q into cells.  Starts and ends with a barrier.
template <int PT>
__device__ void build_cells(int n, Cells& c, Sh<double3> q, double x0, double y0, double side) {
    c.x0 = x0;
    c.y0 = y0;
    c.G = min(kCG, max(1, __double2int_rd(side / kCellW)));
    c.inv = (double)c.G / side;
    if (!(c.inv > 0.0 && c.inv * kCellMinW <= 1.0)) c.inv = 0.0, c.G = 1;  // a side below one cell, or not finite
    const int ncell = c.G * c.G, t = threadIdx.x;
    __syncthreads();
    for (int k = t; k <= ncell; k += PT) c.start[k] = 0;
    __syncthreads();
    int rank[kPer<PT>], cell[kPer<PT>];
#pragma unroll
    for (int m = 0; m < kPer<PT>; ++m) {
        const int i = t + m * PT;
        if (i < n) {
            cell[m] = c.cy(q[i]) * c.G + c.cx(q[i]);
            rank[m] = atomicAdd(&c.start[cell[m]], 1);
        }
    }
    __syncthreads();
    if (t < 32) {  // exclusive scan, a run of cells a lane
        const int per = (ncell + 31) / 32, lo = t * per, hi = min(lo + per, ncell);
        int sum = 0;
        for (int k = lo; k < hi; ++k) sum += c.start[k];
        int incl = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (t >= o) incl += v;
        }
        int run = incl - sum;
        for (int k = lo; k < hi; ++k) {
            const int v = c.start[k];
            c.start[k] = run;
            run += v;
        }
        if (t == 31) c.start[ncell] = incl;
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < kPer<PT>; ++m) {
        const int i = t + m * PT;
        if (i < n) c.order[c.start[cell[m]] + rank[m]] = (uint16_t)i;
    }
    __syncthreads();
}

// Build the list for state q from its cells; false when a square has more
// than kNbK partners (the callers then use all pairs).
template <int PT>
__device__ bool build_nbr(int n, const NbrList& nb, const Cells& c, Sh<double3> q) {
    bool over = false;
    for (int i = threadIdx.x; i < n; i += PT) {
        const double3 p = q[i];
        const Sh<uint16_t> L = nb.idx + i * kNbK;
        const int cx = c.cx(p), cy = c.cy(p);
        const int xa = max(cx - 1, 0), xb = min(cx + 1, c.G - 1);
        int m = 0;
        for (int y = max(cy - 1, 0); y <= min(cy + 1, c.G - 1); ++y) {
            for (int k = c.start[y * c.G + xa]; k < c.start[y * c.G + xb + 1]; ++k) {
                const int j = c.order[k];
                if (j == i) continue;
                const double dx = q[j].x - p.x, dy = q[j].y - p.y;
                if (dx * dx + dy * dy < kNbR2) {
                    if (m < kNbK) {  // insert in ascending order
                        int w = m;
                        for (; w > 0 && L[w - 1] > j; --w) L[w] = L[w - 1];
                        L[w] = (uint16_t)j;
                    }
                    ++m;
                }
            }
        }
        nb.cnt[i] = (uint8_t)min(m, kNbK);
        over |= m > kNbK;
    }
    return !__syncthreads_or(over);
}

// Energy of the state q at side L, its gradient into g, and the largest
// squared centre gradient into gmax2: over the neighbour list when nb != nullptr, else
// over all pairs.  The energy is kPS partial sums, added by butterflies and
// then warp by warp: partial s takes squares s, s + kPS, ..., of each the wall
// first, then the partners above it in ascending order -- one order whatever
// the number of threads.  For n <= kPS over a list, 2, 4 or 8 lanes evaluate a
// square's partners at once and add the nonzero terms in that order.  For
// larger n a thread takes whole squares and leaves their nonzero energy terms
// (at most kTerms; a square with more is summed again) to the threads that
// add up the partials.  The barrier that publishes the state before a call
// also ends the reads of the call before.
struct Red {
    Sh<double> e;       // [kPS / 32]
    Sh<double> m;       // [kWideT / 32]
    Sh<double> es;      // [kPS]: squares' sums of the lane-parallel form
    Sh<double> terms;   // [n][kTerms]
    Sh<uint8_t> nterm;  // [n]: terms there, kTerms + 1: more than fit
};

// Energy terms of square i added to e in their order (no gradient).
__device__ __noinline__ double add_square(double e, int i, int n, Sh<double3> q, Sh<double2> cs, double L,
                                          const NbrList& nb, bool listed) {
    const double3 p = q[i];
    const double2 pc = cs[i];
    double gx = 0, gy = 0, ga = 0;
    e += wall_smooth(p.x, p.y, pc.x, pc.y, L, gx, gy, ga);
    const int m = listed ? nb.cnt[i] : n;
    for (int k = 0; k < m; ++k) {
        const int j = listed ? (int)nb.idx[i * kNbK + k] : k;
        if (j <= i) continue;
        const double3 o = q[j];
        const double2 oc = cs[j];
        e += pair_smooth(p.x, p.y, pc.x, pc.y, o.x, o.y, oc.x, oc.y, gx, gy, ga);
    }
    return e;
}

template <int PT>
__device__ double energy(int n, Sh<double3> q, Sh<double2> cs, double L, Sh<double3> g, double& gmax2, const Red& red,
                         const NbrList& nb, bool listed) {
    double e = 0.0, gm = 0.0;
    const int t = threadIdx.x;
    const int w = !listed || 2 * n > min(PT, 2 * kPS) ? 1 : (4 * n > PT ? 2 : (8 * n > PT ? 4 : 8));
    if (w == 1) {
        for (int i = t; i < n; i += PT) {
            const double3 p = q[i];
            const double2 pc = cs[i];
            double gx = 0, gy = 0, ga = 0;
            const Sh<double> T = red.terms + i * kTerms;
            int nt = 0;
            auto term = [&](double v) {
                if (v != 0.0) {
                    if (nt < kTerms) T[nt] = v;
                    nt = min(nt + 1, kTerms + 1);
                }
            };
            term(wall_smooth(p.x, p.y, pc.x, pc.y, L, gx, gy, ga));
            const int m = listed ? nb.cnt[i] : n;
            for (int k = 0; k < m; ++k) {
                const int j = listed ? (int)nb.idx[i * kNbK + k] : k;
                if (j == i) continue;
                const double3 o = q[j];
                const double2 oc = cs[j];
                double hx = 0, hy = 0, ha = 0;
                const double pe = pair_smooth(p.x, p.y, pc.x, pc.y, o.x, o.y, oc.x, oc.y, hx, hy, ha);
                if (j > i) term(pe);
                gx += hx;
                gy += hy;
                ga += ha;
            }
            red.nterm[i] = (uint8_t)nt;
            g[i] = make_double3(gx, gy, ga);
            gm = fmax(gm, gx * gx + gy * gy);
        }
        __syncthreads();
        for (int i = t; t < kPS && i < n; i += kPS) {
            const int nt = red.nterm[i];
            if (nt > kTerms) {
                e = add_square(e, i, n, q, cs, L, nb, listed);
                continue;
            }
            for (int k = 0; k < nt; ++k) e += red.terms[i * kTerms + k];
        }
    } else {
        const int i = t / w, l = t % w, lane = t & 31, base = lane - l;
        double gx = 0, gy = 0, ga = 0, ei = 0;
        double3 p = make_double3(0, 0, 0);
        double2 pc = make_double2(1, 0);
        int m = 0;
        if (i < n) {
            p = q[i];
            pc = cs[i];
            ei += wall_smooth(p.x, p.y, pc.x, pc.y, L, gx, gy, ga);
            m = nb.cnt[i];
        }
        const int most = __reduce_max_sync(0xffffffffu, m);
        for (int k0 = 0; k0 < most; k0 += w) {
            double hx = 0, hy = 0, ha = 0, pe = 0;
            int j = -1;
            if (k0 + l < m) {
                j = nb.idx[i * kNbK + k0 + l];
                const double3 o = q[j];
                const double2 oc = cs[j];
                pe = pair_smooth(p.x, p.y, pc.x, pc.y, o.x, o.y, oc.x, oc.y, hx, hy, ha);
            }
            // the lanes with a nonzero term, in order
            unsigned hit = __ballot_sync(0xffffffffu, pe > 0.0) >> base & ((1u << w) - 1u);
            const int rounds = __reduce_max_sync(0xffffffffu, __popc(hit));
            for (int r = 0; r < rounds; ++r) {
                const int src = base + (hit ? __ffs(hit) - 1 : 0);
                const double ax = __shfl_sync(0xffffffffu, hx, src), ay = __shfl_sync(0xffffffffu, hy, src);
                const double aa = __shfl_sync(0xffffffffu, ha, src), ae = __shfl_sync(0xffffffffu, pe, src);
                const int aj = __shfl_sync(0xffffffffu, j, src);
                if (hit) {
                    gx += ax;
                    gy += ay;
                    ga += aa;
                    if (aj > i) ei += ae;
                    hit &= hit - 1;
                }
            }
        }
        if (i < n && l == 0) {
            g[i] = make_double3(gx, gy, ga);
            red.es[i] = ei;
            gm = gx * gx + gy * gy;
        }
        __syncthreads();
        e = t < n ? red.es[t] : 0.0;
    }
    for (int o = 16; o > 0; o >>= 1) {
        e += __shfl_xor_sync(0xffffffffu, e, o);
        gm = fmax(gm, __shfl_xor_sync(0xffffffffu, gm, o));
    }
    if ((t & 31) == 0) {
        if (t < kPS) red.e[t >> 5] = e;
        red.m[t >> 5] = gm;
    }
    __syncthreads();
    double s = 0.0, mx = 0.0;
    for (int k = 0; k < min(kPS, PT) / 32; ++k) s += red.e[k];  // (a narrow CTA's squares are all in these)
    for (int k = 0; k < PT / 32; ++k) mx = fmax(mx, red.m[k]);
    gmax2 = mx;
    return s;
}

// Certified side of q (dilation lambda, bounding box of the dilated state).
template <int PT>
__device__ double cert_side_all(int n, Sh<double3> q, Sh<double2> cs, const Cells& c, Sh<double> red,
                                double& lam_out, double& x0, double& y0) {
    double lam = 1.0;
    for (int i = threadIdx.x; i < n; i += PT) {
        const double3 p = q[i];
        const double ci = cs[i].x, si = cs[i].y;
        const int cx = c.cx(p), cy = c.cy(p);
        const int xa = max(cx - 1, 0), xb = min(cx + 1, c.G - 1);
        for (int yy = max(cy - 1, 0); yy <= min(cy + 1, c.G - 1); ++yy) {
            for (int k = c.start[yy * c.G + xa]; k < c.start[yy * c.G + xb + 1]; ++k) {
                const int j = c.order[k];
                if (j <= i) continue;
                const double dx = p.x - q[j].x, dy = p.y - q[j].y;
                if (dx * dx + dy * dy >= 2.05) continue;
                const double cj = cs[j].x, sj = cs[j].y;
                const double c12 = fabs(ci * cj + si * sj), s12 = fabs(-si * cj + ci * sj);
                const double r = 0.5 + 0.5 * (c12 + s12);
                const double v = fmax(fmax(fabs(dx * ci + dy * si), fabs(-dx * si + dy * ci)),
                                      fmax(fabs(dx * cj + dy * sj), fabs(-dx * sj + dy * cj)));
                lam = fmax(lam, v > 1e-12 ? (r + 2.6e-8) / v : 1e9);
            }
        }
    }
    lam = block_max<PT>(lam, red);
    lam_out = lam;
    if (lam > 1.008) return 1e30;
    double a0 = 1e300, a1 = -1e300, b0 = 1e300, b1 = -1e300;
    for (int i = threadIdx.x; i < n; i += PT) {
        const double r = 0.5 * (fabs(cs[i].x) + fabs(cs[i].y));
        const double x = q[i].x * lam, y = q[i].y * lam;
        a0 = fmin(a0, x - r);
        a1 = fmax(a1, x + r);
        b0 = fmin(b0, y - r);
        b1 = fmax(b1, y + r);
    }
    x0 = -block_max<PT>(-a0, red);
    const double xm = block_max<PT>(a1, red);
    y0 = -block_max<PT>(-b0, red);
    const double ym = block_max<PT>(b1, red);
    return fmax(xm - x0, ym - y0);
}

__device__ __forceinline__ double wrap_q(double a) {
    if (!(fabs(a) < 1.57079632679489661923)) a = fmod(a, 1.57079632679489661923);  // fmod(a, b) is a below b
    return a < 0.0 ? a + 1.57079632679489661923 : a;
}

template <int PT>
__device__ void trig_of(int n, Sh<double3> q, Sh<double2> cs) {
    for (int i = threadIdx.x; i < n; i += PT) {
        double s, c;
        sincos(q[i].z, &s, &c);
        cs[i] = make_double2(c, s);
    }
    __syncthreads();
}

// Shared-memory views of one polish CTA.
struct PolishBufs {
    Sh<double3> q0;  // accepted state of the descent
    Sh<double3> q;   // trial state
    Sh<double3> g;   // gradient at q0
    Sh<double3> tg;  // gradient at q
    Sh<double3> sv;  // best so far (translated, dilated)
    Sh<double2> cs;  // cos/sin of the state being evaluated
    Sh<double> max;  // [kWideT / 32] partials of block_max
    NbrList nb;   // neighbour list of the descent
    Cells cells;
    Red red;
};

// The evaluation's share of the layout (from `off` on), then the polish's.
constexpr int kRedDoubles = kPS / 32 + 2 * (kWideT / 32) + kPS;
__device__ __forceinline__ int eval_bufs(int off, int n, Red& red, NbrList& nb, Cells& cells) {
    red.e = Sh<double>{off};
    red.m = red.e + kPS / 32;
    red.es = red.m + 2 * (kWideT / 32);  // (block_max's partials lie between)
    red.terms = red.es + kPS;
    cells.start = Sh<int>{red.terms.off + 8 * kTerms * n};
    nb.idx = Sh<uint16_t>{cells.start.off + 4 * (kCG * kCG + 1)};
    cells.order = nb.idx + n * kNbK;
    nb.cnt = Sh<uint8_t>{cells.order.off + 2 * n};
    red.nterm = nb.cnt + n;
    return red.nterm.off + n;
}
constexpr size_t eval_bytes(size_t n) {
    return 8 * kRedDoubles + n * (8 * kTerms + 2 * kNbK + 2 + 2) + (kCG * kCG + 1) * 4;
}

__device__ __forceinline__ PolishBufs polish_bufs(int n) {
    PolishBufs b;
    b.cs = Sh<double2>{0};
    b.q0 = Sh<double3>{16 * n};
    b.q = b.q0 + n;
    b.g = b.q + n;
    b.tg = b.g + n;
    b.sv = b.tg + n;
    eval_bufs(b.sv.off + 24 * n, n, b.red, b.nb, b.cells);
    b.max = b.red.m + kWideT / 32;
    return b;
}

// q0, q, g, tg, sv (double3), cs (double2), and the evaluation's
size_t polish_smem_bytes(int n) { return (size_t)n * (5 * 24 + 16) + eval_bytes(n) + 16; }

// Descend the energy of state q0 (inside [0, Lt] up to its overhang) at side
// Lt until it vanishes (at most *budget gradient steps, each with up to 8
// backtracking trials).  Ends with the cells and trig of q0.
template <int PT>
__device__ void descend(int n, PolishBufs& B, double Lt, int* budget) {
    trig_of<PT>(n, B.q0, B.cs);
    build_cells<PT>(n, B.cells, B.q0, 0.0, 0.0, Lt);
    bool listed = build_nbr<PT>(n, B.nb, B.cells, B.q0);
    double gm2;
    double E = energy<PT>(n, B.q0, B.cs, Lt, B.g, gm2, B.red, B.nb, listed);
    double gmax = sqrt(gm2);
    double moved_by = 0.0;  // bound on any centre's distance from where the list was built
    double alpha = 0.05;
    while (*budget > 0 && E > 1e-26) {
        --*budget;
        bool moved = false;
        for (int ls = 0; ls < 8 && !moved; ++ls) {
            for (int i = threadIdx.x; i < n; i += PT) {
                const double3 p = B.q0[i], d = B.g[i];
                const double3 v = make_double3(p.x - alpha * d.x, p.y - alpha * d.y, wrap_q(p.z - alpha * d.z));
                double s, c;
                sincos(v.z, &s, &c);
                B.q[i] = v;
                B.cs[i] = make_double2(c, s);
            }
            __syncthreads();
            const double step = alpha * gmax;
            bool rebuilt = false;
            if (!(moved_by + step <= kNbMove)) {  // past the list's reach: a list of the trial itself
                build_cells<PT>(n, B.cells, B.q, 0.0, 0.0, Lt);
                listed = build_nbr<PT>(n, B.nb, B.cells, B.q);
                rebuilt = true;
            }
            const double En = energy<PT>(n, B.q, B.cs, Lt, B.tg, gm2, B.red, B.nb, listed);
            if (En < E) {
                E = En;
                moved = true;
                alpha = fmin(alpha * 1.5, 0.5);
                moved_by = rebuilt ? 0.0 : moved_by + step;
                gmax = sqrt(gm2);
                Sh<double3> s = B.q0;
                B.q0 = B.q;
                B.q = s;
                s = B.g;
                B.g = B.tg;
                B.tg = s;
            } else {
                alpha *= 0.3;
                if (rebuilt) moved_by = step;
            }
        }
        if (!moved) break;
    }
    __syncthreads();
    trig_of<PT>(n, B.q0, B.cs);
    build_cells<PT>(n, B.cells, B.q0, 0.0, 0.0, Lt);
}

// Compress-and-descend attempts on the certified state sv of side *Lb
// (delta shrinking by 0.3 after every attempt that does not certify a
// smaller side); sv and *Lb are updated in place.
template <int PT>
__device__ void polish_loop(int n, PolishBufs& B, double* Lb, int* budget, Sh<double> red) {
    double delta = 1e-4;
    for (int attempt = 0; attempt < 12 && *budget > 0 && delta > 1e-9; ++attempt) {
        const double f = 1.0 - delta, Lt = *Lb * f;
        for (int i = threadIdx.x; i < n; i += PT) B.q0[i] = make_double3(B.sv[i].x * f, B.sv[i].y * f, B.sv[i].z);
        __syncthreads();
        descend<PT>(n, B, Lt, budget);
        double lam = 0, x0 = 0, y0 = 0;
        const double Lc = cert_side_all<PT>(n, B.q0, B.cs, B.cells, red, lam, x0, y0);
        if (Lc < *Lb) {
            *Lb = Lc;
            for (int i = threadIdx.x; i < n; i += PT)
                B.sv[i] = make_double3(B.q0[i].x * lam - x0, B.q0[i].y * lam - y0, B.q0[i].z);
            __syncthreads();
        } else {
            delta *= 0.3;
        }
    }
}

template <int PT>
__global__ void __launch_bounds__(PT, kResident<PT>) polish_kernel(const int32_t* __restrict__ job_list,
                                                     const JobDev* __restrict__ jdev, JobMut* __restrict__ jmut,
                                                     double* __restrict__ best) {
    const int job = job_list[blockIdx.x];
    const JobDev jd = jdev[job];
    const int n = jd.n;
    double Lb = jmut[job].best_L;
    if (jd.polish_iters <= 0 || Lb >= 1e29 || jmut[job].status < 0) return;
    PolishBufs B = polish_bufs(n);
    const Sh<double> red = B.max;
    double* b = best + jd.best_off;
    for (int i = threadIdx.x; i < n; i += PT) B.sv[i] = make_double3(b[3 * i], b[3 * i + 1], b[3 * i + 2]);
    __syncthreads();
    int budget = jd.polish_iters;
    polish_loop<PT>(n, B, &Lb, &budget, red);
    for (int i = threadIdx.x; i < n; i += PT) {
        b[3 * i] = B.sv[i].x;
        b[3 * i + 1] = B.sv[i].y;
        b[3 * i + 2] = B.sv[i].z;
    }
    if (threadIdx.x == 0) jmut[job].best_L = Lb;
}

// Standalone polish of arbitrary states (state k: n_of[k] rows at
// xya + 3 * row0[k], polished in place).  The input's dilation-certified
// side is the incumbent; an input too overlapped to certify (dilation above
// 1.008) first descends its energy inside its own bounding box and, if
// overlaps remain, has its centres spread by that dilation (at most 1.5x)
// and descends in a box scaled alike.
// res[k] = {L_in, L_out, iterations used}.  CTA b takes state order[b] (b when order is null).
template <int PT>
__global__ void __launch_bounds__(PT, kResident<PT>) polish_states_kernel(const int32_t* __restrict__ order,
                                                            const int32_t* __restrict__ n_of,
                                                            const int64_t* __restrict__ row0, int iters,
                                                            double* __restrict__ xya, double* __restrict__ res) {
    const int k = order ? order[blockIdx.x] : (int)blockIdx.x;
    const int n = n_of[k];
    double* st = xya + 3 * row0[k];
    PolishBufs B = polish_bufs(n);
    const Sh<double> red = B.max;
    for (int i = threadIdx.x; i < n; i += PT) B.q0[i] = make_double3(st[3 * i], st[3 * i + 1], wrap_q(st[3 * i + 2]));
    __syncthreads();
    trig_of<PT>(n, B.q0, B.cs);
    int budget = iters;
    double lam = 0, x0 = 0, y0 = 0;
    // bounding box of the input
    double a0 = 1e300, a1 = -1e300, b0 = 1e300, b1 = -1e300;
    for (int i = threadIdx.x; i < n; i += PT) {
        const double r = 0.5 * (fabs(B.cs[i].x) + fabs(B.cs[i].y));
        a0 = fmin(a0, B.q0[i].x - r);
        a1 = fmax(a1, B.q0[i].x + r);
        b0 = fmin(b0, B.q0[i].y - r);
        b1 = fmax(b1, B.q0[i].y + r);
    }
    a0 = -block_max<PT>(-a0, red);
    a1 = block_max<PT>(a1, red);
    b0 = -block_max<PT>(-b0, red);
    b1 = block_max<PT>(b1, red);
    const double side = fmax(a1 - a0, b1 - b0);
    build_cells<PT>(n, B.cells, B.q0, a0, b0, side);
    double Lb = cert_side_all<PT>(n, B.q0, B.cs, B.cells, red, lam, x0, y0);
    const double L_in = Lb, lam_in = lam;
    if (Lb >= 1e29) {
        // translated to the origin, with the bounding box as the side
        for (int i = threadIdx.x; i < n; i += PT) {
            B.sv[i] = make_double3(B.q0[i].x - a0, B.q0[i].y - b0, B.q0[i].z);  // the input, at the origin
            B.q0[i] = B.sv[i];
        }
        __syncthreads();
        // first remove the overlaps inside the input's own bounding box (half
        // the budget); where they do not vanish there, spread the input's
        // centres by the dilation that would separate its close pairs (at
        // most 1.5x) and descend in a box scaled alike
        int half = budget / 2;
        budget -= half;
        descend<PT>(n, B, side, &half);
        budget += half;
        Lb = cert_side_all<PT>(n, B.q0, B.cs, B.cells, red, lam, x0, y0);
        if (Lb >= 1e29) {
            const double f = fmin(fmax(lam_in, 1.0), 1.5);
            for (int i = threadIdx.x; i < n; i += PT)
                B.q0[i] = make_double3(B.sv[i].x * f, B.sv[i].y * f, B.sv[i].z);
            __syncthreads();
            descend<PT>(n, B, side * f, &budget);
            Lb = cert_side_all<PT>(n, B.q0, B.cs, B.cells, red, lam, x0, y0);
        }
    }
    if (Lb < 1e29) {
        for (int i = threadIdx.x; i < n; i += PT)
            B.sv[i] = make_double3(B.q0[i].x * lam - x0, B.q0[i].y * lam - y0, B.q0[i].z);
        __syncthreads();
        polish_loop<PT>(n, B, &Lb, &budget, red);
        for (int i = threadIdx.x; i < n; i += PT) {
            st[3 * i] = B.sv[i].x;
            st[3 * i + 1] = B.sv[i].y;
            st[3 * i + 2] = B.sv[i].z;
        }
    }
    if (threadIdx.x == 0) {
        res[3 * k] = L_in;
        res[3 * k + 1] = Lb;
        res[3 * k + 2] = (double)(iters - budget);
    }
}

// FP64 energy and gradient of arbitrary states, one CTA per state: the
// polish's own energy function over a neighbour list (all pairs, bit for
// bit), with cos and sin taken of the angles as given.  State k has n_of[k]
// rows at xya + 3 * row0[k] and side side[k]; energy[k], and the gradient rows
// at the same offsets of grad when grad is not null; order as above.
template <int PT>
__global__ void __launch_bounds__(PT, kResident<PT>) energy_states_kernel(const int32_t* __restrict__ order,
                                                            const int32_t* __restrict__ n_of,
                                                            const int64_t* __restrict__ row0,
                                                            const double* __restrict__ side,
                                                            const double* __restrict__ xya,
                                                            double* __restrict__ energy_out,
                                                            double* __restrict__ grad) {
    const int k = order ? order[blockIdx.x] : (int)blockIdx.x;
    const int n = n_of[k];
    const Sh<double2> cs{0};
    const Sh<double3> q{16 * n}, g = q + n;
    Red red;
    NbrList nb;
    Cells cells;
    eval_bufs(g.off + 24 * n, n, red, nb, cells);
    const double* st = xya + 3 * row0[k];
    for (int i = threadIdx.x; i < n; i += PT) q[i] = make_double3(st[3 * i], st[3 * i + 1], st[3 * i + 2]);
    __syncthreads();
    trig_of<PT>(n, q, cs);
    build_cells<PT>(n, cells, q, 0.0, 0.0, side[k]);
    const bool listed = build_nbr<PT>(n, nb, cells, q);
    double gm2;
    const double e = energy<PT>(n, q, cs, side[k], g, gm2, red, nb, listed);
    if (threadIdx.x == 0) energy_out[k] = e;
    if (grad) {
        double* go = grad + 3 * row0[k];
        for (int i = threadIdx.x; i < n; i += PT) {
            go[3 * i] = g[i].x;
            go[3 * i + 1] = g[i].y;
            go[3 * i + 2] = g[i].z;
        }
    }
}

size_t energy_smem_bytes(int n) { return (size_t)n * (2 * sizeof(double3) + sizeof(double2)) + eval_bytes(n) + 16; }

// Launches of a batch whose sizes n[0 .. count) descend, or of any order up to
// one CTA an SM: launch(width tag, stream, first, count, largest n).
// Up to one packing an SM each has an SM to itself and takes the widest CTA
// (64 of n 5..1000 x 200 steps: 7.8 ms with 256 threads and all-pairs lists,
// 3.2 now).  Beyond that a wide CTA leaves most of its threads and registers
// idle on a small packing while others wait, so the width goes by size, each
// class with the shared memory of its own largest, side by side and the
// longest first: 1,000 of n <= 30 x 100 steps took 4.9 ms a call with 512
// threads for all and 3.3 now, 444 of n = 250 4.2 and 3.8, 300 of n 5..1000
// 3.4 and 3.0.
template <class Launch>
static int launch_widths(sqs_ctx* ctx, const std::vector<int32_t>& n, Launch&& launch) {
    const int count = (int)n.size();
    if (count == 0) return SQS_OK;
    if (count <= ctx->sm_count)
        return launch(std::integral_constant<int, kWideT>{}, ctx->stream, 0, count, *std::max_element(n.begin(), n.end()));
    auto below = [&](int limit) {
        return (int)(std::partition_point(n.begin(), n.end(), [&](int32_t v) { return v > limit; }) - n.begin());
    };
    const int mid = below(kWidthN<kMidT>), small = below(kWidthN<kSmallT>);
    const bool fork = (mid > 0) + (small > mid) + (count > small) > 1;
    cudaStream_t s_mid = ctx->stream, s_small = ctx->stream;
    if (fork) {
        SQS_CUDA(cudaEventRecord(ctx->fork, ctx->stream));
        s_mid = ctx->aux[0];
        s_small = ctx->aux[1];
        for (int a = 0; a < 2; ++a) SQS_CUDA(cudaStreamWaitEvent(ctx->aux[a], ctx->fork, 0));
    }
    int rc = SQS_OK;
    if (mid > 0) rc = launch(std::integral_constant<int, kWideT>{}, ctx->stream, 0, mid, n[0]);
    if (!rc && small > mid)
        rc = launch(std::integral_constant<int, kMidT>{}, s_mid, mid, small - mid, n[(size_t)mid]);
    if (!rc && count > small)
        rc = launch(std::integral_constant<int, kSmallT>{}, s_small, small, count - small, n[(size_t)small]);
    if (fork) {  // join the side streams, also after a failed launch
        for (int a = 0; a < 2; ++a) {
            SQS_CUDA(cudaEventRecord(ctx->join[a], ctx->aux[a]));
            SQS_CUDA(cudaStreamWaitEvent(ctx->stream, ctx->join[a], 0));
        }
    }
    return rc;
}

std::vector<int32_t> width_order(sqs_ctx* ctx, std::vector<int32_t>& n) {
    std::vector<int32_t> order;
    if ((int)n.size() <= ctx->sm_count) return order;
    int32_t start[kMaxN + 2] = {0};  // counting sort, the largest first
    for (int32_t v : n) ++start[kMaxN - v + 1];
    for (int k = 1; k <= kMaxN + 1; ++k) start[k] += start[k - 1];
    order.resize(n.size());
    std::vector<int32_t> sorted(n.size());
    for (size_t k = 0; k < n.size(); ++k) {
        const int32_t at = start[kMaxN - n[k]]++;
        order[(size_t)at] = (int32_t)k;
        sorted[(size_t)at] = n[k];
    }
    n.swap(sorted);
    return order;
}

// Room for the largest dynamic shared memory, set once per device and kernel
// (idempotent if repeated).
template <class Kernel>
static int polish_attr(sqs_ctx* ctx, Kernel kernel, std::atomic<bool>* done) {
    if (!done[ctx->device & 63]) {
        SQS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 222 * 1024));
        done[ctx->device & 63] = true;
    }
    return SQS_OK;
}

int launch_energy_states(sqs_ctx* ctx, const std::vector<int32_t>& n, const int32_t* order, const int32_t* n_of,
                         const int64_t* row0, const double* side, const double* xya, double* energy_out, double* grad) {
    return launch_widths(ctx, n, [&](auto width, cudaStream_t st, int first, int count, int nmax) -> int {
        constexpr int PT = decltype(width)::value;
        static std::atomic<bool> done[64];
        if (int r = polish_attr(ctx, energy_states_kernel<PT>, done)) return r;
        energy_states_kernel<PT><<<count, PT, energy_smem_bytes(nmax), st>>>(order ? order + first : nullptr, n_of, row0,
                                                                             side, xya, energy_out, grad);
        SQS_CUDA(cudaGetLastError());
        ctx->launches += 1;
        return SQS_OK;
    });
}

int launch_polish_states(sqs_ctx* ctx, const std::vector<int32_t>& n, const int32_t* order, const int32_t* n_of,
                         const int64_t* row0, int iters, double* xya, double* res) {
    return launch_widths(ctx, n, [&](auto width, cudaStream_t st, int first, int count, int nmax) -> int {
        constexpr int PT = decltype(width)::value;
        static std::atomic<bool> done[64];
        if (int r = polish_attr(ctx, polish_states_kernel<PT>, done)) return r;
        polish_states_kernel<PT><<<count, PT, polish_smem_bytes(nmax), st>>>(order ? order + first : nullptr, n_of, row0,
                                                                             iters, xya, res);
        SQS_CUDA(cudaGetLastError());
        ctx->launches += 1;
        return SQS_OK;
    });
}

int launch_polish(sqs_ctx* ctx, const std::vector<int32_t>& n, const int32_t* job_list, const JobDev* jdev, JobMut* jmut,
                  double* best) {
    return launch_widths(ctx, n, [&](auto width, cudaStream_t st, int first, int count, int nmax) -> int {
        constexpr int PT = decltype(width)::value;
        static std::atomic<bool> done[64];
        if (int r = polish_attr(ctx, polish_kernel<PT>, done)) return r;
        polish_kernel<PT><<<count, PT, polish_smem_bytes(nmax), st>>>(job_list + first, jdev, jmut, best);
        SQS_CUDA(cudaGetLastError());
        ctx->launches += 1;
        return SQS_OK;
    });
}

}  // namespace ann
}  // namespace sqs
