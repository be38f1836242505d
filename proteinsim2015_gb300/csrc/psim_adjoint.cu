// psim_adjoint.cu -- gradients of a trajectory loss through the vGB step.
//
// The loss of the differentiable-trajectory workload is the squared distance
// between the time-averaged, Gaussian-smoothed g(r) of a trajectory and a
// target; its gradient with respect to the plugin parameters (and the
// initial positions) is taken with the noise held fixed, by an adjoint
// (reverse-time) recursion through the positions-only form of the vGB
// normal step (brownianIntegrator.cpp:225-296):
//
//   x_1     = x_0 + c_v v_0 + c_f F(x_0) + N_0                    (firstStep)
//   x_{t+1} = c0 x_t - a0 x_{t-1} + b1 F(x_t) - b2 F(x_{t-1}) + N_t
//
// with c0 = 1 + coEff0, a0 = coEff0, b1 = dt^2 (coEff1 + coEff2) / m,
// b2 = dt^2 coEff2 / m, c_v = coEff1 dt, c_f = coEff3 dt^2 / m, and N_t the
// noise terms (Philox-keyed by particle and step, as the system's).  Writing
// u_t = b1 lam_{t+1} - b2 lam_{t+2} (u_0 = c_f lam_1 - b2 lam_2) and J the
// force Jacobian (symmetric: F is minus a potential gradient),
//
//   lam_t  = dL/dx_t + c0 lam_{t+1} - a0 lam_{t+2} + J(x_t) u_t   (lam_0: 1, -a0)
//   dL/dth = sum_t u_t . dF/dth (x_t)
//
// A forward step is one launch (force and update), a reverse step one (J u,
// dF/dth . u and the loss's position gradient), both over one neighbour list kept for
// tens of steps.  The forward pass keeps the positions of its last K steps and a
// checkpoint (x_t, x_{t-1}, F(x_{t-1})) every K steps; the reverse pass goes back through
// the last segment as it stands and recomputes each earlier one from its checkpoint, so
// memory is (T/K + K) positions.  K is the caller's interval or, where that is longer,
// what 256 MB hold (kAdjTraj): a trajectory that fits is never computed twice.
// All sums are taken in an order that the positions decide: two runs agree bit for
// bit (but for the counts of more than 3072 bins, which are added as they come).  What bounds it is the FP64 unit: 33 FP64 operations a pair forward and ~65
// back with the lanes of an instruction 75% full at 32768 particles.  Gradient of 60
// steps, with a cell list and a thread per particle for every pass before, and now:
// 4096 particles 186 -> 5.6 ms, 32768 286 -> 22.8 ms (7.7 and 29.7 with each segment
// recomputed).
//
// All arithmetic is FP64 and the forward matches the system's plain form
// (same coefficients and Philox draws) up to rounding.  The pair force is the
// AO plugin (AOPotential.cpp:50-130), the Yukawa term of the LennardJones
// plugin with ljNum = 0 and the plugin's LJ(n) term (LJPotential.cpp:96-109),
// each inside its own cutoff; parameters th = (c1, c2, Y, lambda, eps,
// sigma): the AO coefficients, the Yukawa amplitude kT wellDepth
// yukawaStrength and its length, and the LJ energy kT wellDepth and contact
// diameter (the plugin's size, L = (sigma/r)^n).  The cutoffs are fixed: a
// pair crossing a cutoff changes the force by a step, which no derivative of
// the smooth part carries.
#include <cmath>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "../../include/psim_gb300.h"
#include "psim_exp.cuh"
#include "psim_kernels.cuh"

namespace psim {
namespace {

constexpr int kAdjTh = 6;    // parameters: c1, c2, Y, lambda, eps, sigma

struct AdjPair {
    double c1, c2, ao_rc2;   // ao_rc2 = 0: no AO term
    double Y, lam, y_rc2;    // y_rc2 = 0: no Yukawa term
    double inv_lam;          // 1 / lam
    double eps, sig, lj_rc2; // lj_rc2 = 0: no LJ(n) term
    int ljn;
    double eps4n, eps_n_sig; // 4n eps, n eps / sig
    const double2* e2;       // exp_table_values
};

// r2 < rc2 on the bit patterns (a NaN is above), off the FP64 unit
__device__ __forceinline__ bool below_rc(double r2, double rc2) {
    return __double_as_longlong(r2) < __double_as_longlong(rc2);
}

// s(r) = F_pair / r (force on i along x_j - x_i)
__device__ __forceinline__ double pair_s(const AdjPair& q, double r2) {
    const double ri = rsqrt64(r2), i2 = __dmul_rn(ri, ri), i3 = __dmul_rn(i2, ri);
    double s = 0.0;
    if (below_rc(r2, q.ao_rc2)) {
        const double i4 = __dmul_rn(i2, i2), i8 = __dmul_rn(i4, i4), i16 = __dmul_rn(i8, i8);
        const double i39 = __dmul_rn(__dmul_rn(__dmul_rn(i16, i16), i4), i3);
        s -= __fma_rn(36.0, i39, __fma_rn(q.c1, i2, q.c2));
    }
    if (below_rc(r2, q.y_rc2)) {
        const double r = __dmul_rn(r2, ri);
        const double e = exp_table(-r * q.inv_lam, q.e2);
        s = __fma_rn(-__dmul_rn(__dmul_rn(q.Y, e), __dadd_rn(q.lam, r)), i3, s);
    }
    if (below_rc(r2, q.lj_rc2)) {
        // fNet = -eps (2L - 1) 4n L / r, L = (sigma / r)^n
        const double L = powi_binary(__dmul_rn(q.sig, ri), q.ljn);
        s = __fma_rn(-__dmul_rn(__dmul_rn(q.eps4n, L), __fma_rn(2.0, L, -1.0)), i2, s);
    }
    return s;
}

// s, ds/dr and, added to th, dui ds/dth; returns 1/r
__device__ __forceinline__ double pair_all(const AdjPair& q, double r2, double dui, double& s,
                                           double& ds, double th[kAdjTh]) {
    const double ri = rsqrt64(r2), i2 = __dmul_rn(ri, ri), i3 = __dmul_rn(i2, ri);
    s = 0.0;
    ds = 0.0;
    if (below_rc(r2, q.ao_rc2)) {
        const double i4 = __dmul_rn(i2, i2), i8 = __dmul_rn(i4, i4), i16 = __dmul_rn(i8, i8);
        const double i39 = __dmul_rn(__dmul_rn(__dmul_rn(i16, i16), i4), i3);
        s -= __fma_rn(36.0, i39, __fma_rn(q.c1, i2, q.c2));
        ds += __fma_rn(36.0 * 39.0, __dmul_rn(i39, ri), 2.0 * q.c1 * i3);
        th[0] = __fma_rn(-i2, dui, th[0]);
        th[1] -= dui;
    }
    if (below_rc(r2, q.y_rc2)) {
        // s = -Y e^{-r/lam} (lam + r) / r^3
        const double r = __dmul_rn(r2, ri);
        const double e3 = __dmul_rn(exp_table(-r * q.inv_lam, q.e2), i3);
        const double lr = __dadd_rn(q.lam, r), Ye3 = __dmul_rn(q.Y, e3), w = __dmul_rn(e3, lr);
        const double rl = __dmul_rn(r, q.inv_lam);
        s = __fma_rn(-Ye3, lr, s);
        ds = __fma_rn(Ye3, __fma_rn(3.0, __dmul_rn(lr, ri), rl), ds);
        th[2] = __fma_rn(-w, dui, th[2]);
        th[3] = __fma_rn(-__dmul_rn(Ye3, dui), __fma_rn(rl, __dmul_rn(lr, q.inv_lam), 1.0), th[3]);
    }
    if (below_rc(r2, q.lj_rc2)) {
        // fNet = -eps (2L - 1) 4n L / r, L = (sigma / r)^n: s = -4n eps (2L - 1) L / r^2,
        // ds/dr = 4n eps L (n (4L - 1) + 2 (2L - 1)) / r^3,
        // ds/dsigma = -4n^2 eps (4L - 1) L / (sigma r^2)
        const double n = (double)q.ljn;
        const double L = powi_binary(__dmul_rn(q.sig, ri), q.ljn);
        const double b = __dmul_rn(__dmul_rn(4.0 * n, L), i2), l2 = __fma_rn(2.0, L, -1.0),
                     l4 = __fma_rn(4.0, L, -1.0);
        s = __fma_rn(-__dmul_rn(q.eps, b), l2, s);
        ds = __fma_rn(__dmul_rn(q.eps, __dmul_rn(b, ri)), __fma_rn(n, l4, 2.0 * l2), ds);
        th[4] = __fma_rn(-__dmul_rn(b, l2), dui, th[4]);
        th[5] = __fma_rn(-__dmul_rn(q.eps_n_sig, __dmul_rn(b, l4)), dui, th[5]);
    }
    return ri;
}

// ------------------------------------------------------- the neighbour list
//
// Every pass walks one list of the pairs within the largest distance any of them
// needs (the cutoffs, or the g(r) reach) plus a skin, kept while no particle has
// moved skin/2 since it was built -- about 30 steps at dt = 1e-3 -- where each pass
// would otherwise sort the particles and test the 27 cells around each.  Particles are
// held in the cell order of the initial positions (`order`: original index of each
// slot), which keeps the gathers of a list close together, and as double4
// positions (one 256-bit gather) with a float4 copy that the distance test
// reads.  A list's entries are slots, in an order that only the positions
// decide, so every sum of the sweeps is the same from run to run.

struct AdjGrid {
    double L, inv_cs;
    int s, s2, ncell;   // s < 3: no grid, the build tests every pair
};

__device__ __forceinline__ int cell_of(double xw, const AdjGrid& g) {
    int c = (int)(xw * g.inv_cs);
    return c < 0 ? 0 : (c >= g.s ? g.s - 1 : c);
}

// Positions x (and the step before, xp) moved into the box by whole boxes, which the
// recursion x_{t+1} = c0 x_t - a0 x_{t-1} + ... carries along (c0 - a0 = 1), counted
// in img; the float copy and the cell of each.
__global__ void __launch_bounds__(256)
adj_rebase_kernel(int n, double4_32a* x, double4_32a* xp, float4* xf, float4* xbuild, AdjGrid g,
                  int* img, int* key, int* rank, int* count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4_32a a = x[i];
    double v[3] = {a.x, a.y, a.z};
    int k = 0, mul = 1;
    bool moved = false;
    double sh[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double m = floor(v[d] / g.L);
        sh[d] = g.L * m;
        if (m != 0.0) {
            v[d] -= sh[d];
            moved = true;
            if (img) img[3 * i + d] += (int)m;
        }
        k += mul * cell_of(v[d], g);
        mul *= g.s;
    }
    if (moved) {
        x[i] = make_double4_32a(v[0], v[1], v[2], 0.0);
        double4_32a p = xp[i];
        xp[i] = make_double4_32a(p.x - sh[0], p.y - sh[1], p.z - sh[2], 0.0);
    }
    const float4 f = make_float4((float)v[0], (float)v[1], (float)v[2], 0.f);
    xf[i] = f;
    xbuild[i] = f;
    key[i] = k;
    rank[i] = atomicAdd(&count[k], 1);
}

__global__ void __launch_bounds__(256) adj_scatter_kernel(int n, const int* key, const int* rank,
                                                          const int* start, int* tmp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) tmp[start[key[i]] + rank[i]] = i;
}

// cell order, by index inside a cell: sorted[p] = i, and its float position with
// the index in .w
__global__ void __launch_bounds__(256) adj_sort_kernel(int n, const int* tmp, const int* key,
                                                       const int* start, const int* count,
                                                       const float4* xf, float4* sorted,
                                                       int* order) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int i = tmp[p], c = key[i], st = start[c], cnt = count[c];
    int r = 0;
    for (int q = st; q < st + cnt; ++q) r += tmp[q] < i ? 1 : 0;
    if (order) order[st + r] = i;
    if (sorted) {
        float4 f = xf[i];
        f.w = __int_as_float(i);
        sorted[st + r] = f;
    }
}

// slot i's list: entries [i stride, i stride + count[i])
struct AdjList {
    const int* count;
    const int* entry;
    int stride;
};

// d shifted by whole boxes to the nearest image
__device__ __forceinline__ float near_image(float d, float L, float inv_L) {
    return fmaf(-L, rintf(d * inv_L), d);
}

constexpr int kAdjBuildLanes = 8;

// Eight lanes a particle over the rows of cells around it (or every particle):
// the neighbours within sqrt(R2), counted (and the most of a particle), or written
// in the order of the sorted list.
template <bool kFill>
__global__ void __launch_bounds__(256)
adj_list_kernel(int n, AdjGrid g, const float4* sorted, const int* key, const int* cstart,
                const int* ccount, float R2, int* lcount, int* entry, int stride, int* most) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const int p = t / kAdjBuildLanes, m = t % kAdjBuildLanes;
    const bool active = p < n;
    const float Lf = (float)g.L, inv_L = 1.0f / Lf;
    const uint32_t below = (1u << m) - 1u;
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
    int i = 0, cx = 0, cy = 0, cz = 0, cnt = 0;
    size_t base = 0;
    if (active) {
        h = sorted[p];
        i = __float_as_int(h.w);
        const int c = key[i];
        cx = c % g.s;
        cy = (c / g.s) % g.s;
        cz = c / g.s2;
        if (kFill) base = (size_t)i * stride;
    }
    const int rows = g.s < 3 ? 1 : 9;
    for (int row = 0; row < rows; ++row) {
        int sh;
        const int y = wrap_near(cy + row % 3 - 1, g.s, sh), z = wrap_near(cz + row / 3 - 1, g.s, sh);
        for (int part = 0; part < 2; ++part) {
            int a = 0, len = 0;
            if (active && g.s < 3) {
                len = part == 0 ? n : 0;
            } else if (active) {
                const int c0 = g.s * y + g.s2 * z;
                if (part == 0) {
                    const int xa = max(cx - 1, 0), xb = min(cx + 1, g.s - 1);
                    a = cstart[c0 + xa];
                    len = cstart[c0 + xb] + ccount[c0 + xb] - a;
                } else if (cx == 0 || cx == g.s - 1) {
                    const int xw = cx == 0 ? g.s - 1 : 0;
                    a = cstart[c0 + xw];
                    len = ccount[c0 + xw];
                }
            }
            const int lmax = __reduce_max_sync(0xffffffffu, len);
            for (int t0 = 0; t0 < lmax; t0 += kAdjBuildLanes) {
                const int q = a + t0 + m;
                bool in = t0 + m < len && q != p;
                int j = 0;
                if (in) {
                    const float4 f = sorted[q];
                    const float ex = near_image(f.x - h.x, Lf, inv_L),
                                ey = near_image(f.y - h.y, Lf, inv_L),
                                ez = near_image(f.z - h.z, Lf, inv_L);
                    in = ex * ex + ey * ey + ez * ez < R2;
                    j = __float_as_int(f.w);
                }
                const uint32_t bits =
                    __ballot_sync(0xffffffffu, in) >> (lane & 24) & 255u;
                if (kFill && in) entry[base + cnt + __popc(bits & below)] = j;
                cnt += __popc(bits);
            }
        }
    }
    if (!kFill) {
        if (active && m == 0) lcount[i] = cnt;
        const int top = __reduce_max_sync(0xffffffffu, cnt);
        if (lane == 0) atomicMax(most, top);
    }
}

// ------------------------------------------------------------- the list walk
//
// G lanes a particle.  They test G entries at a time in FP32 (with a margin for
// the rounding) and queue the ones in range, each at its rank in the lanes'
// ballot; lane m evaluates queue entries m, m + G, ... in FP64.  The sweeps are
// bound by the FP64 unit, which takes as long over an instruction with one lane as
// with 32, so what is evaluated is packed and what is tested is not in FP64.

constexpr int kAdjWarps = 2;     // warps per block of the sweeps
constexpr int kAdjQueue = 96;    // queue entries per particle
constexpr int kAdjStride = kAdjQueue + 4;

struct AdjWalk {
    AdjPair q;
    AdjList list;
    int n;
    const double4_32a* x;   // positions of the step, within skin/2 of the box
    const float4* xf;
    double L, half;
    int t;                  // the step whose positions these are
    const int* bad;         // first step with a particle beyond skin/2 of the build
};

// fn(j, d, r2) for every neighbour j of slot i with r2 < rc2; kAll: fn(ok, r2) by all
// lanes together, ok where a lane has such a neighbour
template <int G, bool kAll = false, class Fn>
__device__ __forceinline__ void for_pairs(const AdjWalk& w, double rc2, int i, bool active,
                                          int lane, const double4_32a& xi, uint32_t* q, Fn&& fn) {
    constexpr int U = 2;
    const int m = lane % G;
    const uint32_t below = (1u << m) - 1u;
    constexpr uint32_t kMask = G == 32 ? ~0u : (1u << G) - 1u;
    const float Lf = (float)w.L, inv_L = 1.0f / Lf;
    const float rcf = (float)sqrt(rc2) + 1e-3f + 4e-6f * Lf, pre = rcf * rcf;
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
    const int* e = w.list.entry;
    int len = 0;
    if (active) {
        h = w.xf[i];
        e += (size_t)i * w.list.stride;
        len = w.list.count[i];
    }
    int cnt = 0, done = 0;
    auto drain = [&]() {
        __syncwarp();   // the lanes' entries are written
        const int last = __reduce_max_sync(0xffffffffu, cnt);
        int k = (m - done) & (G - 1);
        for (int it = 0; it < last; it += G, k += G) {
            double r2 = 0.0;
            bool ok = false;
            if (k < cnt) {
                const int j = (int)q[k];
                const double4_32a xj = w.x[j];
                double d[3] = {xj.x - xi.x, xj.y - xi.y, xj.z - xi.z};
                const int hh = __double2hiint(w.half);
                if ((__double2hiint(d[0]) & 0x7fffffff) > hh ||
                    (__double2hiint(d[1]) & 0x7fffffff) > hh ||
                    (__double2hiint(d[2]) & 0x7fffffff) > hh) {
                    // keeps the compiler from doing the additions for every pair
                    asm volatile("" : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]));
#pragma unroll
                    for (int a = 0; a < 3; ++a)
                        if (fabs(d[a]) > w.half) d[a] = d[a] < 0.0 ? d[a] + w.L : d[a] - w.L;
                }
                r2 = __fma_rn(d[2], d[2], __fma_rn(d[1], d[1], __dmul_rn(d[0], d[0])));
                ok = below_rc(r2, rc2);
                if constexpr (!kAll)
                    if (ok) fn(j, d, r2);
            }
            if constexpr (kAll) fn(ok, r2);
        }
        done += cnt;
        cnt = 0;
        __syncwarp();   // the entries are read
    };
    const int lmax = __reduce_max_sync(0xffffffffu, len);
    for (int t0 = 0; t0 < lmax; t0 += G * U) {
        int j[U];
        float4 f[U];
#pragma unroll
        for (int u = 0; u < U; ++u) j[u] = t0 + G * u + m < len ? __ldg(e + t0 + G * u + m) : -1;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (j[u] >= 0) f[u] = w.xf[j[u]];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float ex = near_image(f[u].x - h.x, Lf, inv_L),
                        ey = near_image(f[u].y - h.y, Lf, inv_L),
                        ez = near_image(f[u].z - h.z, Lf, inv_L);
            const bool in = j[u] >= 0 && ex * ex + ey * ey + ez * ez < pre;
            const uint32_t bits = __ballot_sync(0xffffffffu, in) >> (lane & ~(G - 1)) & kMask;
            if (in) q[cnt + __popc(bits & below)] = (uint32_t)j[u];
            cnt += __popc(bits);
        }
        if (__any_sync(0xffffffffu, cnt > kAdjQueue - G * U)) drain();
    }
    drain();
}

// the sum over a particle's G lanes, in every lane
template <int G>
__device__ __forceinline__ double lanes_sum(double v) {
#pragma unroll
    for (int k = 1; k < G; k <<= 1) v += __shfl_xor_sync(0xffffffffu, v, k);
    return v;
}
__device__ __forceinline__ double pick(int m, double a, double b, double c) {
    return m == 0 ? a : (m == 1 ? b : c);
}

struct AdjStep {
    int n;
    double c0, a0, b1, b2, cv, cf;
    double sig1, sig2, corr, dev, coeff0;
    uint32_t seed;
};

struct AdjForward {
    AdjStep c;
    const double4_32a* xp;    // x_{t-1}
    const double* Fp;         // F(x_{t-1})
    double* F;                // F(x_t) (out)
    const double* v0;
    double4_32a* xn;          // x_{t+1} (out)
    float4* xnf;
    const float4* xbuild;     // float positions at the list's build
    float disp2;              // (skin/2)^2, less the rounding of the test
    const int* order;
    int* bad;
};

// Step t -> t + 1: the pair force, then lane k < 3 updates axis k.  The noise
// memory is the draws of the step before, drawn again (Philox is a function of
// the step), so a step can be retaken from any stored position.  Each of
// four lanes makes one Philox call: groups 0 and 1 of step t and of step t - 1.
template <int G>
__global__ void __launch_bounds__(kAdjWarps * 32) adj_forward_kernel(AdjWalk w, double rc2,
                                                                     AdjForward a) {
    __shared__ uint32_t sq[kAdjWarps][32 / G][kAdjStride];
    if (*w.bad <= w.t) return;   // the list does not hold for x_t: the host takes the step again
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int i = (blockIdx.x * kAdjWarps + wid) * (32 / G) + lane / G, m = lane % G;
    const bool active = i < w.n;
    double4_32a xi = make_double4_32a(0.0, 0.0, 0.0, 0.0);
    if (active) xi = w.x[i];
    double f0 = 0.0, f1 = 0.0, f2 = 0.0;
    for_pairs<G>(w, rc2, i, active, lane, xi, sq[wid][lane / G],
                 [&](int, const double* d, double r2) {
                     const double s = pair_s(w.q, r2);
                     f0 = __fma_rn(s, d[0], f0);
                     f1 = __fma_rn(s, d[1], f1);
                     f2 = __fma_rn(s, d[2], f2);
                 });
    f0 = lanes_sum<G>(f0);
    f1 = lanes_sum<G>(f1);
    f2 = lanes_sum<G>(f2);
    // the Gaussians: z[0..3] of this lane's call
    const AdjStep& c = a.c;
    const uint32_t step = (uint32_t)w.t;
    float z[4];
    {
        const uint32_t tag = active ? (uint32_t)a.order[i] : 0u;
        const Philox4 r = philox4x32_10(step - (uint32_t)((m >> 1) & 1), (uint32_t)(m & 1), tag, 0u,
                                        c.seed, 0x5053494Du);
        box_muller(r.v[0], r.v[1], z[0], z[1]);
        box_muller(r.v[2], r.v[3], z[2], z[3]);
    }
    const int b = lane & ~(G - 1);
    float zz[4][4];
#pragma unroll
    for (int l = 0; l < 4; ++l)
#pragma unroll
        for (int k = 0; k < ((l & 1) ? 2 : 4); ++k) zz[l][k] = __shfl_sync(0xffffffffu, z[k], b + l);
    const bool mine = active && m < 3;
    const double F = pick(m, f0, f1, f2), x = pick(m, xi.x, xi.y, xi.z);
    // draws k and 3 + k of this step; the noise memory: draw 3 + k of the step
    // before, or draw k of step 0 (firstStep)
    const double xk = widen_f32(m == 0 ? zz[0][0] : (m == 1 ? zz[0][1] : zz[0][2]));
    const size_t o = 3 * (size_t)i + m;
    double xn = 0.0;
    if (!mine) {
    } else if (w.t == 0) {
        xn = x + c.cv * a.v0[o] + c.cf * F + c.sig1 * xk;
    } else {
        const double xm = widen_f32(m == 0 ? zz[0][3] : (m == 1 ? zz[1][0] : zz[1][1]));
        const float pm = w.t == 1 ? (m == 0 ? zz[2][0] : (m == 1 ? zz[2][1] : zz[2][2]))
                                  : (m == 0 ? zz[2][3] : (m == 1 ? zz[3][0] : zz[3][1]));
        const double mc = c.sig2 * (c.corr * widen_f32(pm) + c.dev * xk);
        const double xp = reinterpret_cast<const double*>(a.xp)[4 * (size_t)i + m];
        xn = c.c0 * x - c.a0 * xp + c.b1 * F - c.b2 * a.Fp[o] + c.sig1 * xm + c.coeff0 * mc;
    }
    float d2 = 0.f;   // |x_{t+1} - build|^2
    if (mine) {
        const float f = (float)xn;
        a.F[o] = F;
        reinterpret_cast<double*>(a.xn)[4 * (size_t)i + m] = xn;
        reinterpret_cast<float*>(a.xnf)[4 * (size_t)i + m] = f;
        const float e = f - reinterpret_cast<const float*>(a.xbuild)[4 * (size_t)i + m];
        d2 = e * e;
    }
    d2 += __shfl_xor_sync(0xffffffffu, d2, 1);
    d2 += __shfl_xor_sync(0xffffffffu, d2, 2);
    if (mine && d2 > a.disp2) atomicMin(a.bad, w.t + 1);
}

// smoothed g(r): Gaussian kernels at the bin centres, summed over ordered pairs
struct AdjHist {
    double r_min, dr, inv_sig, norm;   // norm: 1 / (sqrt(2 pi) sigma)
    double dz, qq, inv_dr;             // dr / sigma, e^{-dz^2}, 1 / dr
    int n_bins, reach;                 // bins within reach of a distance contribute
};

// The kernel values G_b = norm exp(-z_b^2 / 2) of distance r at the bins
// lo..hi, z_b = (r - r_b) / sigma, by the recurrence of consecutive bins
// (z_{b+1} = z_b - dz): G_{b+1} = G_b q_b, q_{b+1} = q_b e^{-dz^2},
// q_b = e^{dz z_b - dz^2 / 2} -- two exponentials per distance.
struct GaussBins {
    int lo, hi;     // no bin: lo > hi
    double z, G, q;
    // G starts at g times the kernel
    __device__ __forceinline__ GaussBins(const AdjHist& h, double r, double g, const double2* e2) {
        const int b0 = __double2int_rd((r - h.r_min) * h.inv_dr);
        lo = max(0, b0 - h.reach);
        hi = min(h.n_bins - 1, b0 + h.reach);
        z = (r - (h.r_min + (lo + 0.5) * h.dr)) * h.inv_sig;
        G = g * h.norm * exp_table(-0.5 * z * z, e2);
        q = exp_table(h.dz * z - 0.5 * h.dz * h.dz, e2);
    }
    __device__ __forceinline__ void next(const AdjHist& h) {
        G *= q;
        q *= h.qq;
        z -= h.dz;
    }
};

// The smoothed counts of x_t.  Each warp has bins of its own in shared memory, to which its
// lanes add in a fixed order: a lane waits a few steps where needed, so that no two lanes
// are at the same bin in any step.  So the sums are FP64's, to the far tails of the kernel,
// and the same from run to run.  A block takes every gridDim-th group of its particles and
// adds its warps' bins, in order, to its own row of part.  Bound by the FP64 unit and the
// latency of a step's load, addition and store.  20 steps, each sampled, with 64-bit
// integer sums (whose unit the tails fall below) and so: 4096 particles 1716 -> 1775 us,
// 32768 8057 -> 8273; with one copy of a warp's bins 1848 and 8680; 400 bins 7687 -> 7441,
// 2900 8332 -> 9016.
constexpr int kAdjHistBins = 3072;          // the most bins in shared memory
constexpr int kAdjHistBlocks = 152 * 16;    // the most rows
// Warps of a block, fewer where their bins are many; and copies of a warp's bins, more
// where they are few, for its lanes would wait for one another.
int hist_warps(int bins) { return bins <= 384 ? 8 : 2; }
int hist_copies(int bins) {
    int c = 8;
    while (c > 1 && c * bins > 512) c /= 2;
    return c;
}
int hist_blocks(int n, int lanes, int bins) {
    const int per = hist_warps(bins) * (32 / lanes);
    return std::min(kAdjHistBlocks, (n + per - 1) / per);
}
constexpr int kAdjHistSmem = 60 << 10;      // the most that hist_smem says
size_t hist_smem(int lanes, int bins) {
    return hist_warps(bins) *
           (8 * (size_t)bins * hist_copies(bins) + 4 * (size_t)(32 / lanes) * kAdjStride);
}
template <int G>
__global__ void __launch_bounds__(256)
adj_hist_kernel(AdjWalk w, double rc2, AdjHist h, int copies, double* part) {
    extern __shared__ double bins[];
    if (*w.bad <= w.t) return;
    const int warps = blockDim.x >> 5, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int held = copies * h.n_bins, first = lane * copies / 32 * h.n_bins;
    double* mine = bins + wid * held;
    uint32_t* q = reinterpret_cast<uint32_t*>(bins + warps * held) +
                  (wid * (32 / G) + lane / G) * kAdjStride;
    for (int b = lane; b < held; b += 32) mine[b] = 0.0;
    mine += first;
    __syncwarp();
    const int per = warps * (32 / G);
    for (int g0 = blockIdx.x * per; g0 < w.n; g0 += gridDim.x * per) {
        const int i = g0 + wid * (32 / G) + lane / G;
        const bool active = i < w.n;
        double4_32a xi = make_double4_32a(0.0, 0.0, 0.0, 0.0);
        if (active) xi = w.x[i];
        for_pairs<G, true>(w, rc2, i, active, lane, xi, q, [&](bool ok, double r2) {
            GaussBins a(h, ok ? sqrt64(r2, rsqrt64(r2)) : h.r_min, h.dr, w.q.e2);
            const int len = ok ? max(0, a.hi - a.lo + 1) : 0;
            // lane by lane, a wait before the first bin that keeps it from every other lane's:
            // at step t the lane is at bin lo + t - wait
            int wait = 0;
            for (bool again = true; __any_sync(0xffffffffu, again); wait += again ? 1 : 0) {
                const uint32_t same = __match_any_sync(
                    0xffffffffu, len > 0 ? first + a.lo - wait : held + lane);
                again = len > 0 && (same & ((1u << lane) - 1u)) != 0;
            }
            const int steps = __reduce_max_sync(0xffffffffu, len > 0 ? len + wait : 0);
            for (int t = 0; t < steps; ++t) {
                const int k = t - wait;
                if (k >= 0 && k < len) {
                    mine[a.lo + k] += a.G;
                    a.next(h);
                }
                __syncwarp();
            }
        });
    }
    __syncthreads();
    for (int b = threadIdx.x; b < h.n_bins; b += blockDim.x) {
        double t = 0.0;
        for (int k = 0; k < warps * copies; ++k) t += bins[k * h.n_bins + b];
        part[(size_t)blockIdx.x * h.n_bins + b] += t;
    }
}

// The same with more bins than shared memory holds: added to global doubles, in any order.
template <int G>
__global__ void __launch_bounds__(kAdjWarps * 32)
adj_hist_global_kernel(AdjWalk w, double rc2, AdjHist h, double* sum) {
    __shared__ uint32_t sq[kAdjWarps][32 / G][kAdjStride];
    if (*w.bad <= w.t) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int i = (blockIdx.x * kAdjWarps + wid) * (32 / G) + lane / G;
    const bool active = i < w.n;
    double4_32a xi = make_double4_32a(0.0, 0.0, 0.0, 0.0);
    if (active) xi = w.x[i];
    for_pairs<G>(w, rc2, i, active, lane, xi, sq[wid][lane / G],
                 [&](int, const double*, double r2) {
                     GaussBins a(h, sqrt64(r2, rsqrt64(r2)), h.dr, w.q.e2);
                     for (int b = a.lo; b <= a.hi; ++b, a.next(h)) atomicAdd(&sum[b], a.G);
                 });
}

// out[b] = the sum of column b of part[rows][cols], rows in order
__global__ void __launch_bounds__(256) adj_columns_kernel(const double* part, int rows, int cols,
                                                          double* out) {
    __shared__ double red[256];
    double t = 0.0;
    for (int r = threadIdx.x; r < rows; r += blockDim.x) t += part[(size_t)r * cols + blockIdx.x];
    red[threadIdx.x] = t;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}

// out[k][b] = block b's share of the sum of row k of part[kAdjTh][m], in an order of
// its own
__global__ void __launch_bounds__(256) adj_rows_kernel(const double* part, int m, double* out) {
    __shared__ double red[256];
    double t = 0.0;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < m; r += gridDim.x * blockDim.x)
        t += part[(size_t)blockIdx.y * m + r];
    red[threadIdx.x] = t;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = red[0];
}

struct AdjReverse {
    const double4_32a* u;  // u_t
    const double* lam1;    // lam_{t+1}, 3n
    const double* lam2;    // lam_{t+2}
    double* lam0;          // lam_t (out)
    double4_32a* u_prev;   // u_{t-1} (out)
    double c_self1, c_self2;   // lam_t = g + c_self1 lam1 + c_self2 lam2 + J u
    double cu0, cu1;           // u_{t-1} = cu0 lam_t + cu1 lam1
    const double* wgt;     // per bin: dL/d(smoothed count) of this step, or null
    AdjHist h;
    double* part;          // parameter sums per thread, [kAdjTh][threads]
};

// lam_t and u_{t-1}, and each thread's share of u_t . dF/dth added to its own
// running sums.
template <int G>
__global__ void __launch_bounds__(kAdjWarps * 32) adj_reverse_kernel(AdjWalk w, double rc2,
                                                                     AdjReverse a) {
    __shared__ uint32_t sq[kAdjWarps][32 / G][kAdjStride];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int i = (blockIdx.x * kAdjWarps + wid) * (32 / G) + lane / G, m = lane % G;
    const bool active = i < w.n;
    double4_32a xi = make_double4_32a(0.0, 0.0, 0.0, 0.0), ui = xi;
    if (active) {
        xi = w.x[i];
        ui = a.u[i];
    }
    double th[kAdjTh] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double ju[3] = {0.0, 0.0, 0.0}, gl[3] = {0.0, 0.0, 0.0};
    for_pairs<G>(w, rc2, i, active, lane, xi, sq[wid][lane / G],
                 [&](int j, const double* d, double r2) {
        const double4_32a uj = a.u[j];
        const double du[3] = {uj.x - ui.x, uj.y - ui.y, uj.z - ui.z};
        const double ddu = __fma_rn(d[2], du[2], __fma_rn(d[1], du[1], __dmul_rn(d[0], du[0])));
        const double dui = __fma_rn(d[2], ui.z, __fma_rn(d[1], ui.y, __dmul_rn(d[0], ui.x)));
        double s, ds;
        const double ri = pair_all(w.q, r2, dui, s, ds, th);
        const double c = __dmul_rn(__dmul_rn(ds, ri), ddu);
#pragma unroll
        for (int k = 0; k < 3; ++k) ju[k] = __fma_rn(s, du[k], __fma_rn(c, d[k], ju[k]));
        if (a.wgt) {
            // d/dx_i of the smoothed counts of pairs (i, j) and (j, i)
            double wr = 0.0;
            GaussBins g(a.h, sqrt64(r2, ri), 1.0, w.q.e2);
            for (int b = g.lo; b <= g.hi; ++b, g.next(a.h)) wr = __fma_rn(a.wgt[b] * g.G, g.z, wr);
            wr *= 2.0 * a.h.dr * a.h.inv_sig * ri;
#pragma unroll
            for (int k = 0; k < 3; ++k) gl[k] = __fma_rn(wr, d[k], gl[k]);
        }
    });
    const size_t threads = (size_t)gridDim.x * blockDim.x;
    double* part = a.part + blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
    for (int k = 0; k < kAdjTh; ++k) {
        const bool on = k < 2 ? w.q.ao_rc2 > 0.0 : (k < 4 ? w.q.y_rc2 > 0.0 : w.q.lj_rc2 > 0.0);
        if (on) part[k * threads] += th[k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        ju[k] = lanes_sum<G>(ju[k]);
        if (a.wgt) gl[k] = lanes_sum<G>(gl[k]);
    }
    if (!active || m >= 3) return;
    const size_t o = 3 * (size_t)i + m;
    const double l0 = pick(m, gl[0], gl[1], gl[2]) + a.c_self1 * a.lam1[o] + a.c_self2 * a.lam2[o] +
                      pick(m, ju[0], ju[1], ju[2]);
    a.lam0[o] = l0;
    reinterpret_cast<double*>(a.u_prev)[4 * (size_t)i + m] = a.cu0 * l0 + a.cu1 * a.lam1[o];
}

// 3n host-layout values in original order into slots (as double4, or 3n)
__global__ void __launch_bounds__(256) adj_gather_kernel(int n, const double* aos, const int* order,
                                                         double4_32a* x4, double* x3) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* v = aos + 3 * (size_t)(order ? order[i] : i);
    if (x4) x4[i] = make_double4_32a(v[0], v[1], v[2], 0.0);
    if (x3)
        for (int k = 0; k < 3; ++k) x3[3 * (size_t)i + k] = v[k];
}
// and back: x4 with its box images, or x3
__global__ void __launch_bounds__(256) adj_ungather_kernel(int n, const double4_32a* x4,
                                                           const double* x3, const int* img,
                                                           double L, const int* order,
                                                           double* aos) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* v = aos + 3 * (size_t)order[i];
    if (x4) {
        const double4_32a p = x4[i];
        v[0] = p.x + L * img[3 * i];
        v[1] = p.y + L * img[3 * i + 1];
        v[2] = p.z + L * img[3 * i + 2];
    } else {
        for (int k = 0; k < 3; ++k) v[k] = x3[3 * (size_t)i + k];
    }
}

__global__ void __launch_bounds__(256) philox_noise_kernel(uint32_t seed, int n, long long first,
                                                           int n_steps, double* out) {
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= (long long)n * n_steps) return;
    const int t = (int)(idx / n), i = (int)(idx % n);
    double xi[6];
    philox_gaussians6(seed, (uint32_t)i, (uint32_t)(first + t), xi);
    for (int k = 0; k < 6; ++k) out[6 * idx + k] = xi[k];
}

}  // namespace
}  // namespace psim

using namespace psim;

extern "C" void psim_internal_set_error(const char* msg);

namespace {

int adj_fail(int code, const char* msg) {
    psim_internal_set_error(msg);
    return code;
}

#define ADJ_CUDA(call)                                                             \
    do {                                                                           \
        cudaError_t e_ = (call);                                                   \
        if (e_ != cudaSuccess) return adj_fail(PSIM_ERR_CUDA, cudaGetErrorString(e_)); \
    } while (0)

struct Buf {
    void* p = nullptr;
    size_t bytes = 0;
    void free() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    cudaError_t ensure(size_t b) {
        if (b <= bytes) return cudaSuccess;
        free();
        cudaError_t e = cudaMalloc(&p, b ? b : 16);
        if (e == cudaSuccess) bytes = b;
        return e;
    }
    template <class T> T* as() const { return static_cast<T*>(p); }
    ~Buf() { if (p) cudaFree(p); }
};

// AO coefficients c1, c2 (AOPotential.cpp:50-55) and their derivatives with
// respect to wellDepth and cutOff
void ao_coeffs_d(double kT, double wd, double rc, double c[2], double dwd[2], double drc[2]) {
    const double q = rc / (rc - 1.0);
    const double a1 = -kT * wd * q * q * q, a2 = -3.0 / (2.0 * rc), a3 = 1.0 / (2.0 * rc * rc * rc);
    c[0] = -a1 * a2;
    c[1] = -3.0 * a1 * a3;
    const double a1_wd = -kT * q * q * q;
    const double a1_rc = 3.0 * kT * wd * rc * rc / std::pow(rc - 1.0, 4);
    const double a2_rc = 3.0 / (2.0 * rc * rc), a3_rc = -3.0 / (2.0 * rc * rc * rc * rc);
    dwd[0] = -a1_wd * a2;
    dwd[1] = -3.0 * a1_wd * a3;
    drc[0] = -(a1_rc * a2 + a1 * a2_rc);
    drc[1] = -3.0 * (a1_rc * a3 + a1 * a3_rc);
}

}  // namespace

struct psim_adjoint {
    psim_adjoint_config cfg{};
    int device = 0, n = 0, T = 0, K = 0, S = 0;
    cudaStream_t st = nullptr;
    AdjStep step{};
    AdjHist hist{};
    double rc2 = 0.0, walk_rc2 = 0.0;
    int lanes = 4;            // lanes per particle of the sweeps
    // the neighbour list: its grid, radius, the build's displacement bound and
    // the most entries of a particle; listed: it holds for the step the host is at
    AdjGrid grid{};
    float list_r2 = 0.f, disp2 = 0.f;
    int most = 0, stride = 0;
    bool listed = false;
    int* host = nullptr;      // pinned: {bad, most}
    Buf key, rank, count, start, scan, tmp, order, sorted, lcount, entry, bad, xbuild,
        img, F, v0, traj, trajf, ck, lam[3], u[2], part, acc, hpart, hsum, wgt, x0, e2;
};

namespace {

// steps enqueued before the host looks whether the list still holds; the forces of
// that many steps and two more are kept, so that a step can be taken again
constexpr int kAdjBlock = 16;
constexpr int kAdjRowBlocks = 64;   // blocks that sum a row of the parameter shares

// Lanes per particle: few particles need many, for warps to fill the chip and short
// chains; many particles few, which leave fewer lanes without a pair.  Gradient of 40
// steps with 16 / 8 / 4 lanes, ms: 1000 particles 2.74 / 3.60 / -, 4096 5.18 / 5.30 /
// 6.2, 16384 13.2 / 11.7 / 11.0, 131072 87.6 / 71.8 / 66.6.
int lanes_for(int n) { return n <= 4096 ? 16 : (n < 12288 ? 8 : 4); }
template <class Fn>
void with_lanes(const psim_adjoint* a, Fn&& fn) {
    if (a->lanes == 16) fn(std::integral_constant<int, 16>{});
    else if (a->lanes == 8) fn(std::integral_constant<int, 8>{});
    else fn(std::integral_constant<int, 4>{});
}
constexpr int kAdjRing = kAdjBlock + 2;
constexpr size_t kAdjTraj = (size_t)256 << 20;   // bytes of positions always worth keeping

double4_32a* pos_at(psim_adjoint* a, int k) {
    return a->traj.as<double4_32a>() + (size_t)k * a->n;
}
float4* posf_at(psim_adjoint* a, int k) { return a->trajf.as<float4>() + (size_t)k * a->n; }
double* force_at(psim_adjoint* a, int t) {
    return a->F.as<double>() + (size_t)((t + kAdjRing) % kAdjRing) * 3 * a->n;
}
int blocks_of(psim_adjoint* a, int warps) {
    const int per = warps * (32 / a->lanes);
    return (a->n + per - 1) / per;
}

// The list's radius and grid for this call's cutoffs: the largest distance of any
// pass and a skin of 0.3 (or less where the box is small: the list radius stays
// below L/2, as cellSize >= the distance and three cells a side leave room for).
int set_list(psim_adjoint* a) {
    const double reach = std::sqrt(std::max(a->rc2, a->walk_rc2));
    const double skin = std::min(0.3, 0.4 * reach), R = reach + skin;
    const double L = a->cfg.geom.box_size;
    const double ulpL = std::ldexp(1.0, std::ilogb(std::max(L, 1.0)) - 23);
    const double Rw = R * (1.0 + 1e-6) + 8.0 * ulpL;
    a->list_r2 = (float)(Rw * Rw * (1.0 + 1e-6));
    const double d = 0.5 * skin * (1.0 - 1e-3) - 4.0 * ulpL;
    a->disp2 = d > 0.0 ? (float)(d * d) : 0.f;
    const int s = std::max(1, std::min(256, (int)(L / (Rw * (1.0 + 1e-6)))));
    a->grid = AdjGrid{L, s / L, s, s * s, s * s * s};
    const size_t nc = (size_t)a->grid.ncell;
    ADJ_CUDA(a->count.ensure(4 * nc));
    ADJ_CUDA(a->start.ensure(4 * nc));
    ADJ_CUDA(a->scan.ensure(4 * (size_t)scan_scratch_ints((int)nc)));
    a->listed = false;
    return PSIM_OK;
}

// the cell order of the positions in slot k (and of slot k - 1, carried along),
// moved into the box; images counted in img
int sort_slot(psim_adjoint* a, int k, bool count_images, int* order, float4* sorted) {
    const int n = a->n, b = (n + 255) / 256;
    ADJ_CUDA(cudaMemsetAsync(a->count.p, 0, 4 * (size_t)a->grid.ncell, a->st));
    adj_rebase_kernel<<<b, 256, 0, a->st>>>(n, pos_at(a, k), pos_at(a, k - 1), posf_at(a, k),
                                            a->xbuild.as<float4>(), a->grid,
                                            count_images ? a->img.as<int>() : nullptr,
                                            a->key.as<int>(), a->rank.as<int>(),
                                            a->count.as<int>());
    ADJ_CUDA(launch_scan(a->count.as<int>(), a->start.as<int>(), a->grid.ncell, a->scan.as<int>(),
                         a->st));
    adj_scatter_kernel<<<b, 256, 0, a->st>>>(n, a->key.as<int>(), a->rank.as<int>(),
                                             a->start.as<int>(), a->tmp.as<int>());
    adj_sort_kernel<<<b, 256, 0, a->st>>>(n, a->tmp.as<int>(), a->key.as<int>(),
                                          a->start.as<int>(), a->count.as<int>(), posf_at(a, k),
                                          sorted, order);
    ADJ_CUDA(cudaGetLastError());
    return PSIM_OK;
}

// The neighbour list of the positions in slot k: counted, then filled.
int build_list(psim_adjoint* a, int k, bool count_images) {
    const int n = a->n, b = (int)(((long long)n * kAdjBuildLanes + 255) / 256);
    float4* sorted = a->sorted.as<float4>();
    int rc = sort_slot(a, k, count_images, nullptr, sorted);
    if (rc) return rc;
    ADJ_CUDA(cudaMemsetAsync(a->bad.p, 0x7f, 4, a->st));       // no step yet
    ADJ_CUDA(cudaMemsetAsync(a->bad.as<int>() + 1, 0, 4, a->st));
    adj_list_kernel<false><<<b, 256, 0, a->st>>>(n, a->grid, sorted, a->key.as<int>(),
                                                 a->start.as<int>(), a->count.as<int>(), a->list_r2,
                                                 a->lcount.as<int>(), nullptr, 0,
                                                 a->bad.as<int>() + 1);
    ADJ_CUDA(cudaMemcpyAsync(a->host + 1, a->bad.as<int>() + 1, 4, cudaMemcpyDeviceToHost, a->st));
    ADJ_CUDA(cudaStreamSynchronize(a->st));
    a->most = a->host[1];
    a->stride = (a->most + 7) & ~7;
    // room for eight entries more, so that most later lists need no allocation
    const size_t need = 4 * (size_t)n * a->stride;
    if (need > a->entry.bytes) ADJ_CUDA(a->entry.ensure(need + 32 * (size_t)n));
    adj_list_kernel<true><<<b, 256, 0, a->st>>>(n, a->grid, sorted, a->key.as<int>(),
                                                a->start.as<int>(), a->count.as<int>(), a->list_r2,
                                                nullptr, a->entry.as<int>(), a->stride, nullptr);
    ADJ_CUDA(cudaGetLastError());
    a->listed = true;
    return PSIM_OK;
}

AdjWalk walk_at(psim_adjoint* a, const AdjPair& q, int slot, int t) {
    return AdjWalk{q, AdjList{a->lcount.as<int>(), a->entry.as<int>(), a->stride}, a->n,
                   pos_at(a, slot), posf_at(a, slot), a->cfg.geom.box_size,
                   0.5 * a->cfg.geom.box_size, t, a->bad.as<int>()};
}

int add_hist(psim_adjoint* a, const AdjWalk& w) {
    const int nb = a->cfg.n_bins;
    cudaError_t e = cudaSuccess;
    with_lanes(a, [&](auto g) {
        constexpr int G = decltype(g)::value;
        if (nb > kAdjHistBins) {
            adj_hist_global_kernel<G><<<blocks_of(a, kAdjWarps), kAdjWarps * 32, 0, a->st>>>(
                w, a->walk_rc2, a->hist, a->hsum.as<double>());
            return;
        }
        const size_t smem = hist_smem(G, nb);
        e = cudaFuncSetAttribute(adj_hist_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kAdjHistSmem);
        if (e == cudaSuccess)
            adj_hist_kernel<G><<<hist_blocks(a->n, G, nb), hist_warps(nb) * 32, smem, a->st>>>(
                w, a->walk_rc2, a->hist, hist_copies(nb), a->hpart.as<double>());
    });
    ADJ_CUDA(e);
    ADJ_CUDA(cudaGetLastError());
    return PSIM_OK;
}

// Steps t0 .. t1 (x_t0 in slot 1, x_{t0-1} in slot 0, F(x_{t0-1}) in its place of
// the force ring), storing x_t in slot 1 + t - t0, with the smoothed counts of
// the sampled steps (of x_t1 when hist_t1).  The steps run a block at a time on
// one list; where a particle left it (x_bad), the list is built anew at
// x_bad, whose own step was still good, and the steps from there are taken again.
// builds (may be null) gets the steps a list was built at, or is to be.
int run_forward(psim_adjoint* a, const AdjPair& q, int t0, int t1, bool do_hist, bool hist_t1,
                bool count_images, std::vector<int>* builds) {
    const int blocks = blocks_of(a, kAdjWarps), threads = kAdjWarps * 32;
    auto sampled = [&](int t) { return do_hist && t > 0 && t % a->cfg.sample_every == 0; };
    int rc;
    for (int t = t0;;) {
        if (!a->listed) {
            if ((rc = build_list(a, 1 + t - t0, count_images))) return rc;
            if (builds) builds->push_back(t);
        }
        const int te = std::min(t1, t + kAdjBlock);
        for (int k = t; k < te; ++k) {
            const int slot = 1 + k - t0;
            const AdjWalk w = walk_at(a, q, slot, k);
            if (sampled(k) && (rc = add_hist(a, w))) return rc;
            AdjForward f{a->step, pos_at(a, slot - 1), force_at(a, k - 1), force_at(a, k),
                         a->v0.as<double>(), pos_at(a, slot + 1), posf_at(a, slot + 1),
                         a->xbuild.as<float4>(), a->disp2, a->order.as<int>(), a->bad.as<int>()};
            with_lanes(a, [&](auto g) {
                adj_forward_kernel<decltype(g)::value><<<blocks, threads, 0, a->st>>>(w, a->rc2,
                                                                                      f);
            });
        }
        if (te == t1 && hist_t1 && sampled(t1) &&
            (rc = add_hist(a, walk_at(a, q, 1 + t1 - t0, t1))))
            return rc;
        ADJ_CUDA(cudaGetLastError());
        ADJ_CUDA(cudaMemcpyAsync(a->host, a->bad.p, 4, cudaMemcpyDeviceToHost, a->st));
        ADJ_CUDA(cudaStreamSynchronize(a->st));
        if (a->host[0] <= te) {
            t = a->host[0];
            a->listed = false;
            if (t < t1) continue;
            if (builds) builds->push_back(t1);
            if (hist_t1 && sampled(t1)) {
                if ((rc = build_list(a, 1 + t1 - t0, count_images))) return rc;
                if ((rc = add_hist(a, walk_at(a, q, 1 + t1 - t0, t1)))) return rc;
            }
            return PSIM_OK;
        }
        t = te;
        if (t == t1) return PSIM_OK;
    }
}

}  // namespace

namespace {

void set_pair(const psim_adjoint_params* p, AdjPair& q, double dwd[2], double drc[2]) {
    double c[2] = {0.0, 0.0};
    dwd[0] = dwd[1] = drc[0] = drc[1] = 0.0;
    q = AdjPair{};
    if (p->ao_cutoff > 0.0) {
        // the coefficients' range (1 + q) and the cutoff distance: the same
        // unless ao_range is given, which holds the cutoff while q moves
        const double range = p->ao_range > 0.0 ? p->ao_range : p->ao_cutoff;
        ao_coeffs_d(p->kT, p->ao_well_depth, range, c, dwd, drc);
        q.c1 = c[0];
        q.c2 = c[1];
        q.ao_rc2 = p->ao_cutoff * p->ao_cutoff;
    }
    if (p->yuk_cutoff > 0.0) {
        q.Y = p->yuk_amplitude;
        q.lam = p->yuk_length;
        q.inv_lam = 1.0 / p->yuk_length;
        q.y_rc2 = p->yuk_cutoff * p->yuk_cutoff;
    }
    if (p->lj_cutoff > 0.0) {
        q.eps = p->lj_epsilon;
        q.sig = p->lj_sigma;
        q.ljn = p->lj_n;
        q.lj_rc2 = p->lj_cutoff * p->lj_cutoff;
        q.eps4n = 4.0 * q.ljn * q.eps;
        q.eps_n_sig = q.ljn * q.eps / q.sig;
    }
}

// host values (3n AoS, original order) to the device
int upload(psim_adjoint* a, const double* host) {
    ADJ_CUDA(cudaMemcpyAsync(a->x0.p, host, 24 * (size_t)a->n, cudaMemcpyHostToDevice, a->st));
    return PSIM_OK;
}

// The whole forward in K-step segments (slots 0, 1, ... hold x_{t0-1}, x_t0 ..
// x_t0+K), with a checkpoint (x_t0, x_{t0-1}, F(x_{t0-1})) of each and the smoothed
// counts of the sampled steps.
// builds (may be null) gets the steps of the last segment that a list was built at.
int forward_all(psim_adjoint* a, const AdjPair& q, const double* pos0, const double* vel0,
                std::vector<int>* builds) {
    const int n = a->n, b = (n + 255) / 256, nb = a->cfg.n_bins;
    const size_t b4 = 32 * (size_t)n;
    int rc = set_list(a);
    if (rc) return rc;
    // the slots' order: the cell order of the initial positions
    if ((rc = upload(a, pos0))) return rc;
    adj_gather_kernel<<<b, 256, 0, a->st>>>(n, a->x0.as<double>(), nullptr, pos_at(a, 1), nullptr);
    ADJ_CUDA(cudaMemcpyAsync(pos_at(a, 0), pos_at(a, 1), b4, cudaMemcpyDeviceToDevice, a->st));
    if ((rc = sort_slot(a, 1, false, a->order.as<int>(), nullptr))) return rc;
    adj_gather_kernel<<<b, 256, 0, a->st>>>(n, a->x0.as<double>(), a->order.as<int>(), pos_at(a, 1),
                                            nullptr);
    ADJ_CUDA(cudaMemcpyAsync(pos_at(a, 0), pos_at(a, 1), b4, cudaMemcpyDeviceToDevice, a->st));
    ADJ_CUDA(cudaMemsetAsync(a->img.p, 0, 12 * (size_t)n, a->st));
    if (vel0) {
        if ((rc = upload(a, vel0))) return rc;
        adj_gather_kernel<<<b, 256, 0, a->st>>>(n, a->x0.as<double>(), a->order.as<int>(), nullptr,
                                                a->v0.as<double>());
    } else {
        ADJ_CUDA(cudaMemsetAsync(a->v0.p, 0, 24 * (size_t)n, a->st));
    }
    ADJ_CUDA(cudaMemsetAsync(force_at(a, -1), 0, 24 * (size_t)n, a->st));
    ADJ_CUDA(cudaMemsetAsync(a->hsum.p, 0, 8 * (size_t)nb, a->st));
    const bool shared = nb <= kAdjHistBins;
    const int rows = hist_blocks(n, a->lanes, nb);
    if (shared) ADJ_CUDA(cudaMemsetAsync(a->hpart.p, 0, 8 * (size_t)nb * rows, a->st));
    for (int t0 = 0; t0 < a->T; t0 += a->K) {
        const int t1 = std::min(t0 + a->K, a->T);
        char* c = a->ck.as<char>() + (size_t)(t0 / a->K) * 88 * n;
        ADJ_CUDA(cudaMemcpyAsync(c, pos_at(a, 0), 2 * b4, cudaMemcpyDeviceToDevice, a->st));
        ADJ_CUDA(cudaMemcpyAsync(c + 2 * b4, force_at(a, t0 - 1), 24 * (size_t)n,
                                 cudaMemcpyDeviceToDevice, a->st));
        // the last segment's lists are all built within it: the reverse pass builds
        // them again
        const bool last = t1 == a->T;
        if (last && builds) a->listed = false;
        // the counts of x_t1 belong to the next segment unless it is the last
        if ((rc = run_forward(a, q, t0, t1, true, last, true, last ? builds : nullptr))) return rc;
        if (t1 < a->T) {   // carry x_{t1-1}, x_t1 to the front
            const int k = t1 - t0;
            for (int s = 0; s < 2; ++s) {
                ADJ_CUDA(cudaMemcpyAsync(pos_at(a, s), pos_at(a, k + s), b4,
                                         cudaMemcpyDeviceToDevice, a->st));
                ADJ_CUDA(cudaMemcpyAsync(posf_at(a, s), posf_at(a, k + s), 16 * (size_t)n,
                                         cudaMemcpyDeviceToDevice, a->st));
            }
        }
    }
    if (shared) adj_columns_kernel<<<nb, 256, 0, a->st>>>(a->hpart.as<double>(), rows, nb,
                                                          a->hsum.as<double>());
    ADJ_CUDA(cudaGetLastError());
    return PSIM_OK;
}

int mean_g(psim_adjoint* a, std::vector<double>& g) {
    const int nb = a->cfg.n_bins;
    std::vector<double> h((size_t)nb);
    ADJ_CUDA(cudaMemcpyAsync(h.data(), a->hsum.p, 8 * (size_t)nb, cudaMemcpyDeviceToHost, a->st));
    ADJ_CUDA(cudaStreamSynchronize(a->st));
    const double L = a->cfg.geom.box_size;
    const double rho = a->n / (L * L * L);
    g.assign((size_t)nb, 0.0);
    for (int b = 0; b < nb; ++b) {
        const double rb = a->hist.r_min + (b + 0.5) * a->hist.dr;
        const double Cb = a->n * rho * 4.0 * M_PI * rb * rb * a->hist.dr;
        g[(size_t)b] = h[(size_t)b] / (a->S * Cb);
    }
    return PSIM_OK;
}

}  // namespace

extern "C" {

psim_adjoint* psim_adjoint_create(const psim_adjoint_config* cfg, int32_t device) {
    if (!cfg) { adj_fail(PSIM_ERR_INPUT, "NULL config"); return nullptr; }
    const psim_geometry& gm = cfg->geom;
    const int n = gm.n_particles;
    if (n <= 0 || gm.cell_scale < 3 || !(gm.box_size > 0.0) ||
        std::fabs(gm.cell_size * gm.cell_scale - gm.box_size) > 1e-9 * gm.box_size) {
        adj_fail(PSIM_ERR_INPUT, "adjoint: bad geometry (n > 0, cellScale >= 3, cellSize * cellScale == box)");
        return nullptr;
    }
    if (cfg->n_steps <= 0 || cfg->checkpoint_every <= 0 || cfg->sample_every <= 0 ||
        cfg->sample_every > cfg->n_steps || cfg->n_bins <= 0 || !(cfg->r_max > cfg->r_min) ||
        !(cfg->sigma > 0.0) || !(cfg->mass > 0.0)) {
        adj_fail(PSIM_ERR_INPUT, "adjoint: bad steps, checkpoint/sample interval, bins, sigma or mass");
        return nullptr;
    }
    const double reach = cfg->r_max + 4.0 * cfg->sigma;
    if (reach > gm.cell_size) {
        adj_fail(PSIM_ERR_INPUT, "adjoint: cellSize must cover r_max + 4 sigma");
        return nullptr;
    }
    psim_vgb_coeffs vc;
    if (psim_vgb_coefficients(cfg->integ.gamma, cfg->integ.dt, cfg->integ.kT, &vc)) return nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        adj_fail(PSIM_ERR_NO_DEVICE, "adjoint: no such CUDA device");
        return nullptr;
    }
    cudaSetDevice(device);
    psim_adjoint* a = new psim_adjoint();
    a->cfg = *cfg;
    a->device = device;
    a->n = n;
    a->T = cfg->n_steps;
    const int asked = std::min(std::max(cfg->checkpoint_every, 2), cfg->n_steps);
    a->K = std::max(asked, (int)std::min((size_t)a->T, kAdjTraj / (48 * (size_t)n)));
    a->S = cfg->n_steps / cfg->sample_every;
    const double dt = cfg->integ.dt, dt2 = dt * dt, m = 1.0 / cfg->mass;
    a->step = AdjStep{n, 1.0 + vc.coeff0, vc.coeff0, m * dt2 * (vc.coeff1 + vc.coeff2),
                      m * dt2 * vc.coeff2, vc.coeff1 * dt, vc.coeff3 * dt2 * m, vc.sig1, vc.sig2,
                      vc.corr, vc.dev, vc.coeff0, (uint32_t)cfg->integ.seed};
    const double dr = (cfg->r_max - cfg->r_min) / cfg->n_bins;
    const double dz = dr / cfg->sigma;
    a->hist = AdjHist{cfg->r_min, dr, 1.0 / cfg->sigma, 1.0 / (std::sqrt(2.0 * M_PI) * cfg->sigma),
                      dz, std::exp(-dz * dz), 1.0 / dr, cfg->n_bins,
                      (int)std::ceil(4.0 * cfg->sigma / dr) + 1};
    a->walk_rc2 = reach * reach;
    a->lanes = lanes_for(n);
    const size_t b3 = 24 * (size_t)n, b4 = 32 * (size_t)n, b1 = 4 * (size_t)n;
    const size_t threads = (size_t)blocks_of(a, kAdjWarps) * kAdjWarps * 32;
    bool ok = cudaStreamCreateWithFlags(&a->st, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMallocHost(&a->host, 16) == cudaSuccess && !a->key.ensure(b1) &&
              !a->rank.ensure(b1) && !a->tmp.ensure(b1) && !a->order.ensure(b1) &&
              !a->sorted.ensure(16 * (size_t)n) && !a->lcount.ensure(b1) &&
              !a->bad.ensure(8) && !a->xbuild.ensure(16 * (size_t)n) && !a->img.ensure(3 * b1) &&
              !a->F.ensure(b3 * kAdjRing) && !a->v0.ensure(b3) &&
              !a->lam[0].ensure(b3) && !a->lam[1].ensure(b3) && !a->lam[2].ensure(b3) &&
              !a->u[0].ensure(b4) && !a->u[1].ensure(b4) && !a->x0.ensure(b3) &&
              !a->part.ensure(8 * kAdjTh * threads) && !a->acc.ensure(8 * kAdjTh * (1 + kAdjRowBlocks)) &&
              !a->e2.ensure(16 * kExpTable) &&
              (cfg->n_bins > kAdjHistBins ||
               !a->hpart.ensure(8 * (size_t)cfg->n_bins * hist_blocks(n, a->lanes, cfg->n_bins))) &&
              !a->hsum.ensure(8 * (size_t)cfg->n_bins) && !a->wgt.ensure(8 * (size_t)cfg->n_bins);
    // the segments' positions and the checkpoints: shorter segments where the memory
    // does not hold K steps
    while (ok) {
        const int nck = (a->T + a->K - 1) / a->K + 1;
        if (!a->traj.ensure(b4 * (size_t)(a->K + 2)) &&
            !a->trajf.ensure(16 * (size_t)n * (size_t)(a->K + 2)) &&
            !a->ck.ensure((2 * b4 + b3) * (size_t)nck))
            break;
        cudaGetLastError();
        a->traj.free();
        a->trajf.free();
        a->ck.free();
        ok = a->K > 2;
        a->K = a->K > asked ? asked : std::max(2, a->K / 2);
    }
    if (ok) {
        double2 e2[kExpTable];
        exp_table_values(e2);
        ok = cudaMemcpy(a->e2.p, e2, sizeof e2, cudaMemcpyHostToDevice) == cudaSuccess;
    }
    if (!ok) {
        adj_fail(PSIM_ERR_CUDA, "adjoint: device allocation failed");
        psim_adjoint_destroy(a);
        return nullptr;
    }
    return a;
}

int psim_philox_noise(uint32_t seed, int32_t n, int64_t first_step, int32_t n_steps,
                      double* out, int32_t device) {
    if (!out || n < 0 || n_steps < 0 || first_step < 0)
        return adj_fail(PSIM_ERR_INPUT, "philox noise: bad arguments");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
        return adj_fail(PSIM_ERR_NO_DEVICE, "philox noise: no such CUDA device");
    const long long cnt = (long long)n * n_steps;
    if (cnt == 0) return PSIM_OK;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    cudaError_t e;
    {   // the buffer is freed with `device` current
        Buf b;
        e = b.ensure(48 * (size_t)cnt);
        if (e == cudaSuccess) {
            philox_noise_kernel<<<(unsigned)((cnt + 255) / 256), 256>>>(seed, n, first_step,
                                                                        n_steps, b.as<double>());
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpy(out, b.p, 48 * (size_t)cnt, cudaMemcpyDeviceToHost);
    }
    cudaSetDevice(prev);
    return e == cudaSuccess ? PSIM_OK : adj_fail(PSIM_ERR_CUDA, cudaGetErrorString(e));
}

void psim_adjoint_destroy(psim_adjoint* a) {
    if (!a) return;
    cudaSetDevice(a->device);
    if (a->st) {
        cudaStreamSynchronize(a->st);
        cudaStreamDestroy(a->st);
    }
    if (a->host) cudaFreeHost(a->host);
    delete a;
}

int psim_adjoint_forward(psim_adjoint* a, const psim_adjoint_params* p, const double* pos0,
                         const double* vel0, double* g_mean, double* pos_final) {
    if (!a || !p || !pos0 || !g_mean) return adj_fail(PSIM_ERR_INPUT, "NULL argument");
    cudaSetDevice(a->device);
    AdjPair q;
    double dwd[2], drc[2];
    set_pair(p, q, dwd, drc);
    q.e2 = a->e2.as<double2>();
    a->rc2 = std::max(std::max(q.ao_rc2, q.y_rc2), q.lj_rc2);
    if (a->rc2 > a->cfg.geom.cell_size * a->cfg.geom.cell_size)
        return adj_fail(PSIM_ERR_INPUT, "adjoint: a cutoff exceeds the cell size");
    int rc = forward_all(a, q, pos0, vel0, nullptr);
    if (rc) return rc;
    std::vector<double> g;
    if ((rc = mean_g(a, g))) return rc;
    std::copy(g.begin(), g.end(), g_mean);
    if (pos_final) {
        const int last = a->T - ((a->T - 1) / a->K) * a->K;   // slot of x_T in the last segment
        adj_ungather_kernel<<<(a->n + 255) / 256, 256, 0, a->st>>>(
            a->n, pos_at(a, 1 + last), nullptr, a->img.as<int>(), a->cfg.geom.box_size,
            a->order.as<int>(), a->x0.as<double>());
        ADJ_CUDA(cudaMemcpyAsync(pos_final, a->x0.p, 24 * (size_t)a->n, cudaMemcpyDeviceToHost,
                                 a->st));
        ADJ_CUDA(cudaStreamSynchronize(a->st));
    }
    return PSIM_OK;
}

int psim_adjoint_gradient(psim_adjoint* a, const psim_adjoint_params* p, const double* pos0,
                          const double* vel0, const double* g_target, double* loss,
                          double* g_mean, double* grad, double* grad_pos0) {
    if (!a || !p || !pos0 || !g_target || !loss || !grad)
        return adj_fail(PSIM_ERR_INPUT, "NULL argument");
    cudaSetDevice(a->device);
    const int n = a->n, T = a->T, K = a->K, nb = a->cfg.n_bins;
    const size_t b3 = 24 * (size_t)n;
    AdjPair q;
    double dwd[2], drc[2];
    set_pair(p, q, dwd, drc);
    q.e2 = a->e2.as<double2>();
    a->rc2 = std::max(std::max(q.ao_rc2, q.y_rc2), q.lj_rc2);
    if (a->rc2 > a->cfg.geom.cell_size * a->cfg.geom.cell_size)
        return adj_fail(PSIM_ERR_INPUT, "adjoint: a cutoff exceeds the cell size");
    if (q.lj_rc2 > 0.0 && (!(q.sig > 0.0) || q.ljn < 0 || q.ljn > 64))
        return adj_fail(PSIM_ERR_INPUT, "adjoint: LJ term needs sigma > 0 and 0 <= n <= 64");
    // forward: checkpoints and the loss
    std::vector<int> builds;
    int rc = forward_all(a, q, pos0, vel0, &builds);
    if (rc) return rc;
    std::vector<double> g;
    if ((rc = mean_g(a, g))) return rc;
    double L = 0.0;
    std::vector<double> wgt((size_t)nb);
    const double box = a->cfg.geom.box_size, rho = n / (box * box * box);
    for (int b = 0; b < nb; ++b) {
        const double diff = g[(size_t)b] - g_target[b];
        L += diff * diff;
        const double rb = a->hist.r_min + (b + 0.5) * a->hist.dr;
        const double Cb = n * rho * 4.0 * M_PI * rb * rb * a->hist.dr;
        wgt[(size_t)b] = 2.0 * diff / (a->S * Cb);   // dL / d(smoothed count of one sample)
    }
    *loss = L;
    if (g_mean) std::copy(g.begin(), g.end(), g_mean);
    ADJ_CUDA(cudaMemcpyAsync(a->wgt.p, wgt.data(), 8 * (size_t)nb, cudaMemcpyHostToDevice, a->st));
    // reverse: lam_{T+1} = lam_{T+2} = 0, u_T = 0
    for (int k = 0; k < 3; ++k) ADJ_CUDA(cudaMemsetAsync(a->lam[k].p, 0, b3, a->st));
    const size_t b4 = 32 * (size_t)n;
    ADJ_CUDA(cudaMemsetAsync(a->u[0].p, 0, b4, a->st));
    ADJ_CUDA(cudaMemsetAsync(a->u[1].p, 0, b4, a->st));
    const int blocks = blocks_of(a, kAdjWarps), threads = kAdjWarps * 32;
    ADJ_CUDA(cudaMemsetAsync(a->part.p, 0, 8 * kAdjTh * (size_t)blocks * threads, a->st));
    int l0 = 0, l1 = 1, l2 = 2, uc = 0;   // lam_t, lam_{t+1}, lam_{t+2}; u_t
    const int nseg = (T + K - 1) / K;
    const double rwalk = std::max(a->rc2, a->walk_rc2);
    for (int seg = nseg - 1; seg >= 0; --seg) {
        const int t0 = seg * K, t1 = std::min(t0 + K, T);
        if (seg < nseg - 1) {   // recompute the segment from its checkpoint
            const char* c = a->ck.as<char>() + (size_t)seg * 88 * n;
            ADJ_CUDA(cudaMemcpyAsync(pos_at(a, 0), c, 2 * b4, cudaMemcpyDeviceToDevice, a->st));
            ADJ_CUDA(cudaMemcpyAsync(force_at(a, t0 - 1), c + 2 * b4, b3,
                                     cudaMemcpyDeviceToDevice, a->st));
            a->listed = false;
            builds.clear();
            if ((rc = run_forward(a, q, t0, t1, false, false, false, &builds))) return rc;
        }
        // back through it, each step on the list that holds for it
        int at = a->listed ? (int)builds.size() - 1 : -1;
        for (int t = (seg == nseg - 1 ? t1 : t1 - 1); t >= t0; --t) {
            int want = (int)builds.size() - 1;
            while (builds[(size_t)want] > t) --want;
            if (want != at) {
                if ((rc = build_list(a, 1 + builds[(size_t)want] - t0, false))) return rc;
                at = want;
            }
            const AdjWalk w = walk_at(a, q, 1 + t - t0, t);
            AdjReverse r{};
            r.u = a->u[uc].as<double4_32a>();
            r.lam1 = a->lam[l1].as<double>();
            r.lam2 = a->lam[l2].as<double>();
            r.lam0 = a->lam[l0].as<double>();
            r.u_prev = a->u[1 - uc].as<double4_32a>();
            r.c_self1 = t > 0 ? a->step.c0 : 1.0;
            r.c_self2 = -a->step.a0;
            r.cu0 = t - 1 >= 1 ? a->step.b1 : a->step.cf;
            r.cu1 = -a->step.b2;
            r.wgt = (t > 0 && t % a->cfg.sample_every == 0) ? a->wgt.as<double>() : nullptr;
            r.h = a->hist;
            r.part = a->part.as<double>();
            const double walk = r.wgt ? rwalk : a->rc2;   // the cutoffs alone between samples
            with_lanes(a, [&](auto g) {
                adj_reverse_kernel<decltype(g)::value><<<blocks, threads, 0, a->st>>>(w, walk, r);
            });
            ADJ_CUDA(cudaGetLastError());
            // lam_t becomes lam_{t+1} of the next (earlier) step
            const int old2 = l2;
            l2 = l1;
            l1 = l0;
            l0 = old2;
            uc = 1 - uc;
        }
    }
    double* sums = a->acc.as<double>() + kAdjTh;
    adj_rows_kernel<<<dim3(kAdjRowBlocks, kAdjTh), 256, 0, a->st>>>(a->part.as<double>(),
                                                                    blocks * threads, sums);
    adj_rows_kernel<<<dim3(1, kAdjTh), 256, 0, a->st>>>(sums, kAdjRowBlocks, a->acc.as<double>());
    double th[kAdjTh];
    ADJ_CUDA(cudaMemcpyAsync(th, a->acc.p, 8 * kAdjTh, cudaMemcpyDeviceToHost, a->st));
    if (grad_pos0) {   // lam_0 (now lam[l1]) in original order
        adj_ungather_kernel<<<(n + 255) / 256, 256, 0, a->st>>>(n, nullptr, a->lam[l1].as<double>(),
                                                                nullptr, 0.0, a->order.as<int>(),
                                                                a->x0.as<double>());
        ADJ_CUDA(cudaMemcpyAsync(grad_pos0, a->x0.p, b3, cudaMemcpyDeviceToHost, a->st));
    }
    ADJ_CUDA(cudaStreamSynchronize(a->st));
    // th = dL/d(c1, c2, Y, lambda, eps, sigma) -> dL/d(AO wellDepth, AO range,
    // Y, lambda, eps, sigma)
    grad[0] = th[0] * dwd[0] + th[1] * dwd[1];
    grad[1] = th[0] * drc[0] + th[1] * drc[1];
    grad[2] = th[2];
    grad[3] = th[3];
    grad[4] = th[4];
    grad[5] = th[5];
    return PSIM_OK;
}

}  // extern "C"
