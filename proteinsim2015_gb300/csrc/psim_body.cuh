// psim_body.cuh -- the per-pair bodies the force-pass templates
// (psim_force.cuh, psim_force_cell.cuh, psim_force_list.cuh) are
// instantiated with, one per precision form, each over a plugin's pair
// functor:
//   F64Body<Pair>    the plain FP64 form: the reference's own decisions (images,
//                    cutoff, overlap), pair terms in an order of its own (a
//                    translation unit built with --fmad=false)
//   MixedBody<Pair>  FP32 pair terms, Kahan-compensated FP32 sums over
//                    float-pair positions
// Header-only, so that a force plugin compiles the same passes with its own
// functor (psim_plugin.cuh).
#pragma once

#include <type_traits>

#include "psim_force.cuh"

namespace psim {

struct ComboPair {  // AO + LJ(n) summed; each part inside its own cutoff
    AOPair ao;
    LJPair lj;
    double rc2;
    static constexpr bool kCheckNan = true;
    __host__ __device__ __forceinline__ double fnet64(double r2, double r, double rinv, double size) const {
        double f = 0.0;
        if (r2 < ao.rc2) f += ao.fnet64(r2, r, rinv, size);
        if (r2 < lj.rc2) f += lj.fnet64(r2, r, rinv, size);
        return f;
    }
};

// F(r)/r of a pair at r^2 in FP64: a functor's own fr64(r2, size, size^2) of
// 1/r or 1/r^2 (rsqrt64 / rcp64) with fused multiply-adds, or fnet64 / r for a
// functor without one (a plugin's, the composite), which may test r or
// r^2 against distances of its own and so gets them as the reference rounds
// them (sqrt64).
// GB300 issues two FP64 operations a clock and SM, so the FP64 pass takes as
// long as it has FP64 operations: sqrt, 1/r and fnet64 in the reference's order
// were ~180 a pair, the LJ(6) form here is 12 and AO's 17.
// A functor has an fr64 of its own where its Fr64 names the functor itself: one
// derived from a library functor, with a force of its own, inherits both and is
// asked for that force.
template <class P, class = void>
struct HasFr64 : std::false_type {};
template <class P>
struct HasFr64<P, std::void_t<typename P::Fr64>> : std::is_same<typename P::Fr64, P> {};
template <class P>
__device__ __forceinline__ double pair_fr64(const P& p, double r2, double size, double s2) {
    if constexpr (HasFr64<P>::value) {
        return p.fr64(r2, size, s2);
    } else {
        const double ri = rsqrt64(r2);
        return __dmul_rn(p.fnet64(r2, sqrt64(r2, ri), ri, size), ri);
    }
}

// Plain form of one pair (i <- j), as the reference decides it: pbcDist's
// minimum image |dx| > L/2.0 (utilities.cpp:79-104) and r^2 < rc^2 on the
// r^2 it rounds product by product, the overlap check r < 0.8 size
// (AOPotential.cpp:83-88) and, for AO, the NaN check (:105-109).  Its tests run
// on the bit patterns as integers, which order like the non-negative values, and
// the exact ones only next to a threshold; the force itself is pair_fr64 on an
// r^2 summed with fused multiply-adds.  The image that unitVectorAdv takes by
// |dx| > int(L)/2 (utilities.cpp:114-142) is the same one for a pair in range
// where rc <= int(L)/2: its |dx| is below rc or above L - rc.  With
// rc <= cellSize <= L/3 that leaves a box of edge 1, whose int(L)/2 is 0: kUnitBox (a
// test per pair in every box costs a step of 4000 LJ particles 4 to 7%).
template <class Pair, bool kUnitBox = false>
struct F64Body {
    Pair pf;
    using Aux = double4_32a;  // the FP64 neighbour positions {x, y, z, R}
    static constexpr bool kBatchable = !std::is_same<Pair, ComboPair>::value;
    static constexpr bool kQuadWalk = true;   // force_quad_kernel
    static constexpr bool kUnit = kUnitBox;
    struct Home {
        double4_32a p;
        double size, s2;      // contact diameter with a neighbour of the same radius, squared
        int over_hi;          // high word of r^2 at or below which such a pair may overlap
    };
    using Shifted = Home;     // the FP64 form takes raw differences
    struct Acc {
        double n0, n1, n2;
        int cnt;
    };
    __device__ __forceinline__ const Aux* aux(const CellView& cv) const { return cv.posd; }
    // the body of replica r of a batch: its own pair functor and box
    __device__ __forceinline__ F64Body for_replica(const void* pairs, int r,
                                                   const DevGeom& g) const {
        F64Body b = *this;
        b.pf = static_cast<const Pair*>(pairs)[r];
        b.geom = g;
        return b;
    }
    __device__ __forceinline__ void init(Acc& a) const {
        a.n0 = a.n1 = a.n2 = 0.0;
        a.cnt = 0;
    }
    __device__ __forceinline__ void load_home(const CellView& cv, int i, Home& h) const {
        h.p = cv.posd[i];
        h.size = h.p.w + h.p.w;
        h.s2 = __dmul_rn(h.size, h.size);
        h.over_hi = __double2hiint(__dmul_rn(0.64, h.s2)) + 1;
    }
    __device__ __forceinline__ void shift(const Home& h, const float4&, int, int, int,
                                          const DevGeom&, Shifted& o) const {
        o = h;
    }
    // r^2 as the reference rounds it
    static __device__ __forceinline__ double r2_exact(double d0, double d1, double d2) {
        return __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
    }
    __device__ __forceinline__ void eval(const float4&, const double4_32a& pj, const Home& h,
                                         Acc& a, uint32_t& err) const {
        const DevGeom& g = geom;
        double d0 = pj.x - h.p.x, d1 = pj.y - h.p.y, d2 = pj.z - h.p.z;
        int moved = 0;   // the axes that pbcDist's image moved
        if (abs_above(d0, g.half) | abs_above(d1, g.half) | abs_above(d2, g.half)) {
            if (kUnitBox && unit_box())
                moved = (abs_above(d0, g.half) ? 1 : 0) | (abs_above(d1, g.half) ? 2 : 0) |
                        (abs_above(d2, g.half) ? 4 : 0);
            // keeps the compiler from doing the additions for every pair
            asm volatile("" : "+d"(d0), "+d"(d1), "+d"(d2));
            if (abs_above(d0, g.half)) d0 += toward(g.L, d0);
            if (abs_above(d1, g.half)) d1 += toward(g.L, d1);
            if (abs_above(d2, g.half)) d2 += toward(g.L, d2);
        }
        const double r2 = HasFr64<Pair>::value
                              ? __fma_rn(d2, d2, __fma_rn(d1, d1, __dmul_rn(d0, d0)))
                              : r2_exact(d0, d1, d2);
        // updateInteractions' test: r = sqrt(pbcDist) < 1.2 (systemHandling.cpp:112-115)
        if (count && sqrt(r2_exact(d0, d1, d2)) < cont) ++a.cnt;
        // r^2 < rc^2 by the high words (a NaN is above); where they differ by no more than
        // one, either way, the reference's r^2 decides: rounded otherwise, it can lie on the
        // other side of a change of the high word
        const int hr = __double2hiint(r2), hc = __double2hiint(pf.rc2);
        bool in = hr < hc;
        if ((unsigned)(hc - hr + 1) <= 2u) {
            asm volatile("" : "+d"(d0));
            in = r2_exact(d0, d1, d2) < pf.rc2;
        }
        if (in) {
            double size = h.size, s2 = h.s2;
            bool close = hr <= h.over_hi;
            if (__double_as_longlong(pj.w) != __double_as_longlong(h.p.w)) {
                size = h.p.w + pj.w;
                s2 = __dmul_rn(size, size);
                close = true;
            }
            if (close && sqrt(r2_exact(d0, d1, d2)) < 0.8 * size) err |= EBIT_OVERLAP;
            const double f = pair_fr64(pf, r2, size, s2);
            // a NaN, by its bits (isnan would be an FP64 operation)
            if (Pair::kCheckNan &&
                (__double_as_longlong(f) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll)
                err |= EBIT_NAN;
            if (kUnitBox && unit_box()) {
                if (!(moved & 1)) d0 = unit_image(d0);
                if (!(moved & 2)) d1 = unit_image(d1);
                if (!(moved & 4)) d2 = unit_image(d2);
            }
            a.n0 = __fma_rn(f, d0, a.n0);
            a.n1 = __fma_rn(f, d1, a.n1);
            a.n2 = __fma_rn(f, d2, a.n2);
        }
    }
    __device__ __forceinline__ void eval_quad(int, const double4_32a& pj, const Home& h, Acc& a,
                                              uint32_t& err) const {
        eval(make_float4(0.f, 0.f, 0.f, 0.f), pj, h, a, err);
    }
    // A box of edge 1 (half_uv is 0), where unitVectorAdv may take another image (a batch's
    // replicas differ).
    __device__ __forceinline__ bool unit_box() const { return __double2hiint(geom.half_uv) == 0; }
    // unitVectorAdv's image of a difference that pbcDist leaves as it is (one that
    // pbcDist moves, it moves alike)
    __device__ __forceinline__ double unit_image(double d) const {
        if (fabs(d) > geom.half_uv) d = d < 0.0 ? d + geom.L : d - geom.L;
        return d;
    }
    // L for d < 0, else -L
    static __device__ __forceinline__ double toward(double L, double d) {
        return __hiloint2double(__double2hiint(L) | (~__double2hiint(d) & 0x80000000),
                                __double2loint(L));
    }
    // |d| > h for h > 0, to 20 bits: an image's |d| is never near L/2
    static __device__ __forceinline__ bool abs_above(double d, double h) {
        return (__double2hiint(d) & 0x7fffffff) > __double2hiint(h);
    }
    __device__ __forceinline__ void fold(Acc&) const {}
    // the sums of the four lanes of a particle, added in lane order
    __device__ __forceinline__ void add_quad(Acc& a) const {
#pragma unroll
        for (int k = 1; k < 4; k <<= 1) {
            a.n0 += __shfl_xor_sync(0xffffffffu, a.n0, k);
            a.n1 += __shfl_xor_sync(0xffffffffu, a.n1, k);
            a.n2 += __shfl_xor_sync(0xffffffffu, a.n2, k);
            a.cnt += __shfl_xor_sync(0xffffffffu, a.cnt, k);
        }
    }
    // the FP64 form takes raw differences; only the FP32 test copy is imaged
    __device__ __forceinline__ void image(float4& h, double4_32a&, int sx, int sy, int sz,
                                          const DevGeom& g) const {
        h.x += (float)sx * g.Lhi;
        h.y += (float)sy * g.Lhi;
        h.z += (float)sz * g.Lhi;
    }
    __device__ __forceinline__ void partial(const Acc& a, double* red, int tid,
                                            int stride) const {
        red[0 * stride + tid] = a.n0;
        red[1 * stride + tid] = a.n1;
        red[2 * stride + tid] = a.n2;
    }
    __device__ __forceinline__ void reduce_store(const ForceOut& out, int i, const double* red,
                                                 int stride, int h, int nh, int k) const {
        double t0 = 0.0, t1 = 0.0, t2 = 0.0;
        for (int q = 0; q < k; ++q) {
            const int t = q * nh + h;
            t0 += red[0 * stride + t];
            t1 += red[1 * stride + t];
            t2 += red[2 * stride + t];
        }
        out.fx[i] = t0;
        out.fy[i] = t1;
        out.fz[i] = t2;
    }
    __device__ __forceinline__ void store(const ForceOut& out, int i, const Acc& a) const {
        out.fx[i] = a.n0;
        out.fy[i] = a.n1;
        out.fz[i] = a.n2;
        if (out.coor) out.coor[i] = a.cnt;
    }
    DevGeom geom;
    double cont = 0.0;   // count the neighbours closer than cont (ForceOut::coor)
    bool count = false;
};

struct ComboPairF {
    AOPair ao;
    LJPair lj;
    __device__ __forceinline__ float fnet32(float r2, float r, float rinv, float size) const {
        float f = 0.0f;
        if (r2 < ao.rc2f) f += ao.fnet32(r2, r, rinv, size);
        if (r2 < lj.rc2f) f += lj.fnet32(r2, r, rinv, size);
        return f;
    }
};

// The FP32 cutoff of a pair functor (the larger one for the composite).
template <class P>
__device__ __forceinline__ float pair_rc2f(const P& p) { return p.rc2f; }
__device__ __forceinline__ float pair_rc2f(const ComboPairF& p) {
    return p.ao.rc2f > p.lj.rc2f ? p.ao.rc2f : p.lj.rc2f;
}

__device__ __forceinline__ void kahan_add(float& s, float& c, float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

// One pair (i <- j) in FP32; each row's plain FP32 partial is added to the
// particle's total with Kahan compensation.
template <class Pair>
struct MixedBody {
    Pair pf;
    float rc2f;
    float cont2f = 0.f;  // > 0: count the neighbours with r^2 < cont2f (ForceOut::coor)
    using Aux = float4;  // the low parts of the neighbour positions
    static constexpr bool kBatchable = !std::is_same<Pair, ComboPairF>::value;
    static constexpr bool kQuadWalk = false;   // force_direct_kernel, force_pass_kernel
    struct Home {
        float4 lo;
    };
    struct Shifted {     // home position minus the row's image, as a float pair
        float4 h;        // xyz: high part, w: radius
        float lx, ly, lz;
    };
    struct Acc {
        float s0, s1, s2, k0, k1, k2, p0, p1, p2;
        int cnt;
    };
    __device__ __forceinline__ const Aux* aux(const CellView& cv) const { return cv.posl; }
    // the body of replica r of a batch: its own pair functor and cutoff
    __device__ __forceinline__ MixedBody for_replica(const void* pairs, int r,
                                                     const DevGeom&) const {
        MixedBody b = *this;
        b.pf = static_cast<const Pair*>(pairs)[r];
        b.rc2f = pair_rc2f(b.pf);
        return b;
    }
    __device__ __forceinline__ void init(Acc& a) const {
        a.s0 = a.s1 = a.s2 = a.k0 = a.k1 = a.k2 = a.p0 = a.p1 = a.p2 = 0.f;
        a.cnt = 0;
    }
    __device__ __forceinline__ void load_home(const CellView& cv, int i, Home& h) const {
        h.lo = cv.posl[i];
    }
    __device__ __forceinline__ void shift(const Home& h, const float4& hi, int sx, int sy, int sz,
                                          const DevGeom& g, Shifted& o) const {
        float ex, ey, ez;
        two_sum(hi.x, -(float)sx * g.Lhi, o.h.x, ex);
        two_sum(hi.y, -(float)sy * g.Lhi, o.h.y, ey);
        two_sum(hi.z, -(float)sz * g.Lhi, o.h.z, ez);
        o.h.w = hi.w;
        o.lx = (ex + h.lo.x) - (float)sx * g.Llo;
        o.ly = (ey + h.lo.y) - (float)sy * g.Llo;
        o.lz = (ez + h.lo.z) - (float)sz * g.Llo;
    }
    __device__ __forceinline__ void eval(const float4& hj, const float4& lj, const Shifted& hs,
                                         Acc& a, uint32_t& err) const {
        const float d0 = (hj.x - hs.h.x) + (lj.x - hs.lx);
        const float d1 = (hj.y - hs.h.y) + (lj.y - hs.ly);
        const float d2 = (hj.z - hs.h.z) + (lj.z - hs.lz);
        const float r2 = d0 * d0 + d1 * d1 + d2 * d2;
        if (cont2f > 0.f && r2 < cont2f) ++a.cnt;
        if (r2 < rc2f) {
            const float rinv = rsqrtf(r2);
            const float r = r2 * rinv;
            const float size = hs.h.w + hj.w;
            if (r < 0.8f * size) err |= EBIT_OVERLAP;
            const float f = pf.fnet32(r2, r, rinv, size) * rinv;
            a.p0 += f * d0;
            a.p1 += f * d1;
            a.p2 += f * d2;
        }
    }
    // the pair-list pass: one entry at separation d (the float-pair difference
    // already formed), masked by the cutoff.  kUniform: every pair has the
    // contact diameter `size` (s2 = size^2), and the overlap test runs once
    // per particle on the smallest r^2 (rmin); otherwise per pair.  bias is
    // added to r^2: 0, or the compact ghost record's kGhostBias.
    template <bool kUniform, bool kCount = false>
    __device__ __forceinline__ void eval_list(float d0, float d1, float d2, float size, float s2,
                                              Acc& a, float& rmin, uint32_t& err,
                                              float bias = 0.f) const {
        const float r2 = fmaf(d0, d0, fmaf(d1, d1, fmaf(d2, d2, bias)));
        if (kCount) a.cnt += r2 < cont2f ? 1 : 0;
        const bool in = r2 < rc2f;
        const float fr = list_fr32(pf, r2, size, s2);
        if (kUniform)
            rmin = fminf(rmin, r2);
        else if (in && r2 < 0.64f * s2)
            err |= EBIT_OVERLAP;
        const float f = in ? fr : 0.0f;
        a.p0 += f * d0;
        a.p1 += f * d1;
        a.p2 += f * d2;
    }
    // the overlap test of eval_list<true>: r < 0.8 size for an in-range pair
    __device__ __forceinline__ void list_overlap(float rmin, float s2, uint32_t& err) const {
        if (rmin < fminf(0.64f * s2, rc2f)) err |= EBIT_OVERLAP;
    }
    // the sums `own` of another lane of the same particle (mask: that
    // particle's lanes, src: the lane within its width-lane segment), added
    // into a with compensation; every lane of the mask calls it with its own
    // unmerged sums, and lane 0 keeps the result
    __device__ __forceinline__ void merge_lane(Acc& a, const Acc& own, unsigned mask, int src,
                                               int width) const {
        const float t[6] = {__shfl_sync(mask, own.s0, src, width),
                            __shfl_sync(mask, own.s1, src, width),
                            __shfl_sync(mask, own.s2, src, width),
                            __shfl_sync(mask, own.k0, src, width),
                            __shfl_sync(mask, own.k1, src, width),
                            __shfl_sync(mask, own.k2, src, width)};
        const int c = __shfl_sync(mask, own.cnt, src, width);
        kahan_add(a.s0, a.k0, t[0]);
        kahan_add(a.s1, a.k1, t[1]);
        kahan_add(a.s2, a.k2, t[2]);
        kahan_add(a.s0, a.k0, -t[3]);
        kahan_add(a.s1, a.k1, -t[4]);
        kahan_add(a.s2, a.k2, -t[5]);
        a.cnt += c;
    }
    __device__ __forceinline__ void fold(Acc& a) const {
        kahan_add(a.s0, a.k0, a.p0);
        kahan_add(a.s1, a.k1, a.p1);
        kahan_add(a.s2, a.k2, a.p2);
        a.p0 = a.p1 = a.p2 = 0.f;
    }
    // a staged neighbour with its periodic image s L applied, exactly as a
    // float pair: (h + l) + s (Lhi + Llo)
    __device__ __forceinline__ void image(float4& h, float4& l, int sx, int sy, int sz,
                                          const DevGeom& g) const {
        image_shift(h, l, sx, sy, sz, g.Lhi, g.Llo);
    }
    // per-lane partial sums for the cross-lane reduction: 6 floats per lane
    __device__ __forceinline__ void partial(const Acc& a, double* red, int tid,
                                            int stride) const {
        float* f = reinterpret_cast<float*>(red);
        f[0 * stride + tid] = a.s0;
        f[1 * stride + tid] = a.s1;
        f[2 * stride + tid] = a.s2;
        f[3 * stride + tid] = a.k0;
        f[4 * stride + tid] = a.k1;
        f[5 * stride + tid] = a.k2;
    }
    // the k lanes of home h (slots h, h + nh, ...), Kahan-summed in lane order
    __device__ __forceinline__ void reduce_store(const ForceOut& out, int i, const double* red,
                                                 int stride, int h, int nh, int k) const {
        const float* f = reinterpret_cast<const float*>(red);
        float S0 = 0.f, S1 = 0.f, S2 = 0.f, C0 = 0.f, C1 = 0.f, C2 = 0.f;
        for (int q = 0; q < k; ++q) {
            const int t = q * nh + h;
            kahan_add(S0, C0, f[0 * stride + t]);
            kahan_add(S1, C1, f[1 * stride + t]);
            kahan_add(S2, C2, f[2 * stride + t]);
            kahan_add(S0, C0, -f[3 * stride + t]);
            kahan_add(S1, C1, -f[4 * stride + t]);
            kahan_add(S2, C2, -f[5 * stride + t]);
        }
        out.fx[i] = widen_f32(S0) - widen_f32(C0);
        out.fy[i] = widen_f32(S1) - widen_f32(C1);
        out.fz[i] = widen_f32(S2) - widen_f32(C2);
    }
    // the compensated sum s - k formed in FP64 (exact: both parts fit 48
    // bits); the floats are widened with integer operations, as the FP64
    // unit that would convert them runs at 1/64 of the FP32 rate on GB300
    __device__ __forceinline__ void sum(const Acc& a, double F[3]) const {
        F[0] = widen_f32(a.s0) - widen_f32(a.k0);
        F[1] = widen_f32(a.s1) - widen_f32(a.k1);
        F[2] = widen_f32(a.s2) - widen_f32(a.k2);
    }
    __device__ __forceinline__ void store(const ForceOut& out, int i, const Acc& a) const {
        double F[3];
        sum(a, F);
        out.fx[i] = F[0];
        out.fy[i] = F[1];
        out.fz[i] = F[2];
        if (out.coor) out.coor[i] = a.cnt;
    }
};

// The plugin's pair functor handed to run(pair, rc2f): LennardJones without
// a Yukawa term gets its exponent fixed at compile time for the common ljNum
// values 6, 12 and 18, the pure Yukawa form (ljNum 0) likewise; other
// LennardJones settings run the general functor.
template <class Run>
cudaError_t with_pair(const ForceSetup& fs, Run&& run) {
    switch (fs.kind) {
    case 1: return run(fs.ao, fs.ao.rc2f);
    case 2: {
        auto fixed = [&](auto p) {
            static_cast<LJPair&>(p) = fs.lj;
            return run(p, fs.lj.rc2f);
        };
        if (fs.lj_pure) {
            switch (fs.lj.n) {
            case 6: return fixed(LJPure<6>{});
            case 12: return fixed(LJPure<12>{});
            case 18: return fixed(LJPure<18>{});
            }
        }
        if (fs.lj.n == 0) return fixed(LJFixed<0>{});
        return run(fs.lj, fs.lj.rc2f);
    }
    case 3: return run(fs.cal, fs.cal.rc2f);
    case 4: {
        const float rc2f = fs.ao.rc2f > fs.lj.rc2f ? fs.ao.rc2f : fs.lj.rc2f;
        return run(ComboPairF{fs.ao, fs.lj}, rc2f);
    }
    }
    return cudaErrorInvalidValue;
}


}  // namespace psim
