// psim_observe.cu -- observables of the device-resident state: the analysis
// the reference runs between steps, on the GPU so the state stays in HBM.
//
//   temperature          analysisManager::getTemperature  (analysisGeneral.cpp:26-43)
//   mean displacement    analysisManager::meanDisplacement (analysisGeneral.cpp:45-55)
//   tracked displacement trackedDisplacement (analysisTracker.cpp:26-85), every wrap counted
//   potential ("EAP")    particle::calculatePotential (particle.cpp:133-149), summed
//   coordination         system::updateInteractions (systemHandling.cpp:94-161)
//   g(r)                 a pair-distance histogram over the same 27-cell walk
//   energy and virial    FP64 sums over pairs of the plugin's u(r) and r.f
//
// Sums are deterministic: each block writes its partial, one block adds the
// partials in block order.
#include <algorithm>
#include <cmath>

#include "psim_force.cuh"

namespace psim {

namespace {

constexpr int kRedThreads = 256;
constexpr int kRedBlocks = 512;

__device__ double block_sum(double v, double* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += sh[k];
    __syncthreads();
    return t;  // valid in thread 0
}

// out[b] = the sum of partials b n .. b n + n - 1 (block b)
__global__ void __launch_bounds__(kRedThreads) finish_kernel(const double* part, int n, double* out) {
    __shared__ double sh[kRedThreads / 32];
    // each thread adds a fixed stride of partials, then the block in lane order
    double v = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) v += part[(size_t)blockIdx.x * n + k];
    const double t = block_sum(v, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = t;
}

// sum of |v|^2 over count values
__global__ void __launch_bounds__(kRedThreads) sumsq_kernel(long long count, const double* v,
                                                            double* part) {
    __shared__ double sh[kRedThreads / 32];
    double s = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
         i += (long long)gridDim.x * blockDim.x)
        s += v[i] * v[i];
    const double t = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

__global__ void __launch_bounds__(kRedThreads) observe_kernel(ObserveArgs a, double* part) {
    __shared__ double sh[kRedThreads / 32];
    double s = 0.0;
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < a.n; f += gridDim.x * blockDim.x) {
        const double x[3] = {a.x[f], a.y[f], a.z[f]};
        if (a.what == OBS_MEAN_DISP) {
            const double d0 = x[0] - a.x0[f], d1 = x[1] - a.y0[f], d2 = x[2] - a.z0[f];
            s += d0 * d0 + d1 * d1 + d2 * d2;
        } else if (a.what == OBS_TRACKED) {
            const int t = a.tag[f];
            for (int k = 0; k < 3; ++k) {
                // the reference sums this in FP32 (analysisTracker.cpp:68-83)
                const double d = (x[k] + a.L * a.img[3 * (size_t)t + k]) - a.start[3 * (size_t)t + k];
                s += d * d;
            }
        } else {  // OBS_POTENTIAL: particle::calculatePotential in FP32
            const int o = a.perm_prev ? a.perm_prev[f] : f;
            const float dx = (float)(x[0] - a.x0[f]), dy = (float)(x[1] - a.y0[f]),
                        dz = (float)(x[2] - a.z0[f]);
            const double F[3] = {a.fx[f], a.fy[f], a.fz[f]};
            const double G[3] = {a.gx[o], a.gy[o], a.gz[o]};
            const float dfx = (float)(F[0] - G[0]), dfy = (float)(F[1] - G[1]),
                        dfz = (float)(F[2] - G[2]);
            const float dr = sqrtf(dx * dx + dy * dy + dz * dz);
            const float df = sqrtf(dfx * dfx + dfy * dfy + dfz * dfz);
            const float f0 = sqrtf((float)(G[0] * G[0] + G[1] * G[1] + G[2] * G[2]));
            const float p = (f0 * dr) + (0.5f * df * dr);
            s += (double)(-p);
        }
    }
    const double t = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// ------------------------------------------------------------ pair walks
//
// The pairs of the current cell list through the four-lane walk of the FP64 force
// pass (force_quad_kernel): FP32 positions with a margin reject the candidates out of
// range, so that the FP64 distance, pbcDist's minimum image (utilities.cpp:79-104), is
// formed for the others only, with full warps.  At 131072 particles, a thread per
// particle with FP64 distances to all 27 cells before, and now (whole calls): energy
// 1050 -> 175 us, coordination 1251 -> 141, g(r) 1314 -> 166.

__device__ __forceinline__ CellView scan_cells(const PairScanArgs& a) {
    return CellView{a.posd, a.posh, nullptr, a.cellid, a.cstart, a.ccount};
}
__device__ __forceinline__ double scan_r2(const DevGeom& g, const double4_32a& pi,
                                          const double4_32a& pj) {
    double d0 = fabs(pj.x - pi.x), d1 = fabs(pj.y - pi.y), d2 = fabs(pj.z - pi.z);
    if (d0 > g.half) d0 -= g.L;
    if (d1 > g.half) d1 -= g.L;
    if (d2 > g.half) d2 -= g.L;
    return d0 * d0 + d1 * d1 + d2 * d2;
}

constexpr int kScanBlocks = 152 * 12;   // at most; each block takes every gridDim-th group

// updateInteractions' count (systemHandling.cpp:94-161): neighbours closer than
// r_contact; distances in [r_min, r_max) are binned for g(r).
struct ScanBody {
    PairScanArgs a;
    unsigned int* hist;
    using Aux = double4_32a;
    struct Home {
        double4_32a p;
    };
    struct Acc {
        int coor;
    };
    __device__ __forceinline__ const Aux* aux(const CellView& cv) const { return cv.posd; }
    __device__ __forceinline__ void init(Acc& c) const { c.coor = 0; }
    __device__ __forceinline__ void load_home(const CellView& cv, int i, Home& h) const {
        h.p = cv.posd[i];
    }
    __device__ __forceinline__ void eval_quad(int, const double4_32a& pj, const Home& h, Acc& c,
                                              uint32_t&) const {
        const double r = sqrt(scan_r2(a.g, h.p, pj));
        if (r < a.r_contact) ++c.coor;
        if (a.n_bins > 0 && r >= a.r_min && r < a.r_max) {
            const int b = (int)((r - a.r_min) * a.inv_dr);
            atomicAdd(&hist[b < a.n_bins ? b : a.n_bins - 1], 1u);
        }
    }
};

__global__ void __launch_bounds__(kQuadWarps * 32) pairs_kernel(PairScanArgs a) {
    extern __shared__ unsigned int hist[];
    __shared__ uint32_t s_q[kQuadWarps][8][kQuadStride];
    for (int b = threadIdx.x; b < a.n_bins; b += blockDim.x) hist[b] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const ScanBody body{a, hist};
    const CellView cv = scan_cells(a);
    const int per = 8 * kQuadWarps, groups = (a.g.n + per - 1) / per;
    long long total = 0;
    for (int k = blockIdx.x; k < groups; k += gridDim.x) {
        const int i = k * per + 8 * w + (lane >> 2);
        ScanBody::Acc c;
        uint32_t err = 0;
        quad_walk(body, a.g, cv, a.pre_r2, i, lane, s_q[w], c, err);
        int coor = c.coor + __shfl_xor_sync(0xffffffffu, c.coor, 1);
        coor += __shfl_xor_sync(0xffffffffu, coor, 2);
        if (i < a.g.n && (lane & 3) == 0) {
            if (a.coor) a.coor[a.tag[i]] = coor;
            total += coor;
        }
    }
    if (a.n_pairs) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        if (lane == 0 && total) atomicAdd(a.n_pairs, (unsigned long long)total);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < a.n_bins; b += blockDim.x)
        if (hist[b]) atomicAdd(&a.hist[b], (unsigned long long)hist[b]);
}

// ---------------------------------------------------------------- clusters
// Connected components of the contact graph (r < r_contact), the clusters of
// analysisManager::findClusters (analysisCluster.cpp:26-62), by lock-free
// union-find over original indices: an edge hooks the larger of its two roots
// under the smaller with atomicCAS, so each component's root ends as its
// smallest original index -- the order findClusters visits clusters in.
// Parents always have smaller indices, so a chain is at most n long and a
// failed hook means the root was hooked by another thread (at most n times);
// both loops are capped at n + 1 anyway and report EBIT_INDEX past it.

__device__ int uf_find(const int* label, int x, int n, uint32_t& err) {
    int p = ((const volatile int*)label)[x];
    for (int k = 0; p != x; ++k) {
        if (k > n) {
            err |= EBIT_INDEX;
            return x;
        }
        x = p;
        p = ((const volatile int*)label)[x];
    }
    return x;
}

__device__ void uf_union(int* label, int a, int b, int n, uint32_t& err) {
    for (int it = 0; it <= n; ++it) {
        a = uf_find(label, a, n, err);
        b = uf_find(label, b, n, err);
        if (a == b || err) return;
        if (a > b) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicCAS(&label[b], b, a);
        if (old == b) return;   // hooked; else b gained a parent meanwhile: retry
    }
    err |= EBIT_INDEX;
}

__global__ void __launch_bounds__(256) uf_init_kernel(int n, int* label) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) label[i] = i;
}

struct EdgeBody {
    PairScanArgs a;
    int* label;
    using Aux = double4_32a;
    struct Home {
        double4_32a p;
        int tag;
    };
    struct Acc {};
    __device__ __forceinline__ const Aux* aux(const CellView& cv) const { return cv.posd; }
    __device__ __forceinline__ void init(Acc&) const {}
    __device__ __forceinline__ void load_home(const CellView& cv, int i, Home& h) const {
        h.p = cv.posd[i];
        h.tag = a.tag[i];
    }
    __device__ __forceinline__ void eval_quad(int j, const double4_32a& pj, const Home& h, Acc&,
                                              uint32_t& err) const {
        const int tj = a.tag[j];
        if (tj <= h.tag) return;   // each undirected edge once
        if (sqrt(scan_r2(a.g, h.p, pj)) < a.r_contact) uf_union(label, h.tag, tj, a.g.n, err);
    }
};

__global__ void __launch_bounds__(kQuadWarps * 32)
uf_edges_kernel(PairScanArgs a, int* label, uint32_t* err_out) {
    __shared__ uint32_t s_q[kQuadWarps][8][kQuadStride];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    EdgeBody::Acc c;
    uint32_t err = 0;
    quad_walk(EdgeBody{a, label}, a.g, scan_cells(a), a.pre_r2,
              (blockIdx.x * kQuadWarps + w) * 8 + (lane >> 2), lane, s_q[w], c, err);
    if (err) atomicOr(err_out, err);
}

__global__ void __launch_bounds__(256) uf_final_kernel(int n, const int* label, int* root,
                                                        int* size, uint32_t* err_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t err = 0;
    const int r = uf_find(label, i, n, err);
    root[i] = r;
    atomicAdd(&size[r], 1);
    if (err) atomicOr(err_out, err);
}

// ------------------------------------------------------ energy and virial
// AO with its cutoff's constants, formed once for all pairs.
struct AOEnergy : AOPair {
    double rc, e37;
    explicit AOEnergy(const AOPair& p) : AOPair(p), rc(std::sqrt(p.rc2)) {
        e37 = pow36(1.0 / rc) * (1.0 / rc);
    }
    __device__ __forceinline__ double u64(double r2, double, double rinv, double) const {
        return u64_at(r2, rinv, rc, e37);
    }
};
// One pair term of the energy walk: u(r) and fNet(r) inside the cutoff.
template <class Pair>
struct OneTerm {
    Pair p;
    __device__ double rc2() const { return p.rc2; }
    __device__ void eval(double r2, double r, double rinv, double size, double& u,
                         double& f) const {
        if (r2 < p.rc2) {
            u += p.u64(r2, r, rinv, size);
            f += p.fnet64(r2, r, rinv, size);
        }
    }
};
struct ComboTerms {  // the AO + LJ(n) composite: each part inside its own cutoff
    AOEnergy ao;
    LJPair lj;
    __device__ double rc2() const { return ao.rc2 > lj.rc2 ? ao.rc2 : lj.rc2; }
    __device__ void eval(double r2, double r, double rinv, double size, double& u,
                         double& f) const {
        if (r2 < ao.rc2) {
            u += ao.u64(r2, r, rinv, size);
            f += ao.fnet64(r2, r, rinv, size);
        }
        if (r2 < lj.rc2) {
            u += lj.u64(r2, r, rinv, size);
            f += lj.fnet64(r2, r, rinv, size);
        }
    }
};

// Per particle i: half the sum over its neighbours j of u(r_ij) and of
// r_ij . f_ij = -fNet(r_ij) r_ij, in FP64, then summed over the particles in a fixed
// order.
template <class Terms>
struct EnergyBody {
    Terms t;
    DevGeom g;
    double rc2;
    using Aux = double4_32a;
    struct Home {
        double4_32a p;
    };
    struct Acc {
        double u, w;
    };
    __device__ __forceinline__ const Aux* aux(const CellView& cv) const { return cv.posd; }
    __device__ __forceinline__ void init(Acc& c) const { c.u = c.w = 0.0; }
    __device__ __forceinline__ void load_home(const CellView& cv, int i, Home& h) const {
        h.p = cv.posd[i];
    }
    __device__ __forceinline__ void eval_quad(int, const double4_32a& pj, const Home& h, Acc& c,
                                              uint32_t&) const {
        const double r2 = scan_r2(g, h.p, pj);
        if (!(r2 < rc2)) return;
        const double r = sqrt(r2), rinv = 1.0 / r;
        double u = 0.0, f = 0.0;
        t.eval(r2, r, rinv, h.p.w + pj.w, u, f);
        c.u += u;
        c.w -= f * r;
    }
};

template <class Terms>
__global__ void __launch_bounds__(kQuadWarps * 32)
energy_kernel(PairScanArgs a, Terms t, double* part) {
    __shared__ uint32_t s_q[kQuadWarps][8][kQuadStride];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = (blockIdx.x * kQuadWarps + w) * 8 + (lane >> 2);
    const EnergyBody<Terms> body{t, a.g, t.rc2()};
    typename EnergyBody<Terms>::Acc c;
    uint32_t err = 0;
    quad_walk(body, a.g, scan_cells(a), a.pre_r2, i, lane, s_q[w], c, err);
#pragma unroll
    for (int k = 1; k < 4; k <<= 1) {
        c.u += __shfl_xor_sync(0xffffffffu, c.u, k);
        c.w += __shfl_xor_sync(0xffffffffu, c.w, k);
    }
    if (i < a.g.n && (lane & 3) == 0) {
        part[i] = 0.5 * c.u;
        part[a.g.n + i] = 0.5 * c.w;
    }
}

// block partials of the two rows of v[2][n]
__global__ void __launch_bounds__(kRedThreads) rows_kernel(int n, const double* v, double* part) {
    __shared__ double sh[kRedThreads / 32];
    double t = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        t += v[(size_t)blockIdx.y * n + i];
    t = block_sum(t, sh);
    if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = t;
}

template <class Terms>
cudaError_t run_energy(const Terms& t, const PairScanArgs& a, double* scratch, double* out,
                       cudaStream_t st) {
    const int per = 8 * kQuadWarps, n = a.g.n;
    energy_kernel<Terms><<<(n + per - 1) / per, kQuadWarps * 32, 0, st>>>(a, t, scratch);
    double* part = scratch + 2 * (size_t)n;
    rows_kernel<<<dim3(kRedBlocks, 2), kRedThreads, 0, st>>>(n, scratch, part);
    finish_kernel<<<2, kRedThreads, 0, st>>>(part, kRedBlocks, out);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_energy(const ForceSetup& fs, const PairScanArgs& a, double* scratch,
                          double* out, cudaStream_t st) {
    if (a.g.n == 0) return cudaMemsetAsync(out, 0, 2 * sizeof(double), st);
    switch (fs.kind) {
    case 1: return run_energy(OneTerm<AOEnergy>{AOEnergy(fs.ao)}, a, scratch, out, st);
    case 2: return run_energy(OneTerm<LJPair>{fs.lj}, a, scratch, out, st);
    case 3: return run_energy(OneTerm<CalPair>{fs.cal}, a, scratch, out, st);
    case 4: return run_energy(ComboTerms{AOEnergy(fs.ao), fs.lj}, a, scratch, out, st);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_clusters(const PairScanArgs& a, int* label, int* root, int* size,
                            uint32_t* err, cudaStream_t st) {
    const int n = a.g.n;
    if (n == 0) return cudaSuccess;
    uf_init_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, label);
    const int per = 8 * kQuadWarps;
    uf_edges_kernel<<<(n + per - 1) / per, kQuadWarps * 32, 0, st>>>(a, label, err);
    uf_final_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, label, root, size, err);
    return cudaGetLastError();
}

cudaError_t launch_sum_squares(long long count, const double* v, double* scratch, double* out,
                               cudaStream_t st) {
    sumsq_kernel<<<kRedBlocks, kRedThreads, 0, st>>>(count, v, scratch);
    finish_kernel<<<1, kRedThreads, 0, st>>>(scratch, kRedBlocks, out);
    return cudaGetLastError();
}

cudaError_t launch_observe(const ObserveArgs& a, double* scratch, double* out, cudaStream_t st) {
    observe_kernel<<<kRedBlocks, kRedThreads, 0, st>>>(a, scratch);
    finish_kernel<<<1, kRedThreads, 0, st>>>(scratch, kRedBlocks, out);
    return cudaGetLastError();
}

int observe_scratch_doubles() { return kRedBlocks; }
size_t energy_scratch_doubles(int n) { return 2 * (size_t)n + 2 * kRedBlocks; }

cudaError_t launch_pair_scan(const PairScanArgs& a, cudaStream_t st) {
    if (a.g.n == 0) return cudaSuccess;
    const size_t smem = sizeof(unsigned int) * (size_t)(a.n_bins > 0 ? a.n_bins : 1);
    const int per = 8 * kQuadWarps, groups = (a.g.n + per - 1) / per;
    pairs_kernel<<<std::min(groups, kScanBlocks), kQuadWarps * 32, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace psim
