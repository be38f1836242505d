// psim_exact.cu -- FP64 kernels, compiled with --fmad=false so every a*b+c
// rounds twice as in the reference's x86-64 build (no FMA contraction).
//
//   F64Body             plain form of the plugin force pass (the pair body of
//                       force_quad_kernel, psim_force.cuh)
//   step_quad_kernel    that pass and the update of a small system in one
//   vgb_system_kernel   brownianIntegrator::nextSystem fused with the gather
//                       into the new cell order and the cell hash + count of
//                       the next rebuild (brownianIntegrator.cpp:181-356,
//                       systemHandling.cpp:33-48)
//   vgb_aos_kernel      nextSystem on the reference's own AoS arrays
//   hash_count_kernel   system::hashParticles + the counting-sort histogram
#include <cmath>

#include "psim_body.cuh"
#include "psim_force.cuh"
#include "psim_force_cell.cuh"
#include "psim_vgb.cuh"

namespace psim {

// ------------------------------------------------------------------ forces

template <class Pair>
static cudaError_t run_fp64(const Pair& p, const DevGeom& g, const CellView& cv,
                            const ForceOut& out, const ForceSetup& fs, cudaStream_t st,
                            const BatchView* bv) {
    auto run = [&](auto body) {
        body.count = out.coor && out.cont > 0.0;   // updateInteractions fused into the pass
        body.cont = out.cont;
        if constexpr (!decltype(body)::kUnit)
            if (fs.tile && !bv) return launch_force_cells(body, g, cv, out, fs.pre_rc2f, st);
        return launch_force_pass(body, g, cv, out, fs.pre_rc2f, st, bv);
    };
    return fs.unit_box ? run(F64Body<Pair, true>{p, g}) : run(F64Body<Pair>{p, g});
}

template <int N>
static cudaError_t run_lj_fp64(const DevGeom& g, const CellView& cv, const ForceOut& out,
                               const ForceSetup& fs, cudaStream_t st, const BatchView* bv) {
    LJFixed<N> p;
    static_cast<LJPair&>(p) = fs.lj;
    return run_fp64(p, g, cv, out, fs, st, bv);
}

cudaError_t launch_forces_fp64(const ForceSetup& fs, const DevGeom& g, const CellView& cv,
                               const ForceOut& out, cudaStream_t st, const BatchView* bv) {
    switch (fs.kind) {
    case 1: return run_fp64(fs.ao, g, cv, out, fs, st, bv);
    case 2:
        switch (fs.lj.n) {
        case 0: return run_lj_fp64<0>(g, cv, out, fs, st, bv);
        case 6: return run_lj_fp64<6>(g, cv, out, fs, st, bv);
        case 12: return run_lj_fp64<12>(g, cv, out, fs, st, bv);
        case 18: return run_lj_fp64<18>(g, cv, out, fs, st, bv);
        default: return run_fp64(fs.lj, g, cv, out, fs, st, bv);
        }
    case 3: return run_fp64(fs.cal, g, cv, out, fs, st, bv);
    case 4: {
        if (bv) return cudaErrorInvalidValue;  // batches hold single-plugin replicas
        ComboPair cp{fs.ao, fs.lj, fs.ao.rc2 > fs.lj.rc2 ? fs.ao.rc2 : fs.lj.rc2};
        return run_fp64(cp, g, cv, out, fs, st, bv);
    }
    }
    return cudaErrorInvalidValue;
}

// ------------------------------------------------- force and update, few particles
//
// A normal step of a small system in one kernel: the four lanes a particle has in the
// force walk hold its force, and three of them update an axis each.  On few particles a
// step is launches and chains of FP64 operations (~68 clocks each for a lone warp), and
// this shortens both: a launch less, a third of the update's chain, and the state read
// while the walk runs.  Each axis' arithmetic is vgb_particle's.  For many particles the
// update's instructions with three lanes of four full cost more than the launch.
// us a step as two kernels and as one: AO colloids 1001 / 4000 / 8000 / 12000 / 16000 /
// 20001 particles 19.5 / 21.5 / 22.5 / 24.0 / 27.6 / 29.5 against 16.4 / 18.3 / 19.7 / 22.1 /
// 26.5 / 33.6 (its 112 registers hold eight blocks an SM, 19456 particles); the LJ liquid of
// 4000 / 13500 51.5 / 70.4 against 48.1 / 68.8.
template <class Body>
__global__ void __launch_bounds__(kQuadWarps * 32, 8)
step_quad_kernel(Body body, DevGeom g, CellView cv, ForceOut out, float pre_rc2, VgbSystemArgs a,
                 VgbParams p, NoiseView nz) {
    __shared__ uint32_t s_q[kQuadWarps][8][kQuadStride];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (pass_failed(out, lane)) return;  // warp-uniform
    const int i = (blockIdx.x * kQuadWarps + w) * 8 + (lane >> 2), m = lane & 3;
    const bool active = i < g.p1, mine = active && m < 3;
    const long long step = a.state->step;
    int tag = 0;
    double mass = 1.0, x = 0.0, x0 = 0.0, mx = 0.0, F0 = 0.0;
    if (mine) {
        tag = a.tag[i];
        mass = a.inv_mass[i];
        const int o = a.perm[i];
        x = (m == 0 ? a.x : (m == 1 ? a.y : a.z))[o];
        x0 = (m == 0 ? a.x0 : (m == 1 ? a.y0 : a.z0))[o];
        mx = (m == 0 ? a.mx : (m == 1 ? a.my : a.mz))[o];
        F0 = (m == 0 ? a.gx : (m == 1 ? a.gy : a.gz))[o];
    }
    typename Body::Acc acc;
    uint32_t err = 0;
    quad_walk(body, g, cv, pre_rc2, i, lane, s_q[w], acc, err);
    body.add_quad(acc);
    if (active && m == 0) body.store(out, i, acc);
    int cell = 0;
    if (mine) {
        double xi[6], xn, x0n;
        load_noise(nz, p.seed, a.n, tag, tag - g.p0, step, xi, err);
        const double F = m == 0 ? acc.n0 : (m == 1 ? acc.n1 : acc.n2);
        const double xk = m == 0 ? xi[0] : (m == 1 ? xi[1] : xi[2]);
        const double xm = m == 0 ? xi[3] : (m == 1 ? xi[4] : xi[5]);
        vgb_normal_axis(p, g.L, g.half, x, x0, mx, F, F0, xk, xm, mass, xn, x0n, err);
        (m == 0 ? a.ox : (m == 1 ? a.oy : a.oz))[i] = xn;
        (m == 0 ? a.ox0 : (m == 1 ? a.oy0 : a.oz0))[i] = x0n;
        (m == 0 ? a.omx : (m == 1 ? a.omy : a.omz))[i] = mx;
        cell = hash_axis(xn, g, err) * (m == 0 ? 1 : (m == 1 ? g.s : g.s2));
    }
    cell += __shfl_xor_sync(0xffffffffu, cell, 1);
    cell += __shfl_xor_sync(0xffffffffu, cell, 2);
    if (active && m == 0) a.key[i] = g.c0 + cell;
    if (err) atomicOr(out.err, err);
}

template <class Pair>
static cudaError_t run_step_fp64(const Pair& pair, const DevGeom& g, const CellView& cv,
                                 const ForceOut& out, float pre, const VgbSystemArgs& a,
                                 const VgbParams& p, const NoiseView& nz, cudaStream_t st) {
    using Body = F64Body<Pair>;
    Body body{pair, g};
    const int per = 8 * kQuadWarps;
    step_quad_kernel<Body><<<(g.n + per - 1) / per, kQuadWarps * 32, 0, st>>>(body, g, cv, out, pre,
                                                                             a, p, nz);
    return cudaGetLastError();
}

template <int N>
static cudaError_t run_step_lj(const LJPair& lj, const DevGeom& g, const CellView& cv,
                               const ForceOut& out, float pre, const VgbSystemArgs& a,
                               const VgbParams& p, const NoiseView& nz, cudaStream_t st) {
    LJFixed<N> f;
    static_cast<LJPair&>(f) = lj;
    return run_step_fp64(f, g, cv, out, pre, a, p, nz, st);
}

cudaError_t launch_step_fp64(const ForceSetup& fs, const DevGeom& g, const CellView& cv,
                             const ForceOut& out, const VgbSystemArgs& a, const VgbParams& p,
                             const NoiseView& nz, cudaStream_t st) {
    if (g.n == 0) return cudaSuccess;
    const float pre = fs.pre_rc2f;
    switch (fs.kind) {
    case 1: return run_step_fp64(fs.ao, g, cv, out, pre, a, p, nz, st);
    case 2:
        switch (fs.lj.n) {
        case 0: return run_step_lj<0>(fs.lj, g, cv, out, pre, a, p, nz, st);
        case 6: return run_step_lj<6>(fs.lj, g, cv, out, pre, a, p, nz, st);
        case 12: return run_step_lj<12>(fs.lj, g, cv, out, pre, a, p, nz, st);
        case 18: return run_step_lj<18>(fs.lj, g, cv, out, pre, a, p, nz, st);
        default: return run_step_fp64(fs.lj, g, cv, out, pre, a, p, nz, st);
        }
    case 3: return run_step_fp64(fs.cal, g, cv, out, pre, a, p, nz, st);
    case 4: {
        ComboPair cp{fs.ao, fs.lj, fs.ao.rc2 > fs.lj.rc2 ? fs.ao.rc2 : fs.lj.rc2};
        return run_step_fp64(cp, g, cv, out, pre, a, p, nz, st);
    }
    }
    return cudaErrorInvalidValue;
}

// -------------------------------------------------------------- integrator
// The update is psim_vgb.cuh; this translation unit is built without FMA
// contraction, so these instances round every product and sum separately,
// in the reference's order.

cudaError_t launch_vgb_system(const VgbSystemArgs& a, const VgbParams& p, const DevGeom& g,
                              const NoiseView& nz, cudaStream_t st) {
    return launch_vgb_system_t<VgbExact>(a, p, g, nz, st);
}

cudaError_t launch_vgb_aos(const VgbAosArgs& a, const VgbParams& p, double L, cudaStream_t st) {
    if (a.n == 0) return cudaSuccess;
    vgb_aos_kernel<VgbExact><<<(a.n + 255) / 256, 256, 0, st>>>(a, p, L);
    return cudaGetLastError();
}

cudaError_t launch_vgb_host(const VgbHostArgs& a, const VgbParams& p, double L, cudaStream_t st) {
    if (a.n == 0) return cudaSuccess;
    vgb_host_kernel<VgbExact><<<(a.n + kHostBlock - 1) / kHostBlock, kHostBlock, 0, st>>>(a, p, L);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ hashing

__global__ void __launch_bounds__(256)
hash_count_kernel(int n, const double* x, const double* y, const double* z, DevGeom g0,
                  int* key, int* rank, int* count, uint32_t* err_out, const int* rep,
                  const DevGeom* geoms) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t err = 0;
    const double p[3] = {x[i], y[i], z[i]};
    const int k = hash_pos(p, rep ? geoms[rep[i]] : g0, err);
    key[i] = k;
    rank[i] = atomicAdd(&count[k], 1);
    if (err) atomicOr(err_out, err);
}

cudaError_t launch_hash_count(int n, const double* x, const double* y, const double* z,
                              const DevGeom& g, int* key, int* rank, int* count, uint32_t* err,
                              cudaStream_t st, const int* rep, const DevGeom* geoms) {
    if (n == 0) return cudaSuccess;
    hash_count_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, x, y, z, g, key, rank, count, err, rep,
                                                       geoms);
    return cudaGetLastError();
}

}  // namespace psim
