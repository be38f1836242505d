// psim_step.cu -- the mixed form's step through a pair list as one kernel.
//
// The list force pass is bound by the L1 data pipe that serves its record gathers
// and the update by HBM and issue, so a kernel that does both for each particle
// overlaps them, and the force of the step is not read back.  The new list
// records go to a second buffer (the step's parity picks it), since other
// particles still read this step's.  Each particle's arithmetic is that of
// force_list_kernel followed by vgb_system_kernel, bit for bit.
//
// It takes the normal steps of systems whose radii are all equal (compact records),
// with one lane a particle and without a plugin's device entry or the displacement
// tracker.  The first step and velocity steps run the two kernels: a velocity step
// writes the caller-visible velocities in place, which must not happen when
// another particle's force pass reports an error.
//
// Four blocks of 256 threads an SM (64 registers): a batch's kernel, which reads each
// particle's replica, takes 76 otherwise and is 12% slower.  Step time before and
// after, us: the 2^20 LJ liquid 245 -> 217, 64 AO replicas (710k particles) 98 -> 82,
// 4000 AO colloids 19.4 -> 17.
#include "psim_body.cuh"
#include "psim_force.cuh"
#include "psim_force_list.cuh"
#include "psim_vgb.cuh"

namespace psim {

namespace {

template <class Body, bool kReplicas>
__global__ void __launch_bounds__(256, 4)
step_list_kernel(Body body0, DevGeom g0, PairList pl, VgbSystemArgs a, VgbParams p, NoiseView nz) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= a.n || *a.err) return;
    typename Body::Acc acc;
    uint32_t err = 0;
    float rmin = 3.0e38f;
    double F[3];
    {
        const Body body = kReplicas ? body0.for_replica(pl.pairs, pl.rep[f], g0) : body0;
        list_terms<Body, true, false, 1>(body, pl, f, 0, acc, rmin, err);
        body.list_overlap(rmin, (2.0f * pl.radius) * (2.0f * pl.radius), err);
        body.sum(acc, F);
    }
    a.ofx[f] = F[0];
    a.ofy[f] = F[1];
    a.ofz[f] = F[2];
    if constexpr (kReplicas) {
        const int r = a.rep[f];
        VgbParams pr = p;
        pr.seed = a.seeds[r];
        vgb_normal_one(a, pr, a.geoms[r], nz, f, F, err);
    } else {
        vgb_normal_one(a, p, g0, nz, f, F, err);
    }
}

// The normal step without a pair list: the direct walk and the update in one kernel.
// The walk is bound by issue and the update by HBM and the latency of its gathers.
// us a step as two kernels and as one: AO colloids 1001 / 4000 / 20001 / 65537 / 300001
// particles 19.1 / 22.3 / 29.5 / 32.2 / 67.5 -> 16.6 / 19.4 / 26.7 / 29.0 / 65.0, the LJ liquid
// of 13500 / 108000 85.8 / 121.9 -> 77.4 / 109.8; the gel of 2^20 / 2^21 187.6 / 350.7 against
// 192.5 / 361.7 and the liquid of 2^20 706 against 710 (79 registers: fewer warps to walk
// with), so up to 3 2^17 particles.
template <class Body>
__global__ void __launch_bounds__(kForceWarps * 32, 5)
step_direct_kernel(Body body, DevGeom g, CellView cv, ForceOut out, float pre_rc2, VgbSystemArgs a,
                   VgbParams p, NoiseView nz) {
    __shared__ uint32_t s_q[kForceWarps][kQueueCap][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (pass_failed(out, lane)) return;  // warp-uniform
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = i < g.p1;
    typename Body::Acc acc;
    uint32_t err = 0;
    direct_terms(body, g, cv, pre_rc2, i, active, lane, s_q[w], acc, err);
    if (!active) return;
    double F[3];
    body.sum(acc, F);
    a.ofx[i] = F[0];
    a.ofy[i] = F[1];
    a.ofz[i] = F[2];
    vgb_normal_moved(a, p, g, nz, i, F, err);
}

}  // namespace

bool step_direct_fits(const ForceSetup& fs, const DevGeom& g) {
    return !fs.tile && direct_walk(g, fs.walk);
}

cudaError_t launch_step_direct(const ForceSetup& fs, const DevGeom& g, const CellView& cv,
                               const ForceOut& out, const VgbSystemArgs& a, const VgbParams& p,
                               const NoiseView& nz, cudaStream_t st) {
    if (g.n == 0) return cudaSuccess;
    return with_pair(fs, [&](auto pair, float rc2f) -> cudaError_t {
        using Body = MixedBody<decltype(pair)>;
        const int threads = kForceWarps * 32;
        step_direct_kernel<Body><<<(g.n + threads - 1) / threads, threads, 0, st>>>(
            Body{pair, rc2f}, g, cv, out, fs.pre_rc2f, a, p, nz);
        return cudaGetLastError();
    });
}

cudaError_t launch_step_list(const ForceSetup& fs, const DevGeom& g, const PairList& pl,
                             const VgbSystemArgs& a, const VgbParams& p, const NoiseView& nz,
                             cudaStream_t st) {
    if (a.n == 0) return cudaSuccess;
    return with_pair(fs, [&](auto pair, float rc2f) -> cudaError_t {
        using Body = MixedBody<decltype(pair)>;
        const Body body{pair, rc2f};
        const int threads = block_threads(a.n), blocks = (a.n + threads - 1) / threads;
        if (pl.rep) {
            if constexpr (Body::kBatchable) {
                step_list_kernel<Body, true><<<blocks, threads, 0, st>>>(body, g, pl, a, p, nz);
                return cudaGetLastError();
            }
            return cudaErrorInvalidValue;
        }
        step_list_kernel<Body, false><<<blocks, threads, 0, st>>>(body, g, pl, a, p, nz);
        return cudaGetLastError();
    });
}

}  // namespace psim
