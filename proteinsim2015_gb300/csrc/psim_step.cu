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

}  // namespace

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
