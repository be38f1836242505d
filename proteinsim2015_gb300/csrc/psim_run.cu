// psim_run.cu -- many steps of a small system through its pair list in one kernel.
//
// A step of a few thousand particles is a few microseconds of work behind the launch
// of its two kernels.  Here one cluster of 16 blocks, a thread per particle, runs a
// whole stretch of normal steps: a particle's state stays in its thread's registers, a
// step ends at one hardware cluster barrier, and a rebuild (hash, cell order, list) runs
// in the same kernel, a barrier between its phases.  The next step's random numbers are
// drawn while the barrier completes.  The arithmetic per particle, the list order and
// the storage between calls are those of step_list_kernel and the rebuild kernels, so
// the results are the same bit for bit.
//
// Everything a step reads was written by other blocks of this kernel a barrier earlier:
// plain loads, never the read-only path.
//
// What bounds a step is latency: a barrier, then per thread a chain of list groups,
// records and pair terms in order (a particle's sum keeps one lane and its order), then
// the update's FP64 chain.  Up to 8192 particles (a thread each in 16 blocks of 512:
// the registers of an SM) whose cells fit the order's shared memory.
// us a step, one kernel for stretches of 25 against a graph of steps of two kernels:
//   AO 100 / 1001 / 4000 / 8192 particles   5.5 / 5.9 / 6.5 / 8.3 against 8.4 / 9.3 / 9.5 / 9.2
//   LJ liquid (rc 2.5, density 0.38) 4000 / 6912   14.9 / 19.3 against 20.2 / 19.6
// (17.4 to 27.7 when each step had a conditional node for its rebuild).
#include <cooperative_groups.h>

#include "psim_body.cuh"
#include "psim_cells.cuh"
#include "psim_force_list.cuh"
#include "psim_list_build.cuh"
#include "psim_vgb.cuh"

namespace psim {

namespace {

namespace cg = cooperative_groups;

constexpr int kRunBlocks = 16;        // the largest cluster (beyond the portable 8)
constexpr int kRunThreads = 512;      // threads per block at most

// what a thread reports at a step's barrier
constexpr uint32_t kRunMoved = 1u, kRunError = 2u;

__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    cluster_arrive();
    cluster_wait();
}

// A particle's state between steps t - 1 and t: x_t, x_{t-1} (re-imaged), the noise
// memory and the last two forces.
struct RunState {
    double x[3], x0[3], mx[3], F0[3], F00[3];
};

// at the buffers of step t, slot f
__device__ __forceinline__ void load_state(const RunArgs& a, long long t, int f, RunState& s) {
    const int q = (int)(t & 1), r = (int)(t % 3), n = a.n;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s.x[k] = a.pos[q][(size_t)k * n + f];
        s.x0[k] = a.pos0[q][(size_t)k * n + f];
        s.mx[k] = a.mem[q][(size_t)k * n + f];
        s.F0[k] = a.frc[r][(size_t)k * n + f];
        s.F00[k] = a.frc[(r + 2) % 3][(size_t)k * n + f];
    }
}
__device__ __forceinline__ void store_state(const RunArgs& a, long long t, int f,
                                            const RunState& s) {
    const int q = (int)(t & 1), r = (int)(t % 3), n = a.n;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a.pos[q][(size_t)k * n + f] = s.x[k];
        a.pos0[q][(size_t)k * n + f] = s.x0[k];
        a.mem[q][(size_t)k * n + f] = s.mx[k];
        a.frc[r][(size_t)k * n + f] = s.F0[k];
        a.frc[(r + 2) % 3][(size_t)k * n + f] = s.F00[k];
    }
}


// The rebuild before step t: the state into the new cell order, the list on it.
// False, in every thread, where it failed.
__device__ __forceinline__ bool run_rebuild(const RunArgs& a, const DevGeom& g, long long t,
                                            int f, bool active, int* smem,
                                            cg::cluster_group& cluster, RunState& s, int& tag,
                                            double& m) {
    const int q = (int)(t & 1);
    if (active) store_state(a, t, f, s);
    if (active) {
        uint32_t err = 0;
        const int key = hash_pos(s.x, g, err);
        if (err) atomicOr(a.err, err);
        a.key[f] = err ? -1 : key;
    }
    if (f == 0) *a.lhcount = 0;
    cluster_barrier();
    const int block = (int)cluster.block_rank(), T = blockDim.x;
    const int share = (a.order.ncell + kRunBlocks - 1) / kRunBlocks;
    const bool ok = block_order(a.order, a.canon[q], min(a.n, block * T),
                                min(a.n, (block + 1) * T), min(a.order.ncell, block * share),
                                min(a.order.ncell, (block + 1) * share), smem);
    cluster_barrier();
    if (!ok) return false;   // the same in every block
    uint32_t err = 0;
    if (active) {
        load_state(a, t, a.perm[f], s);
        tag = a.tag[1][f];
        m = a.inv_mass[1][f];
        list_build_one<false>(g, a.cv, a.lb, a.lb.pre_r2, f, err);
    }
    if (err) atomicOr(a.err, err);
    cluster_barrier();   // every slot's state is read
    if (active) {
        a.tag[0][f] = tag;
        a.inv_mass[0][f] = m;
        a.radius[0][f] = a.radius[1][f];
    }
    const uint32_t bad = *(volatile const uint32_t*)a.err;
    cluster_barrier();   // all have read it before a step may write it
    return bad == 0;
}

template <class Body>
__global__ void __launch_bounds__(kRunThreads, 1)
run_list_kernel(Body body, DevGeom g, RunArgs a, VgbParams p, NoiseView nz) {
    __shared__ uint32_t flags[3];   // reports of the cluster, by step number mod 3
    extern __shared__ int smem[];   // of a rebuild
    cg::cluster_group cluster = cg::this_cluster();
    const int f = (int)cluster.block_rank() * blockDim.x + threadIdx.x;
    const bool active = f < a.n;
    if (threadIdx.x < 3) flags[threadIdx.x] = 0u;
    const uint32_t failed = *(volatile const uint32_t*)a.err;
    const StepState at = *a.state;
    // every block has read the words before any writes them
    cluster_barrier();
    if (failed) return;   // the same in every block
    RunState s;
    int tag = 0;
    double m = 1.0;
    if (active) {
        load_state(a, at.step, f, s);
        tag = a.tag[0][f];
        m = a.inv_mass[0][f];
    }
    float4 lb = make_float4(0.f, 0.f, 0.f, 0.f);
    int hal = 0;
    if (active) {
        lb = a.lbuild[f];
        hal = a.lhalo[f];
    }
    float xf[6];
    uint32_t nerr = 0;   // an error of the draws in xf
    if (active) load_noise_f(nz, p.seed, a.n, tag, tag, at.step, xf, nerr);
    int done = 0, builds = 0;
    while (done < a.n_steps) {
        const long long t = at.step + done;
        const int q = (int)(t & 1);
        uint32_t err = nerr, report = 0;
        RunState v = s;
        if (active) {
            typename Body::Acc acc;
            float rmin = 3.0e38f;
            PairList pl = a.pl;
            pl.pos = a.lpos[q];
            double F[3];
            list_terms<Body, true, false, 1, false>(body, pl, f, 0, acc, rmin, err);
            body.list_overlap(rmin, (2.0f * pl.radius) * (2.0f * pl.radius), err);
            body.sum(acc, F);
            vgb_normal_fast(p, g.L, g.half, s.x, s.x0, v.mx, F, s.F0, xf, m, v.x, v.x0, err);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                v.F00[k] = s.F0[k];
                v.F0[k] = F[k];
            }
            if (list_record(a.lpos[1 - q], a.linv_unit, a.n, a.ldisp2, f, lb, hal, v.x, g))
                report = kRunMoved;
            if (err) {
                atomicOr(a.err, err);
                report |= kRunError;
            }
        }
        // to every block: flags of this step number; those of the next are free, as
        // every warp has read the ones of two steps ago before the last barrier
        const int slot = done % 3;
        if (threadIdx.x == 0) flags[(slot + 1) % 3] = 0u;
        report = __reduce_or_sync(0xffffffffu, report);
        if (report && (threadIdx.x & 31) < kRunBlocks)
            atomicOr(cluster.map_shared_rank(&flags[slot], threadIdx.x & 31), report);
        cluster_arrive();
        nerr = 0;
        if (active && done + 1 < a.n_steps)
            load_noise_f(nz, p.seed, a.n, tag, tag, t + 1, xf, nerr);
        cluster_wait();
        report = *(volatile uint32_t*)&flags[slot];
        if (report & kRunError) break;   // the state stays that of the failing step
        s = v;
        ++done;
        if (report & kRunMoved) {
            ++builds;
            if (!run_rebuild(a, g, t + 1, f, active, smem, cluster, s, tag, m)) break;
            if (active) {
                lb = a.lbuild[f];
                hal = a.lhalo[f];
                nerr = 0;   // the draws of the particle this slot now holds
                if (done < a.n_steps) load_noise_f(nz, p.seed, a.n, tag, tag, t + 1, xf, nerr);
            }
        }
    }
    if (active) store_state(a, at.step + done, f, s);
    if (f == 0) {
        StepState end = at;
        end.step += done;
        end.vel_counter += done;   // normal steps only: below the velocity step's count
        end.list_builds += builds;
        *a.state = end;
        a.lflag[0] = a.lflag[1] = 0;
        *a.lhcount = 0;
    }
    // no block leaves while another may still write its shared words
    cluster_barrier();
}

template <class Body>
cudaError_t launch(const Body& body, const DevGeom& g, const RunArgs& a, const VgbParams& p,
                   const NoiseView& nz, cudaStream_t st, int* clusters) {
    auto* kernel = run_list_kernel<Body>;
    cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kOrderSmem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kRunBlocks);
    cfg.blockDim = dim3(((a.n + kRunBlocks - 1) / kRunBlocks + 31) / 32 * 32);
    cfg.dynamicSmemBytes = order_smem(a.n, a.order.ncell);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kRunBlocks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (clusters) return cudaOccupancyMaxActiveClusters(clusters, kernel, &cfg);
    return cudaLaunchKernelEx(&cfg, kernel, body, g, a, p, nz);
}

cudaError_t dispatch(const ForceSetup& fs, const DevGeom& g, const RunArgs& a, const VgbParams& p,
                     const NoiseView& nz, cudaStream_t st, int* clusters) {
    return with_pair(fs, [&](auto pair, float rc2f) -> cudaError_t {
        using Body = MixedBody<decltype(pair)>;
        return launch(Body{pair, rc2f}, g, a, p, nz, st, clusters);
    });
}

}  // namespace

bool run_list_fits(const ForceSetup& fs, int n, int ncell) {
    if (n < 1 || n > kRunMaxN || !order_fits(n, ncell)) return false;
    // the device holds a cluster of this kernel's blocks
    int clusters = 0;
    RunArgs a{};
    a.n = n;
    a.order.ncell = ncell;
    if (dispatch(fs, DevGeom{}, a, VgbParams{}, NoiseView{}, nullptr, &clusters) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return clusters > 0;
}

cudaError_t launch_run_list(const ForceSetup& fs, const DevGeom& g, const RunArgs& a,
                            const VgbParams& p, const NoiseView& nz, cudaStream_t st) {
    if (a.n < 1 || a.n > kRunMaxN || a.n_steps < 1) return cudaErrorInvalidValue;
    return dispatch(fs, g, a, p, nz, st, nullptr);
}

}  // namespace psim
