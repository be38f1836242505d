// psim_rebuild.cu -- the end of a step with a pair list: the step state, and the
// rebuild of cell order and list on the steps that need one, as one kernel.
//
// Most steps rebuild nothing: a conditional graph node around the rebuild's kernels
// costs 7.4 us even when its body does not run, and this kernel's blocks, which read
// the flag and leave, 1.7.  A rebuild is the phases of the counting sort, the state's
// permutation and the list build with a barrier of the whole grid between two; the
// launch is cooperative, so all blocks run at once.  Its results are those of the
// separate kernels, bit for bit.
//
// What other blocks wrote in this kernel is read with plain loads, never through the
// read-only path.
//
// us a step with the conditional node and now: AO colloids 20001 / 65537 / 131072
// particles 17.1 / 19.5 / 24.1 -> 10.1 / 12.7 / 17.4, the LJ liquid of 48668 / 256000 /
// 2^20 30.7 / 77.8 / 222.8 -> 25.5 / 73.9 / 221.5, 8 / 64 AO replicas 23.8 / 80.2 -> 17.3 /
// 73.0, 50001 particles through a plugin 34.3 -> 27.5.  A rebuild of the liquid of 2^20
// takes ~0.87 ms: the list 0.58, the canonical order 0.14, the state there and back 0.12.
// The list is taken warp by warp from a counter (with equal shares 0.78 ms); blocks of 256
// rather than 128 halve the barrier's arrivals.
#include <algorithm>

#include "psim_cells.cuh"
#include "psim_list_build.cuh"
#include "psim_vgb.cuh"

namespace psim {

namespace {

constexpr int kRebuildThreads = 256;
constexpr int kRebuildWarps = kRebuildThreads / 32;
// polls of a barrier before it gives up (seconds; all blocks run at once, so a barrier
// completes within the slowest block's phase)
constexpr int kBarrierPolls = 1 << 26;

// All threads of the grid.  counter: arrivals of all barriers so far, a multiple of
// the grid's blocks between two.  False where it gave up, with the error latched.
__device__ __forceinline__ bool grid_barrier(unsigned long long* counter, uint32_t* err) {
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
        const unsigned long long blocks = gridDim.x;
        __threadfence();
        const unsigned long long target = (atomicAdd(counter, 1ull) / blocks + 1) * blocks;
        unsigned long long seen;
        int polls = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(counter)
                         : "memory");
        } while (seen < target && ++polls < kBarrierPolls);
        if (seen < target) {
            atomicOr(err, EBIT_WAIT);
            ok = 0;
        }
        __threadfence();
    }
    return __syncthreads_and(threadIdx.x != 0 || ok) != 0;
}

// start[c] = the counts of the cells before c; a grid barrier in the middle
__device__ __forceinline__ bool grid_scan(const RebuildArgs& a, int* warp) {
    const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int blocks = gridDim.x, b = blockIdx.x;
    const int share = (a.ncell + blocks - 1) / blocks, per = (share + T - 1) / T;
    const long long c0 = (long long)b * share;
    const int c1 = (int)min((long long)a.ncell, c0 + share);
    const int b0 = (int)min((long long)c1, c0 + (long long)tid * per), b1 = min(c1, b0 + per);
    int sum = 0;
    for (int c = b0; c < b1; ++c) sum += a.count[c];
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp[w] = x;
    __syncthreads();
    int run = x - sum, total = 0;
#pragma unroll
    for (int k = 0; k < kRebuildWarps; ++k) {
        if (k < w) run += warp[k];
        total += warp[k];
    }
    if (tid == 0) a.sums[b] = total;
    if (!grid_barrier(a.counter, a.err)) return false;
    int before = 0;
    for (int k = tid; k < b; k += T) before += a.sums[k];
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) warp[w] = before;   // the totals above are read: a barrier lies between
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRebuildWarps; ++k) run += warp[k];
    for (int c = b0; c < b1; ++c) {
        a.start[c] = run;
        run += a.count[c];
    }
    return true;
}

__global__ void __launch_bounds__(kRebuildThreads, 4) step_rebuild_kernel(RebuildArgs a, DevGeom g) {
    __shared__ int warp[kRebuildWarps];
    const bool failed = *(volatile const uint32_t*)a.err != 0;
    const bool rebuild = !failed && *a.lflag != 0;
    const int f = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
    if (f == 0 && !failed) {
        step_advance(a.state, a.vel_freq, rebuild);
    }
    if (!rebuild) return;   // the same in every block: neither word is written before the barrier
    for (int c = f; c < a.ncell; c += threads) a.count[c] = 0;
    if (f == 0) *a.next = 0;
    if (!grid_barrier(a.counter, a.err)) return;
    uint32_t err = 0;
    for (int i = f; i < a.n; i += threads) {
        const double x[3] = {a.canon.x[i], a.canon.y[i], a.canon.z[i]};
        const int key = hash_pos(x, a.lb.rep ? a.lb.geoms[a.lb.rep[i]] : g, err);
        a.key[i] = key;
        a.rank[i] = atomicAdd(&a.count[key], 1);
    }
    if (err) atomicOr(a.err, err);
    if (!grid_barrier(a.counter, a.err)) return;
    if (*(volatile const uint32_t*)a.err) return;   // the order stays as it was
    if (!grid_scan(a, warp)) return;
    if (!grid_barrier(a.counter, a.err)) return;
    for (int i = f; i < a.n; i += threads) a.tmp[a.start[a.key[i]] + a.rank[i]] = i;
    if (!grid_barrier(a.counter, a.err)) return;
    for (int i = f; i < a.n; i += threads) canon_slot(a.canon, i);
    if (!grid_barrier(a.counter, a.err)) return;
    // the list, warp by warp as each is done: a warp across the end of an x-row of cells
    // takes three times the mean
    err = 0;
    for (;;) {
        int i = 0;
        if ((threadIdx.x & 31) == 0) i = atomicAdd(a.next, 32);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= a.n) break;   // every lane
        i += threadIdx.x & 31;
        if (i < a.n) {
            if (a.lb.rep) {   // a batch: the particle's replica's grid and list radius
                const int r = a.lb.rep[i];
                list_build_one<false>(a.lb.geoms[r], a.cv, a.lb, a.lb.pre[r], i, err);
            } else {
                list_build_one<false>(g, a.cv, a.lb, a.lb.pre_r2, i, err);
            }
        }
        __syncwarp();
    }
    // the state into the new order, through the scratch arrays
    for (int i = f; i < a.n; i += threads) {
        const int o = a.canon.perm[i];
#pragma unroll
        for (int k = 0; k < 15; ++k)
            a.scratch[(size_t)k * a.n + i] = a.arr[k / 3][(size_t)(k % 3) * a.n + o];
    }
    if (err) atomicOr(a.err, err);
    if (!grid_barrier(a.counter, a.err)) return;
    for (int i = f; i < a.n; i += threads) {
#pragma unroll
        for (int k = 0; k < 15; ++k)
            a.arr[k / 3][(size_t)(k % 3) * a.n + i] = a.scratch[(size_t)k * a.n + i];
        a.tag[0][i] = a.tag[1][i];
        a.radius[0][i] = a.radius[1][i];
        a.inv_mass[0][i] = a.inv_mass[1][i];
    }
}

}  // namespace

int rebuild_sums() { return 8192; }

cudaError_t launch_step_rebuild(const RebuildArgs& a, const DevGeom& g, cudaStream_t st) {
    int dev = 0, sms = 0, per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, step_rebuild_kernel,
                                                          kRebuildThreads, 0);
    if (e != cudaSuccess) return e;
    // one block at least: an empty system's steps count too
    const int blocks = std::max(1, std::min({sms * per, rebuild_sums(),
                                             (a.n + kRebuildThreads - 1) / kRebuildThreads}));
    RebuildArgs args = a;
    DevGeom geom = g;
    void* params[] = {&args, &geom};
    return cudaLaunchCooperativeKernel((const void*)step_rebuild_kernel, dim3(blocks),
                                       dim3(kRebuildThreads), params, 0, st);
}

}  // namespace psim
