// psim_list_build.cu -- the Verlet pair list's build as a kernel: a system's first list, and
// those of the host arrays' force pass.  (A step's rebuild is psim_rebuild.cu.)
#include <algorithm>

#include "psim_list_build.cuh"

namespace psim {

// A grid of a few blocks per SM striding over the particles.
__global__ void __launch_bounds__(128)
list_build_kernel(DevGeom g, CellView cv, ListBuild lb, uint32_t* errp) {
    if (*errp != 0) return;
    uint32_t err = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.n; i += gridDim.x * blockDim.x) {
        if (lb.rep) {   // a batch: the particle's replica's grid and list radius
            const int r = lb.rep[i];
            list_build_one<true>(lb.geoms[r], cv, lb, lb.pre[r], i, err);
        } else {
            list_build_one<true>(g, cv, lb, lb.pre_r2, i, err);
        }
    }
    if (err) atomicOr(errp, err);
}

cudaError_t launch_list_build(const DevGeom& g, const CellView& cv, const ListBuild& lb,
                              uint32_t* err, cudaStream_t st) {
    if (g.n == 0) return cudaSuccess;
    // 32 blocks per SM of the current device (looked up per call: the
    // attribute query is a cached read in the runtime)
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        sms = 152;
    }
    const int blocks = 32 * sms;
    list_build_kernel<<<std::min(blocks, (g.n + 127) / 128), 128, 0, st>>>(g, cv, lb, err);
    return cudaGetLastError();
}

}  // namespace psim
