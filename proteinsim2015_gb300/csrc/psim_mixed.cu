// psim_mixed.cu -- the mixed-precision form of the plugin force pass.
//
// Pair forces are computed in FP32 and summed in FP32 with Kahan-compensated
// per-particle totals; the update, wrap and coefficients stay FP64 (in
// psim_exact.cu).  Positions are carried as FP32 pairs (hi + lo == the FP64
// position to ~1e-14).  For a row of cells the home position minus the
// row's periodic image (0 or +-L, L itself a float pair) is formed exactly
// as a float pair (h, l) by TwoSum, and a pair separation is
//     d = (x_j,hi - h) + (x_j,lo - l)
// where the first difference is exact for nearby values (Sterbenz), so d
// carries one FP32 rounding of a number of size <= rc, not of the box.
// The pair loops are force_direct_kernel (psim_force.cuh) and force_list_kernel
// (psim_force_list.cuh).
#include <cmath>

#include "psim_body.cuh"
#include "psim_force.cuh"
#include "psim_force_cell.cuh"
#include "psim_force_list.cuh"
#include "psim_vgb.cuh"

namespace psim {

cudaError_t launch_forces_mixed(const ForceSetup& fs, const DevGeom& g, const CellView& cv,
                                const ForceOut& out, cudaStream_t st, const BatchView* bv) {
    if (bv && fs.kind == 4) return cudaErrorInvalidValue;  // batches hold single-plugin replicas
    return with_pair(fs, [&](auto p, float rc2f) {
        MixedBody<decltype(p)> body{p, rc2f};
        body.cont2f = out.coor ? out.cont2f : 0.f;   // updateInteractions fused into the pass
        if (fs.tile && !bv) return launch_force_cells(body, g, cv, out, fs.pre_rc2f, st);
        return launch_force_pass(body, g, cv, out, fs.pre_rc2f, st, bv, fs.walk);
    });
}

cudaError_t launch_forces_list(const ForceSetup& fs, const DevGeom& g, const PairList& pl,
                               const ForceOut& out, cudaStream_t st) {
    return with_pair(fs, [&](auto p, float rc2f) {
        MixedBody<decltype(p)> body{p, rc2f};
        body.cont2f = out.coor ? out.cont2f : 0.f;
        return launch_force_list(body, g, pl, out, st);
    });
}

// The update of the mixed form: the same FP64 arithmetic as psim_exact.cu's
// instance, with a*b+c contracted into FMA by this translation unit.
cudaError_t launch_vgb_system_fast(const VgbSystemArgs& a, const VgbParams& p, const DevGeom& g,
                                   const NoiseView& nz, cudaStream_t st) {
    return launch_vgb_system_t<VgbFast>(a, p, g, nz, st);
}

}  // namespace psim
