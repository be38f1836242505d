// psim_cells.cuh -- the canonical order within a cell, and the whole cell order of a
// small system by one block, shared by psim_cells.cu and psim_run.cu.
#pragma once

#include "psim_kernels.cuh"

namespace psim {

// Particle f's place inside its cell c, whose cnt slots from st on hold the particles
// tmp(st) .. (scattered in any order), and there everything the force pass reads.
// (kTags: a.tag_in holds the tags; otherwise a particle's index is its tag.)
template <bool kTags, class Tmp>
__device__ __forceinline__ void canon_place(const CanonArgs& a, int f, int c, int st, int cnt,
                                            Tmp tmp) {
    auto tag = [&](int i) { return kTags ? a.tag_in[i] : i; };
    // Bound by the latency of its gathers: everything of the particle's own is read before
    // the walk over its mates, four of them at a time (the compiler keeps loads behind the
    // stores and the loop).  The gel of 2^21: a step 384 -> 374 us, 4000 AO colloids in
    // FP64 22.3 -> 21.6.
    const int mine = tag(f);
    const double x = a.x[f], y = a.y[f], z = a.z[f], R = a.radius_in[f];
    const double m = a.inv_mass_out ? a.inv_mass_in[f] : 0.0;
    int r = 0;
    if (a.xorder) {
        // by x, then tag: the bit patterns of the (non-negative) positions
        // order like their values, and every pattern is comparable
        const long long mx = __double_as_longlong(x);
#pragma unroll 4
        for (int q = st; q < st + cnt; ++q) {
            const int fq = tmp(q);
            const long long xq = __double_as_longlong(a.x[fq]);
            r += (xq < mx || (xq == mx && tag(fq) < mine)) ? 1 : 0;
        }
    } else {
#pragma unroll 4
        for (int q = st; q < st + cnt; ++q) r += (tag(tmp(q)) < mine) ? 1 : 0;
    }
    const int g = st + r;
    a.perm[g] = f;
    a.tag_out[g] = mine;
    a.cellid[g] = c;
    a.radius_out[g] = R;
    if (a.inv_mass_out) a.inv_mass_out[g] = m;
    if (a.posd) a.posd[g] = make_double4_32a(x, y, z, R);
    float4 h, l;
    split_f64(x, h.x, l.x);
    split_f64(y, h.y, l.y);
    split_f64(z, h.z, l.z);
    h.w = (float)R;
    l.w = __int_as_float(g);  // the slot, which the pair-list build reads
    a.posh[g] = h;
    if (a.posl) a.posl[g] = l;
    if (a.lbuild) a.lbuild[g] = h;
    if (a.lpos) {
        l.w = 0.f;
        store_record(a.lpos, a.linv_unit, (size_t)g, h, l);
        // images of a particle near a face, as halo records (in a
        // batch, of its replica's box)
        float hr = a.hr, Lf = a.Lf, Lhi = a.Lhi, Llo = a.Llo;
        if (a.rep) {
            const int r = a.rep[g];
            hr = a.hr_rep[r];
            Lf = Lhi = a.geoms[r].Lhi;
            Llo = a.geoms[r].Llo;
        }
        uint32_t fl = halo_flags(h, hr, Lf);
        const int m = halo_copies(fl);
        int base = 0;
        if (m > 0) {
            base = atomicAdd(a.lhcount, m);
            if (base + m > a.hcap) {
                atomicOr(a.err, EBIT_LIST);
                fl = 0;
                base = 0;
            } else {
                halo_write(a.lpos + (a.linv_unit != 0.f ? 1 : 2) * ((size_t)a.n + 1),
                           a.linv_unit, base, fl, h, l, Lhi, Llo);
            }
        }
        a.lhalo[g] = (base << 6) | (int)fl;
    }
}

__device__ __forceinline__ void canon_slot(const CanonArgs& a, int p) {
    const int f = a.tmp[p], c = a.key[f];
    canon_place<true>(a, f, c, a.start[c], a.count[c], [&](int q) { return a.tmp[q]; });
}

// The whole order by one block that holds the cells and the particles' keys in shared
// memory.  The blocks of a kernel each count and scatter every particle -- a few
// microseconds of shared-memory work that needs no other block -- and place only their
// own: particles [f0, f1) and, in o.start and o.count, cells [c0, c1).  False, in every
// thread of every block, when a particle has no cell (a negative key): nothing is
// written.
// The block's shared memory: starts of the cells, then key, rank and scattered order.
__host__ __device__ inline size_t order_smem(int n, int ncell) {
    return 4 * (size_t)(ncell + 1 + 32) + 6 * (size_t)n;
}
constexpr int kOrderIndex = 1 << 16;   // keys and particles are 16-bit
__device__ __forceinline__ bool block_order(const OrderArgs& o, const CanonArgs& c,
                                            int f0, int f1, int c0, int c1, int* smem) {
    const int T = blockDim.x, tid = threadIdx.x, n = c.n, ncell = o.ncell;
    int* start = smem;
    int* warp = smem + ncell + 1;
    uint16_t* key = reinterpret_cast<uint16_t*>(warp + 32);
    uint16_t* rank = key + n;
    uint16_t* tmp = rank + n;
    for (int k = tid; k < ncell; k += T) start[k] = 0;
    __syncthreads();
    bool bad = false;
    for (int i0 = tid; i0 < n; i0 += 4 * T) {   // four loads in flight
        int k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) k[u] = o.key[min(i0 + u * T, n - 1)];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * T;
            bad = bad || k[u] < 0;
            if (i >= n || k[u] < 0) continue;
            key[i] = (uint16_t)k[u];
            rank[i] = (uint16_t)atomicAdd(&start[k[u]], 1);
        }
    }
    if (__syncthreads_or(bad)) return false;
    // counts to starts, a run of cells per thread
    const int per = (ncell + T - 1) / T, b0 = min(ncell, tid * per), b1 = min(ncell, b0 + per);
    int sum = 0;
    for (int k = b0; k < b1; ++k) sum += start[k];
    const int lane = tid & 31, w = tid >> 5;
    int x = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) warp[w] = x;
    __syncthreads();
    int run = x - sum;
    for (int k = 0; k < w; ++k) run += warp[k];
    for (int k = b0; k < b1; ++k) {
        const int m = start[k];
        start[k] = run;
        run += m;
    }
    if (tid == 0) start[ncell] = n;
    __syncthreads();
    for (int i = tid; i < n; i += T) tmp[start[key[i]] + rank[i]] = (uint16_t)i;
    for (int k = c0 + tid; k < c1; k += T) {
        o.start[k] = start[k];
        o.count[k] = start[k + 1] - start[k];
    }
    __syncthreads();
    for (int f = f0 + tid; f < f1; f += T) {
        const int k = key[f], st = start[k];
        const int m = start[k + 1] - st;
        auto at = [&](int q) { return (int)tmp[q]; };
        if (c.tag_in) canon_place<true>(c, f, k, st, m, at);
        else canon_place<false>(c, f, k, st, m, at);
    }
    return true;
}

// The end of a step: brownianIntegrator's velCounter bookkeeping
// (brownianIntegrator.cpp:291-292) runs only after normal steps.
__device__ __forceinline__ void step_advance(StepState* state, int vel_freq, bool rebuild) {
    StepState s = *state;
    if (s.step > 0) s.vel_counter = (s.vel_counter == vel_freq) ? 0 : s.vel_counter + 1;
    s.step += 1;
    if (rebuild) s.list_builds += 1;
    *state = s;
}

}  // namespace psim
