// psim_force_list.cuh -- the mixed form's force pass through a Verlet pair list.
//
// The plugin force on particle i is the sum over the particles j of its 27
// neighbour cells with |x_j - x_i| < rc (AOPotential.cpp:61-175,
// LJPotential.cpp:64-182).  Every such j lies within rc + skin of i's position
// at any earlier time at which neither particle had yet moved skin/2 -- so a
// list of the pairs within rc + skin, built from the cell list at one step,
// holds every pair the cell walk would find for as long as no particle has
// moved more than skin/2 since.  The list is rebuilt on the step after one
// has.  The force of each step is then the same set of pair terms, read from
// ~(rc+skin)^3/(27 cs^3) as many candidates as the cell walk tests.
//
//   build  (psim_list_build.cuh) a thread per particle appends the candidates of
//          its 27 cells within rc + skin (plus the rounding margin of the FP32
//          test).  It runs on the cell order made with it, so list order is the
//          cell order of the build step, and it needs cellSize >= rc + skin.  A pair across the box edge refers to a
//          halo record: a copy of the neighbour shifted by the box, made for
//          every particle within rc + skin of a face and rewritten with it
//          each step, so the force pass does no periodic arithmetic.
//   force  a thread per particle walks its list in FP32 with the plugin's pair
//          body and Kahan-compensated sums (MixedBody, psim_mixed.cu).
//
// Positions in list order are kept as exact float pairs and *unwrapped*: the
// integrator writes each particle's new position as the image nearest its
// build position (and its halo images beside it), so a pair's periodic image
// found at the build stays right for the life of the list (the box is larger
// than 2 (rc + skin)).
#pragma once

#include "psim_force.cuh"

namespace psim {

// One 32-byte record (high and low float4 halves) in a single 256-bit load
// through the read-only path; the records are 32-byte aligned.
__device__ __forceinline__ void load_record(const float4* pos, uint32_t j, float4& h, float4& l) {
    const float4* a = pos + 2 * (size_t)j;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(h.x), "=f"(h.y), "=f"(h.z), "=f"(h.w), "=f"(l.x), "=f"(l.y), "=f"(l.z), "=f"(l.w)
        : "l"(a));
}

// One group of kListFold = 8 list entries (32 bytes, 32-byte aligned) in a
// single 256-bit load through the read-only path: a warp's request covers
// its 1 KB once, where two 128-bit loads would each cover all of it.
template <bool kNc>
__device__ __forceinline__ void load_group(const uint32_t* p, uint4& a, uint4& b) {
    if constexpr (!kNc) {
        a = reinterpret_cast<const uint4*>(p)[0];
        b = reinterpret_cast<const uint4*>(p)[1];
        return;
    }
    asm("ld.global.nc.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
        : "l"(p));
}

// A neighbour record as the force pass holds it between its load and its
// pair term: one float4 (compact) or the high and low halves (full).
template <bool kCompact>
struct ListRec {
    float4 h;
};
template <>
struct ListRec<false> {
    float4 h, l;
};
template <bool kNc>
__device__ __forceinline__ ListRec<true> load_rec(const float4* pos, uint32_t j,
                                                  ListRec<true>) {
    return ListRec<true>{load_as<kNc>(pos + j)};
}
template <bool kNc>
__device__ __forceinline__ ListRec<false> load_rec(const float4* pos, uint32_t j,
                                                   ListRec<false>) {
    ListRec<false> r;
    load_record(pos, j, r.h, r.l);
    return r;
}

// A thread per particle (current storage order f) -- or kLanes threads, lane
// l taking entries [l E, (l + 1) E) of every group of 8 (E = 8 / kLanes) --
// its list slot, its list, its neighbours' records; the force is stored at f.
// With several lanes a warp covers 32 / kLanes particles, mostly of one cell,
// whose entries at the same place of their lists lie close together in the
// same rows of cells: fewer L1 wavefronts per record gather, and the lanes of
// a particle do equal work.  A lane walks its entries in views of 8 (kLanes
// groups' parts; a group past the list's end reads as the ghost record), in
// batches of 4 (lists are padded to multiples of 8, kListFold).  Each
// batch's records are loaded one batch ahead of its pair terms, and its list
// entries -- streamed from DRAM -- one batch ahead of the records, so the
// latency of both overlaps the terms of the batch before.  Every record holds
// the image the pair needs: no periodic arithmetic per pair.  A separation
// is, for compact records, the exact integer difference of the fixed-point
// coordinates, converted and scaled by a power of two (fixed_sep); for full
// records d = (x_j,hi - x_i,hi) + (x_j,lo - x_i,lo), the first difference
// exact for nearby values.  Either way d carries one FP32 rounding.  The
// lanes of a particle are adjacent in one warp; lane 0 adds the others' sums
// in lane order, so the result does not depend on scheduling.
// kNc: no one writes the list or the records while the kernel runs.
template <class Body, bool kCompact, bool kCount, int kLanes, bool kNc = true>
__device__ __forceinline__ void list_terms(const Body& body, const PairList& pl, int s, int lane,
                                           typename Body::Acc& acc, float& rmin, uint32_t& err) {
    constexpr int kBatch = 4;
    static_assert(kListFold == 2 * kBatch, "a fold is two batches");
    static_assert(kLanes == 1 || kLanes == 2 || kLanes == 4, "1, 2 or 4 lanes per particle");
    float4 hh, hl;
    // compact records: the home's fixed-point coordinates
    uint32_t ux = 0u, uy = 0u, uz = 0u;
    const float unit = pl.unit;
    if (kCompact) {
        const float4 c = pl.pos[s];
        ux = __float_as_uint(c.x);
        uy = __float_as_uint(c.y);
        uz = __float_as_uint(c.z);
        hh = make_float4(0.f, 0.f, 0.f, pl.radius);
        hl = hh;
    } else {
        hh = pl.pos[2 * (size_t)s];
        hl = pl.pos[2 * (size_t)s + 1];
    }
    const float usize = 2.0f * pl.radius, us2 = usize * usize;
    body.init(acc);
    // this lane's views of 8 entries: its parts of kLanes groups each
    const int groups = pl.count[s] / kListFold;
    const int views = (groups + kLanes - 1) / kLanes;
    using Rec = ListRec<kCompact>;
    const Rec none{};
    auto terms = [&](const Rec* r) {
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            if constexpr (kCompact) {
                const float d0 = fixed_sep(r[u].h.x, ux, unit);
                const float d1 = fixed_sep(r[u].h.y, uy, unit);
                const float d2 = fixed_sep(r[u].h.z, uz, unit);
                body.template eval_list<true, kCount>(d0, d1, d2, usize, us2, acc, rmin, err,
                                                      r[u].h.w);
            } else {
                const float d0 = (r[u].h.x - hh.x) + (r[u].l.x - hl.x);
                const float d1 = (r[u].h.y - hh.y) + (r[u].l.y - hl.y);
                const float d2 = (r[u].h.z - hh.z) + (r[u].l.z - hl.z);
                const float size = hh.w + r[u].h.w;
                body.template eval_list<false, kCount>(d0, d1, d2, size, size * size, acc, rmin,
                                                       err);
            }
        }
    };
    // groups of 8 entries (one 32-byte load) one group ahead; records one
    // batch of 4 ahead of their pair terms
    constexpr int kE = kListFold / kLanes;   // entries of each group this lane takes
    const uint32_t* gp = pl.list + (size_t)s * kListFold + lane * kE;
    const size_t gs = (size_t)pl.stride * kListFold;   // one group
    const uint32_t gh = (uint32_t)pl.stride;           // the ghost record (slot n)
    // view m of this lane: its parts of groups kLanes m ... kLanes m + kLanes - 1
    // (gp at the first; group kLanes m exists)
    auto load_view = [&](const uint32_t* p, int m, uint4& a, uint4& b) {
        if constexpr (kLanes == 1) {
            load_group<kNc>(p, a, b);
        } else if constexpr (kLanes == 2) {
            a = __ldg(reinterpret_cast<const uint4*>(p));
            b = 2 * m + 1 < groups ? __ldg(reinterpret_cast<const uint4*>(p + gs))
                                   : make_uint4(gh, gh, gh, gh);
        } else {
            const uint2 gg = make_uint2(gh, gh);
            const uint2 q0 = __ldg(reinterpret_cast<const uint2*>(p));
            const uint2 q1 = 4 * m + 1 < groups ? __ldg(reinterpret_cast<const uint2*>(p + gs)) : gg;
            const uint2 q2 =
                4 * m + 2 < groups ? __ldg(reinterpret_cast<const uint2*>(p + 2 * gs)) : gg;
            const uint2 q3 =
                4 * m + 3 < groups ? __ldg(reinterpret_cast<const uint2*>(p + 3 * gs)) : gg;
            a = make_uint4(q0.x, q0.y, q1.x, q1.y);
            b = make_uint4(q2.x, q2.y, q3.x, q3.y);
        }
    };
    // past the list's end the entries read as slot 0, a valid record: the
    // record loads need no condition
    uint4 ea = make_uint4(0u, 0u, 0u, 0u), eb = ea;
    Rec r[kBatch], rn[kBatch];
    if (views > 0) load_view(gp, 0, ea, eb);
    r[0] = load_rec<kNc>(pl.pos, ea.x, none);
    r[1] = load_rec<kNc>(pl.pos, ea.y, none);
    r[2] = load_rec<kNc>(pl.pos, ea.z, none);
    r[3] = load_rec<kNc>(pl.pos, ea.w, none);
    for (int m = 0; m < views; ++m) {
        const bool more = m + 1 < views;
        gp += gs * kLanes;
        uint4 na = make_uint4(0u, 0u, 0u, 0u), nb = na;
        if (more) load_view(gp, m + 1, na, nb);
        rn[0] = load_rec<kNc>(pl.pos, eb.x, none);
        rn[1] = load_rec<kNc>(pl.pos, eb.y, none);
        rn[2] = load_rec<kNc>(pl.pos, eb.z, none);
        rn[3] = load_rec<kNc>(pl.pos, eb.w, none);
        terms(r);
        r[0] = load_rec<kNc>(pl.pos, na.x, none);
        r[1] = load_rec<kNc>(pl.pos, na.y, none);
        r[2] = load_rec<kNc>(pl.pos, na.z, none);
        r[3] = load_rec<kNc>(pl.pos, na.w, none);
        terms(rn);
        body.fold(acc);
        eb = nb;
    }
}

template <class Body, bool kCompact, bool kReplicas, bool kCount = false, int kLanes = 1>
__global__ void __launch_bounds__(256)
force_list_kernel(Body body0, DevGeom g, PairList pl, ForceOut out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int f = t / kLanes;
    const int lane = t % kLanes;
    if (kLanes == 1) {
        if (f >= g.n || *out.err) return;
    } else {
        // every lane of a particle must take the same path: the error word
        // is read once per warp (all 32 threads are present here)
        const bool failed =
            __shfl_sync(0xffffffffu, (threadIdx.x & 31) == 0 ? (*out.err != 0) : false, 0);
        if (failed || f >= g.n) return;   // f is the same for all lanes of a particle
    }
    // a batch: the pair functor of the particle's replica (its neighbours are
    // all of the same replica)
    const Body body = kReplicas ? body0.for_replica(pl.pairs, pl.rep[f], g) : body0;
    typename Body::Acc acc;
    uint32_t err = 0;
    float rmin = 3.0e38f;
    list_terms<Body, kCompact, kCount, kLanes>(body, pl, f, lane, acc, rmin, err);
    const float us2 = (2.0f * pl.radius) * (2.0f * pl.radius);
    if constexpr (kLanes > 1) {
        // lane 0 adds the other lanes' sums in lane order
        const unsigned seg = (threadIdx.x & 31) & ~(unsigned)(kLanes - 1);
        const unsigned mask = ((1u << kLanes) - 1u) << seg;
        const typename Body::Acc own = acc;
#pragma unroll
        for (int o = 1; o < kLanes; ++o) body.merge_lane(acc, own, mask, o, kLanes);
#pragma unroll
        for (int o = kLanes / 2; o > 0; o >>= 1) {
            rmin = fminf(rmin, __shfl_xor_sync(mask, rmin, o, kLanes));
            err |= __shfl_xor_sync(mask, err, o, kLanes);
        }
        if (lane != 0) return;
    }
    if (kCompact) body.list_overlap(rmin, us2, err);
    body.store(out, f, acc);
    if (err) atomicOr(out.err, err);
}

// The list pass with `lanes` threads per particle (kMulti: the 2- and 4-lane
// kernels are built for this variant; otherwise one lane).
template <class Body, bool kCompact, bool kReplicas, bool kCount, bool kMulti>
cudaError_t launch_list_lanes(const Body& body, const DevGeom& g, const PairList& pl,
                              const ForceOut& out, int lanes, cudaStream_t st) {
    const long long items = (long long)g.n * lanes;
    const int threads = block_threads(items), blocks = (int)((items + threads - 1) / threads);
    if constexpr (kMulti) {
        if (lanes == 2 || lanes == 4) {
            if (lanes == 4)
                force_list_kernel<Body, kCompact, kReplicas, kCount, 4>
                    <<<blocks, threads, 0, st>>>(body, g, pl, out);
            else
                force_list_kernel<Body, kCompact, kReplicas, kCount, 2>
                    <<<blocks, threads, 0, st>>>(body, g, pl, out);
            return cudaGetLastError();
        }
    }
    force_list_kernel<Body, kCompact, kReplicas, kCount, 1><<<blocks, threads, 0, st>>>(body, g, pl,
                                                                                    out);
    return cudaGetLastError();
}

template <class Body>
cudaError_t launch_force_list(const Body& body, const DevGeom& g, const PairList& pl,
                              const ForceOut& out, cudaStream_t st) {
    if (g.n == 0) return cudaSuccess;
    // several lanes per particle for compact records without the count; one
    // lane otherwise
    const int lanes = (pl.compact && !out.coor && (pl.lanes == 2 || pl.lanes == 4)) ? pl.lanes : 1;
    if (pl.rep) {
        if constexpr (Body::kBatchable) {
            if (pl.compact)
                return launch_list_lanes<Body, true, true, false, true>(body, g, pl, out, lanes, st);
            return launch_list_lanes<Body, false, true, false, false>(body, g, pl, out, 1, st);
        }
        return cudaErrorInvalidValue;
    }
    if (out.coor) {   // the coordination numbers with the forces (one system)
        if (pl.compact)
            return launch_list_lanes<Body, true, false, true, false>(body, g, pl, out, 1, st);
        return launch_list_lanes<Body, false, false, true, false>(body, g, pl, out, 1, st);
    }
    if (pl.compact)
        return launch_list_lanes<Body, true, false, false, true>(body, g, pl, out, lanes, st);
    return launch_list_lanes<Body, false, false, false, false>(body, g, pl, out, 1, st);
}

}  // namespace psim
