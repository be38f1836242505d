// psim_list_build.cuh -- the Verlet pair list's build, per particle (what the list
// holds: psim_force_list.cuh).
#pragma once

#include "psim_kernels.cuh"

namespace psim {

// The pair-list build, a thread per particle i (sorted order of the build
// step, whose list slots are the sorted positions).  It walks the 27
// neighbour cells as 9 rows of x-adjacent cells -- one contiguous run of the
// sorted list per row, plus a one-cell run where the row wraps in x -- and
// appends every candidate within the list radius (rc + skin, widened by the
// FP32 test's rounding margin).  A neighbour cell beyond that radius from
// the particle (by its distance to the cell's faces) is not read: about a
// quarter of the 27 cells on average when cellSize ~ rc + skin.  A pair
// across the box edge refers to the neighbour's halo record for that image.
// When each cell's particles are sorted by x (ListBuild::xsorted), a row's
// run is sorted by x too, and two binary searches cut it to the particles
// within the row's x reach of the home: about 250 candidates per particle
// instead of about 410 at cellSize ~ rc + skin.
// Lists are padded to a multiple of kListFold with the ghost record, a dummy
// out of range of every particle, so the force pass reads whole batches.
// st.global of v at p when w holds; no branch around it
__device__ __forceinline__ void store_if(uint32_t* p, uint32_t v, bool w) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.u32 [%0], %1;\n\t}"
                 :: "l"(p), "r"(v), "r"((uint32_t)w) : "memory");
}

// A home's list is stored in groups of kListFold = 8 entries: group q of the
// home in slot i is 32 contiguous bytes at element (q stride + i) 8, so the
// force pass reads a group with one 32-byte load per thread.  The build
// appends entry n of home i at element o = ((n / 8) stride + i) 8 + n % 8,
// kept as a 32-bit offset (the host keeps (cap + 8) stride below 2^32);
// entries past the cap go to the scratch group cap / 8 and are counted, so
// that the overflow is reported.
__device__ __forceinline__ void list_append(const ListBuild& lb, uint32_t ocap, uint32_t v,
                                            bool in, int& n, uint32_t& o) {
    store_if(lb.list + min(o, ocap), v, in);
    n += in ? 1 : 0;
    // next element: the following word, or the next group's first
    const uint32_t step = (n & (kListFold - 1)) ? 1u : (uint32_t)lb.stride * kListFold - 7u;
    o += in ? step : 0u;
}

// Appends the candidates of one run [a, a + len) of the sorted list within
// the list radius of the home position (hx, hy, hz) (the home particle i
// minus the run's image s L) to i's list, n entries so far.  Candidates are
// read four at a time, up to three past the run (the sorted positions are
// padded by four), and masked.  Only the home row's run (kSelf) can hold i
// itself; a shifted run appends the neighbour's halo record for that image.
template <bool kShifted, bool kSelf, bool kNc>
__device__ __forceinline__ void list_run(const CellView& cv, const ListBuild& lb, float R2, int i,
                                         int a, int len, float hx, float hy, float hz, int sx,
                                         int sy, int sz, int& n, uint32_t& o, uint32_t& err) {
    const uint32_t ocap = ((uint32_t)(lb.cap / kListFold) * (uint32_t)lb.stride + (uint32_t)i) *
                          kListFold;
    const float4* pp = cv.posh + a;
    for (int t0 = 0; t0 < len; t0 += 4, pp += 4) {
        float4 hj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) hj[u] = load_as<kNc>(pp + u);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float ex = hj[u].x - hx, ey = hj[u].y - hy, ez = hj[u].z - hz;
            const float r2 = ex * ex + ey * ey + ez * ez;
            bool in = (t0 + u < len) & (r2 < R2);
            if (kSelf) in &= (a + t0 + u != i);
            if (!kShifted) {
                list_append(lb, ocap, (uint32_t)(a + t0 + u), in, n, o);
            } else if (in) {
                // image number: one bit per flagged axis, set where this run shifts
                const int j = a + t0 + u;
                const int hal = lb.lhalo[j];
                const uint32_t fl = (uint32_t)(hal & 63);
                const int sh[3] = {sx, sy, sz};
                int num = 0, bit = 0;
                bool ok = true;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int fk = halo_axis(fl, k);
                    if (sh[k] != 0) {
                        ok = ok && fk == sh[k];
                        num |= 1 << bit;
                    }
                    if (fk != 0) ++bit;
                }
                if (!ok)   // no record of that image: the margin failed
                    err |= EBIT_LIST;
                else
                    list_append(lb, ocap, (uint32_t)(lb.ghost + 1 + (hal >> 6) + num - 1),
                                true, n, o);
            }
        }
    }
}

template <bool kNc>
__device__ __forceinline__ void list_build_one(const DevGeom& g, const CellView& cv,
                                               const ListBuild& lb, float R2, int i,
                                               uint32_t& err) {
    const float4 hi = cv.posh[i];
    const int c = cv.cellid[i] - g.c0;
    const int cx = c % g.s, cy = (c / g.s) % g.s, cz = c / g.s2;
    const int ghost = lb.ghost;
    // distances to the lower and upper faces of the home cell, less a margin
    // for the FP32 rounding of the position and of the cell bounds
    const float csf = (float)g.cs;
    const float m = 8.0f * ulp_of(g.Lhi);
    const float fx = hi.x - (float)cx * csf, fy = hi.y - (float)cy * csf,
                fz = hi.z - (float)cz * csf;
    const float lo[3] = {fmaxf(fx - m, 0.f), fmaxf(fy - m, 0.f), fmaxf(fz - m, 0.f)};
    const float up[3] = {fmaxf(csf - fx - m, 0.f), fmaxf(csf - fy - m, 0.f),
                         fmaxf(csf - fz - m, 0.f)};
    int n = 0;
    uint32_t o = (uint32_t)i * kListFold;
    for (int row = 0; row < 9; ++row) {
        const int dz = row / 3 - 1, dy = row % 3 - 1;
        const float ey = dy < 0 ? lo[1] : (dy > 0 ? up[1] : 0.f);
        const float ez = dz < 0 ? lo[2] : (dz > 0 ? up[2] : 0.f);
        const float e2 = ey * ey + ez * ez;
        if (e2 >= R2) continue;
        int sy, sz;
        const int y = wrap_cell(cy + dy, g.s, sy);
        const int z = wrap_cell(cz + dz, g.s, sz);
        const int base = g.c0 + g.s * y + g.s2 * z;
        const bool left = e2 + lo[0] * lo[0] < R2, right = e2 + up[0] * up[0] < R2;
#pragma unroll 1
        for (int part = 0; part < 2; ++part) {
            // part 0: the reachable cells of [cx-1, cx+1] inside the grid;
            // part 1: the one cell that wraps around in x (if reachable)
            int a = 0, len = 0, sx = 0;
            if (part == 0) {
                const int xa = (left && cx > 0) ? cx - 1 : cx;
                const int xb = (right && cx < g.s - 1) ? cx + 1 : cx;
                a = cv.cstart[base + xa];
                len = cv.cstart[base + xb] + cv.ccount[base + xb] - a;
            } else if ((cx == 0 && left) || (cx == g.s - 1 && right)) {
                const int xw = cx == 0 ? g.s - 1 : 0;
                sx = cx == 0 ? -1 : 1;
                a = cv.cstart[base + xw];
                len = cv.ccount[base + xw];
            }
            if (len <= 0) continue;
            // the row's image is applied to the home position
            const float hx = hi.x - (float)sx * g.Lhi;
            const float hy = hi.y - (float)sy * g.Lhi;
            const float hz = hi.z - (float)sz * g.Lhi;
            if (lb.xsorted) {
                // the run is sorted by x: keep the candidates within the
                // row's x reach sqrt(R^2 - e^2) of the home, found by two
                // binary searches.  e^2 is a lower bound of a candidate's
                // y-z distance^2 (the face distances carry the margin m); the
                // reach is widened by 1e-5 R^2 under the root, far above the
                // FP32 rounding of the r^2 test, and by m outside it.
                const float rx = sqrtf(fmaxf(R2 - e2, 0.f) + 1e-5f * R2) + m;
                const float xlo = hx - rx, xhi = hx + rx;
                // the two searches run interleaved (independent load chains)
                const float4* pp = cv.posh + a;
                int l0 = 0, h0 = len, l1 = 0, h1 = len;
                while (l0 < h0 || l1 < h1) {
                    const int m0 = (l0 + h0) >> 1, m1 = (l1 + h1) >> 1;
                    const float x0 = l0 < h0 ? load_as<kNc>(&pp[m0].x) : 0.f;
                    const float x1 = l1 < h1 ? load_as<kNc>(&pp[m1].x) : 0.f;
                    if (l0 < h0) {
                        if (x0 < xlo) l0 = m0 + 1;
                        else h0 = m0;
                    }
                    if (l1 < h1) {
                        if (x1 <= xhi) l1 = m1 + 1;
                        else h1 = m1;
                    }
                }
                a += l0;
                len = l1 - l0;
                if (len <= 0) continue;
            }
            if ((sx | sy | sz) != 0)
                list_run<true, false, kNc>(cv, lb, R2, i, a, len, hx, hy, hz, sx, sy, sz, n, o, err);
            else if (row == 4 && part == 0)
                list_run<false, true, kNc>(cv, lb, R2, i, a, len, hx, hy, hz, 0, 0, 0, n, o, err);
            else
                list_run<false, false, kNc>(cv, lb, R2, i, a, len, hx, hy, hz, 0, 0, 0, n, o, err);
        }
    }
    // the open group padded with the ghost record
    const uint32_t ocap = ((uint32_t)(lb.cap / kListFold) * (uint32_t)lb.stride + (uint32_t)i) *
                          kListFold;
    while (n & (kListFold - 1)) list_append(lb, ocap, (uint32_t)ghost, true, n, o);
    if (n > lb.cap) {
        err |= EBIT_LIST;
        n = lb.cap;
    }
    lb.count[i] = n;
}

}  // namespace psim
