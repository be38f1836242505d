// psim_cells.cuh -- the canonical order of one slot of the counting sort, shared by
// canonicalize_kernel and the kernel that runs small systems (psim_run.cu).
#pragma once

#include "psim_kernels.cuh"

namespace psim {

// Slot p of the scattered order: its particle's place inside its cell, and there
// everything the force pass reads.
__device__ __forceinline__ void canon_slot(const CanonArgs& a, int p) {
    const int f = a.tmp[p];
    const int c = a.key[f];
    const int st = a.start[c];
    const int cnt = a.count[c];
    const int mine = a.tag_in[f];
    int r = 0;
    if (a.xorder) {
        // by x, then tag: the bit patterns of the (non-negative) positions
        // order like their values, and every pattern is comparable
        const long long mx = __double_as_longlong(a.x[f]);
        for (int q = st; q < st + cnt; ++q) {
            const int fq = a.tmp[q];
            const long long xq = __double_as_longlong(a.x[fq]);
            r += (xq < mx || (xq == mx && a.tag_in[fq] < mine)) ? 1 : 0;
        }
    } else {
        for (int q = st; q < st + cnt; ++q) r += (a.tag_in[a.tmp[q]] < mine) ? 1 : 0;
    }
    const int g = st + r;
    a.perm[g] = f;
    a.tag_out[g] = mine;
    a.cellid[g] = c;
    const double R = a.radius_in[f];
    a.radius_out[g] = R;
    if (a.inv_mass_out) a.inv_mass_out[g] = a.inv_mass_in[f];
    // with a pair list, the sorted positions are written only when the
    // list is rebuilt on this order (they are the list's positions)
    const bool pos_out = !a.rebuild || *a.rebuild != 0;
    if (a.lslot_out) a.lslot_out[g] = (pos_out || !a.lslot_in) ? g : a.lslot_in[f];
    if (pos_out) {
        const double x = a.x[f], y = a.y[f], z = a.z[f];
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
}

}  // namespace psim
