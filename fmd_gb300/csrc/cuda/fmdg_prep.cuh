// Per-atom tables formed from the current positions: what the list, density
// and force kernels read.  Written by the refresh kernels (fmdg_bin.cu) for
// every atom as it takes its place, or on their own for a force evaluation
// without a refresh.
#pragma once

#include "fmdg_internal.cuh"

namespace {

// Slot t's binary32 position relative to the cell it had at the last build
// (unwrapped across periodic faces) and the displacement test against its
// build position: sets the rebuild flag beyond skin/2.
__device__ __forceinline__ void slot_rel_build(const Geo &g, Dyn *dyn, int t, const double (&x)[3], float kb)
{
    const double4_32a ob = g.corig[g.cb[t]];
    const double o3[3] = {ob.x, ob.y, ob.z};
    float l3[3];
    double u3[3];
    // (the scale is 1 in binary64 mode, the remainders below are of unscaled values)
    const bool fp64 = g.prec == FMDG_PREC_FP64;
    const double xs = g.xs;
    auto scaled = [&](double u) { return fp64 ? u : u * xs; };
    for (int d = 0; d < 3; d++)
    {
        double u = x[d] - o3[d];
        float uf = d2f_rn(scaled(u));
        // unwrap across a periodic face (binary64 test near half a box)
        if (g.pbc[d] && fabsf(uf) > 0.49f * g.l_f[d])
        {
            if (u > 0.5 * g.l[d]) u -= g.l[d];
            else if (u < -0.5 * g.l[d]) u += g.l[d];
            uf = d2f_rn(scaled(u));
        }
        l3[d] = uf;
        u3[d] = u;
    }
    g.xl[t] = make_float4(l3[0], l3[1], l3[2], kb);
    if (fp64)
    {
        g.xr[2 * (size_t)t] = make_float4(l3[0], l3[1], l3[2], kb);
        g.xr[2 * (size_t)t + 1] =
            make_float4(d2f_rn(u3[0] - f2d(l3[0])), d2f_rn(u3[1] - f2d(l3[1])), d2f_rn(u3[2] - f2d(l3[2])), 0.f);
    }
    const float4 o = g.xb[t];
    const float dx = l3[0] - o.x, dy = l3[1] - o.y, dz = l3[2] - o.z;
    if (!(dx * dx + dy * dy + dz * dz <= g.half_skin2)) dyn->rebuild = 1;
}

// Skin-list tables of the atom at index i, slot t, in cell c.  relative: no
// rebuild is due, so the slot's position relative to its build cell and the
// displacement test too (else the list build that follows writes them).
__device__ __forceinline__ void prep_skin_atom(const Geo &g, Dyn *dyn, int i, int t, int c, int kind, int group,
                                               const double (&x)[3], bool relative)
{
    const float kb = __int_as_float(kind);
    g.pos[t] = i;
    g.xd[t] = make_double4_32a(x[0], x[1], x[2], 0.0);
    g.gslot[t] = group;
    // relative to the current cell (a rebuild starts from these)
    const double4_32a oc = g.corig[c];
    const double ux = x[0] - oc.x, uy = x[1] - oc.y, uz = x[2] - oc.z;
    const bool fp64 = g.prec == FMDG_PREC_FP64;      // (scale 1)
    const double xs = g.xs;
    const float lx = d2f_rn(fp64 ? ux : ux * xs), ly = d2f_rn(fp64 ? uy : uy * xs), lz = d2f_rn(fp64 ? uz : uz * xs);
    g.xf4[i] = make_float4(lx, ly, lz, kb);
    if (relative) slot_rel_build(g, dyn, t, x, kb);
}

// Tables of the exact per-step list: binary32 cell-local coordinates, with
// the remainders beside them in binary64 mode (the double-float cell-local
// position in one 32-byte row)
__device__ __forceinline__ void prep_local_atom(const Geo &g, int i, int c, int kind, const double (&x)[3])
{
    const double4_32a oc = g.corig[c];
    const double ux = x[0] - oc.x, uy = x[1] - oc.y, uz = x[2] - oc.z;
    const float lx = (float)ux, ly = (float)uy, lz = (float)uz;
    const float4 hi = make_float4(lx, ly, lz, __int_as_float(kind));
    g.xf4[i] = hi;
    if (g.prec == FMDG_PREC_FP64)
    {
        g.xdf[2 * (size_t)i] = hi;
        g.xdf[2 * (size_t)i + 1] =
            make_float4((float)(ux - (double)lx), (float)(uy - (double)ly), (float)(uz - (double)lz), 0.f);
    }
}

} // namespace
