// Pair kernels over a Verlet-skin neighbour list: packed (served) systems,
// and single systems whose box allows it (in binary64 those of one kind).
//
// Systems on the per-step path rebuild their list every step in the
// current (reference cell) order.  Skin-list systems keep a list of radius
// rc + skin indexed by a slot number and rebuild it only when an atom has
// moved more than skin/2 since the last build -- the usual Verlet-list
// criterion, which keeps every pair that can come within the cutoff in the
// list.  Pairs are still tested against the exact cutoff at every
// evaluation, so the list only prunes.
//
// Slots.  Every list build numbers the slots in the current cell order (slot
// = index), so the lists and gathers of a warp stay in one part of the box
// however far the atoms have diffused; between builds a slot travels with its
// atom through the re-binnings.  (Slots that stayed the upload positions: a
// fluid of 192 000 LJ atoms at 3000 K went from 277 to 335 us a step in
// 30 000 steps, in mixed precision 152 to 216; 268 and 144 throughout now.)  Packed systems refresh their cells only on rebuild
// steps, so between rebuilds slot and index coincide.
//
// Packed step:
//   k_skin_start    velocity-Verlet start step, per-step slot positions,
//                   displacement test -> rebuild flag
//   (rebuild steps only) k_refresh_cluster (fmdg_bin.cu): reference-order
//                   cell refresh and slot tables (renumbered; k_pack_* for
//                   large systems);
//   k_nlist_skin    stencil scan of the cells within the list radius
//   k_density_skin  EAM pass 1 + embedding
//   k_force_skin    pair forces + velocity-Verlet finish step + thermo
//                   record; 2^lane_log lanes per slot in both
// Single-system step: the reference-order refresh with the slot tables every
// step, k_nlist_skin (when flagged; renumbers the slots), density, forces.
//
// Geometry.  An atom's binary32 position is kept relative to the cell it
// had at the last build (unwrapped across periodic faces: it moves less
// than skin/2 before the next build), and a list entry holds the stencil
// offset between the two build cells, so a pair is formed exactly as on the
// per-step path: x_i - x_j - offset * cellh.  Binary64: the minimum image
// as the reference's ghost copy forms it (x_j + shift, then x_i minus that,
// src/md-ghost.c:85-107, src/forces.h:25-34); every periodic box length
// exceeds twice the list radius, so one image at most lies inside it.
// Pair arithmetic and precision modes are those of the per-step kernels
// (fmdg_force.cu); the lean variants (one kind, no group) are described at
// k_force_skin.
#include <algorithm>
#include <type_traits>

#include "fmdg_pairs.cuh"
#include "fmdg_prep.cuh"

namespace {

// list entry (read as unsigned): neighbour slot | stencil code << 25; code
// < 125 over a stencil of radius R (width W = 2R + 1):
// ((ox + R) W + (oy + R)) W + (oz + R).  Layout: rounds of four entries,
// int4 row (k / 4) * cap + t holds entries k..k+3 of slot t (one 16-byte
// access per round; a row is contiguous over consecutive slots).
constexpr int SLOT_BITS = 25;
constexpr int SLOT_MASK = (1 << SLOT_BITS) - 1;

// Image offsets of the stencil codes in shared memory, in the scaled frame
// (Geo::xs): off = (ox, oy, oz) * cellh_s is exact in binary32 (|o| <= 2);
// the remainder offl = (ox, oy, oz) * (cellh xs - cellh_s) completes it to
// the binary64 offset (in binary32 one more subtraction in the general
// kernels, zero on a cubic grid; binary64 mode forms both from the steps).
template <bool LO>   // LO: with the remainders (general binary32 kernels)
struct SkinOffT
{
    float4 off[125];    // image offset of each stencil code, binary32; .w: the code's bits
    float4 offl[LO ? 125 : 1];   // the remainders (binary64 offset - off)
    unsigned steps[125];         // (ox, oy, oz), for rv_steps
};

template <bool LO>
__device__ __forceinline__ void load_offsets(const Geo &g, SkinOffT<LO> &so)
{
    // (constant divisors: the stencil is 3 or 5 cells wide)
    const int R = g.srad, n = R == 1 ? 27 : 125;
    for (int c = threadIdx.x; c < n; c += blockDim.x)
    {
        const int cx = R == 1 ? c / 9 : c / 25, cy = R == 1 ? c / 3 % 3 : c / 5 % 5, cz = R == 1 ? c % 3 : c % 5;
        const float ox = small_int_f(cx - R), oy = small_int_f(cy - R), oz = small_int_f(cz - R);
        so.off[c] = make_float4(ox * g.cellh_s[0], oy * g.cellh_s[1], oz * g.cellh_s[2], __int_as_float(c));
        if (LO) so.offl[c] = make_float4(ox * g.cellh_slo[0], oy * g.cellh_slo[1], oz * g.cellh_slo[2], 0.f);
        so.steps[c] = __float_as_uint(ox) | __float_as_uint(oy) >> 10 | __float_as_uint(oz) >> 20;
    }
    __syncthreads();
}

__device__ __forceinline__ float norm2(float3 v)
{
    return __fmaf_rn(v.z, v.z, __fmaf_rn(v.y, v.y, __fmul_rn(v.x, v.x)));
}

// spl_der with its roundings spelled out
__device__ __forceinline__ float spl_der_rn(float4 t, float b, float inv_h)
{
    return __fmul_rn(__fmaf_rn(__fmaf_rn(__fmul_rn(3.f, t.w), b, __fmul_rn(2.f, t.z)), b, t.y), inv_h);
}

// binary32 pair vector x_i - x_j - offset without the offset's remainder
// (prefilters, overflow fallback)
__device__ __forceinline__ float3 rv_of(float4 xi, float4 xj, float4 o)
{
    return make_float3(xi.x - xj.x - o.x, xi.y - xj.y - o.y, xi.z - xj.z - o.z);
}

// The same vector, bit for bit, from the cell steps packed in one word: a
// step (-2 .. 2) is the top ten bits of its binary32 form, step * cellh is
// exact, so one fused operation rounds as the subtraction of the offset
// does.  The walks are bound by L1 wavefronts: a 16-byte row of shared
// offsets took 4.4 of them per warp and entry beside the position gather's
// 12, one word takes one or two (EAM 256k density 77 -> 67 us, force
// 112 -> 102; Morse 512k 250 -> 233; binary64 EAM 256k density 194 -> 187).
__device__ __forceinline__ float3 rv_steps(float4 xi, float4 xj, unsigned w, float3 h)
{
    const float sx = __uint_as_float(w & 0xffc00000u), sy = __uint_as_float((w << 10) & 0xffc00000u),
                sz = __uint_as_float(w << 20);
    return make_float3(__fmaf_rn(-sx, h.x, xi.x - xj.x), __fmaf_rn(-sy, h.y, xi.y - xj.y),
                       __fmaf_rn(-sz, h.z, xi.z - xj.z));
}

// binary32 pair vector of a list entry with the offset's remainder: the
// binary32 rounding of (ox, oy, oz) * cellh would otherwise shift every
// pair across a cell face by up to half an ulp of the cell width
// (5e-7 A), as much as the rounding of the coordinates themselves.  o.w
// holds the stencil code (an overflow-fallback occurrence: -1 - code).
template <bool DF>
__device__ __forceinline__ float3 rv_lo(const SkinOffT<DF> &so, float4 xi, float4 xj, float4 o)
{
    const int code = __float_as_int(o.w);
    const float4 ol = so.offl[code ^ (code >> 31)];
    return make_float3(xi.x - xj.x - o.x - ol.x, xi.y - xj.y - o.y - ol.y, xi.z - xj.z - o.z - ol.z);
}

// binary64 minimum-image geometry rv = x_a - (x_b + shift)
__device__ __forceinline__ Geom64 geom64_mi(const Geo &g, double4_32a a, double4_32a b)
{
    const double xa[3] = {a.x, a.y, a.z}, xb[3] = {b.x, b.y, b.z};
    Geom64 p;
    for (int d = 0; d < 3; d++)
    {
        double x2 = xb[d];
        if (g.pbc[d])
        {
            const double dd = xa[d] - x2;
            if (dd > 0.5 * g.l[d]) x2 = __dadd_rn(x2, g.l[d]);
            else if (dd < -0.5 * g.l[d]) x2 = __dadd_rn(x2, -g.l[d]);
        }
        p.rv[d] = __dsub_rn(xa[d], x2);
    }
    p.r2 = __dadd_rn(__dadd_rn(__dmul_rn(p.rv[0], p.rv[0]), __dmul_rn(p.rv[1], p.rv[1])),
                     __dmul_rn(p.rv[2], p.rv[2]));
    return p;
}

// binary32 cutoff test; within 1e-4 relative of the cutoff the decision is
// taken in binary64 from the binary64 positions
__device__ __forceinline__ bool within_cut_skin(const Geo &g, int ta, int tb, float r2f, float rc2f, double rc2)
{
    if (fabsf(r2f - rc2f) > 1e-4f * rc2f) return r2f < rc2f;
    return geom64_mi(g, g.xd[ta], g.xd[tb]).r2 < rc2;
}

// Gap along one axis between a point at u inside its cell box [0, h) and
// the cell at offset o (0 for the cell itself).
__device__ __forceinline__ float axis_gap(int o, float u, float h)
{
    return o > 0 ? fmaxf(0.f, (float)o * h - u) : (o < 0 ? fmaxf(0.f, u + (float)(-o - 1) * h) : 0.f);
}

// Binary64 mode: double-float geometry of a list entry (build frame: the
// slots' rows and the entry's cell steps, times the double-float cell width:
// exact, and rounded once)
__device__ __forceinline__ GeomDF skin_geom_df(float4 ih, float4 il, float4 jh, float4 jl, unsigned w, float3 h, float3 hl)
{
    const float sx = __uint_as_float(w & 0xffc00000u), sy = __uint_as_float((w << 10) & 0xffc00000u),
                sz = __uint_as_float(w << 20);
    return geom_df(ih, il, jh, jl, make_float4(sx * h.x, sy * h.y, sz * h.z, 0.f),
                   make_float4(sx * hl.x, sy * hl.y, sz * hl.z, 0.f));
}

// the cutoff decision within 1e-6 relative of the cutoff is the binary64
// minimum-image one
__device__ __forceinline__ bool within_cut_df_mi(const Geo &g, int t, int js, dfl r2, float rc2f, double rc2)
{
    const float d = __fsub_rn(r2.hi, rc2f);
    if (fabsf(d) > 1e-6f * rc2f) return d < 0.f;
    return geom64_mi(g, g.xd[t], g.xd[js]).r2 < rc2;
}

// Every cell c of the stencil of radius R around cell ci, with its stencil
// code, in a fixed order: f(code, c).  On a periodic axis shorter than the
// stencil a cell recurs with another image (at most one image of a pair
// lies within the list radius).  xi: the atom's binary32 position relative
// to the centre of cell ci; a cell whose box lies farther than the list
// radius from xi (plus 1e-4 relative) holds no candidate and is skipped.
template <typename F>
__device__ __forceinline__ void for_each_stencil_cell(const Geo &g, CellXYZ ci, float4 xi, F &&f)
{
    const int R = g.srad, W = 2 * R + 1;
    const float lim2 = g.rskin2 * 1.0001f;
    // position inside the cell box [0, h) (up to the drift since the build)
    const float ux = xi.x + 0.5f * g.cellh_s[0], uy = xi.y + 0.5f * g.cellh_s[1], uz = xi.z + 0.5f * g.cellh_s[2];
    for (int ox = -R; ox <= R; ox++)
    {
        const float gx = axis_gap(ox, ux, g.cellh_s[0]);
        if (gx * gx > lim2) continue;
        int cx = ci.x + ox;
        if (cx < 0 || cx >= g.nc[0])
        {
            if (!g.pbc[0]) continue;
            cx = (cx + 2 * g.nc[0]) % g.nc[0];
        }
        for (int oy = -R; oy <= R; oy++)
        {
            const float gy = axis_gap(oy, uy, g.cellh_s[1]);
            if (gx * gx + gy * gy > lim2) continue;
            int cy = ci.y + oy;
            if (cy < 0 || cy >= g.nc[1])
            {
                if (!g.pbc[1]) continue;
                cy = (cy + 2 * g.nc[1]) % g.nc[1];
            }
            for (int oz = -R; oz <= R; oz++)
            {
                const float gz = axis_gap(oz, uz, g.cellh_s[2]);
                if (gx * gx + gy * gy + gz * gz > lim2) continue;
                int cz = ci.z + oz;
                if (cz < 0 || cz >= g.nc[2])
                {
                    if (!g.pbc[2]) continue;
                    cz = (cz + 2 * g.nc[2]) % g.nc[2];
                }
                f(((ox + R) * W + (oy + R)) * W + (oz + R), cz + g.nc[2] * (cy + g.nc[1] * cx));
            }
        }
    }
}

// the stencil code of the atom's own cell
__device__ __forceinline__ int home_code(const Geo &g)
{
    const int R = g.srad, W = 2 * R + 1;
    return (R * W + R) * W + R;
}

// every (j, code) of the stencil around i's current cell, j the current
// index, i itself left out
template <typename F>
__device__ __forceinline__ void for_each_candidate(const Geo &g, const Side &S, int i, float4 xi, F &&f)
{
    const int home = home_code(g);
    for_each_stencil_cell(g, cell_xyz(g, S.cell_of[i]), xi, [&](int code, int c) {
        const int je = S.cell_start[c + 1];
        for (int j = S.cell_start[c]; j < je; j++)
            if (!(code == home && j == i)) f(j, code);
    });
}

struct NoRound
{
    __device__ __forceinline__ void operator()(int) const {}
};

// An atom whose list overflowed scans the stencil of its cell directly:
// positions are the current binary64 ones relative to the cells of the
// last refresh (packed systems refresh their cells only at a rebuild; an
// atom has moved less than skin/2 since, so the stencil still covers the
// list radius), and of the occurrences of a neighbour (a cell recurs in the
// stencil when an axis has fewer than 2R + 1 cells) only the image within
// the list radius is passed on.  Share v of V takes every V-th candidate.
// ONE: a single system, whose refresh has just written every atom's binary32
// position in its current cell (xf4): the same numbers without binary64 work
// for each of some thousand candidates.  A laser-heated slab of 10 000 atoms
// whose density outgrew its lists took 26 ms for 25 steps with one lane and
// binary64 positions, 5 now.
template <bool ONE, typename F, bool DF>
__device__ __forceinline__ void for_each_slot_overflow(const Geo &g, const Side &S, const SkinOffT<DF> &so, int t,
                                                       int i, int v, int V, float4 &xi, F &&f)
{
    const double4_32a xdi = g.xd[t], oi = g.corig[S.cell_of[i]];
    const double xs = g.xs;
    xi = make_float4((float)((xdi.x - oi.x) * xs), (float)((xdi.y - oi.y) * xs), (float)((xdi.z - oi.z) * xs), xi.w);
    const float lim2 = g.rskin2 * 1.0001f;
    int turn = 0;
    for_each_candidate(g, S, i, xi, [&](int j, int code) {
        if ((turn++ & (V - 1)) != v) return;
        float4 xj = g.xf4[j];
        const int js = S.slot[j];
        if (!ONE)
        {
            const double4_32a xdj = g.xd[js], oj = g.corig[S.cell_of[j]];
            xj = make_float4((float)((xdj.x - oj.x) * xs), (float)((xdj.y - oj.y) * xs),
                             (float)((xdj.z - oj.z) * xs), xj.w);
        }
        float4 o = so.off[code];
        const float3 d = rv_of(xi, xj, o);
        if (d.x * d.x + d.y * d.y + d.z * d.z > lim2) return;
        o.w = __int_as_float(-1 - code);    // current-cell frame, not the build frame
        f(js, xj, o);
    });
}

// Share v of V of the list walk of slot t (rounds of four entries; share v
// takes rounds v, v + V, ...): f(neighbour slot, its binary32 position,
// image offset); r(k) after every k entries visited (a round of four, or
// one).  PF: the next round's list rows are prefetched into L1 while this
// round is processed (the rows stream from DRAM).
// An atom whose list overflowed: for_each_slot_overflow.
template <bool ONE, bool PF = false, typename F, typename R, bool DF>
__device__ __forceinline__ void for_each_slot_pair(const Geo &g, const Side &S, const SkinOffT<DF> &so, int t, int i,
                                                   int v, int V, float4 &xi, F &&f, R &&r)
{
    const int cnt = g.nbr_count[t];
    if (cnt <= g.maxnb)
    {
        const int cap = g.cap, step = 4 * V;
        const int4 *col = reinterpret_cast<const int4 *>(g.nbr) + t;
        int k = 4 * v;
        for (; k + 4 <= cnt; k += step)
        {
            if (PF && k + step + 4 <= cnt)
                asm volatile("prefetch.global.L1 [%0];" ::"l"(col + (size_t)((k + step) >> 2) * cap));
            const int4 e4 = col[(size_t)(k >> 2) * cap];
            const int e0 = e4.x, e1 = e4.y, e2 = e4.z, e3 = e4.w;
            const float4 x0 = g.xl[e0 & SLOT_MASK], x1 = g.xl[e1 & SLOT_MASK];
            const float4 x2 = g.xl[e2 & SLOT_MASK], x3 = g.xl[e3 & SLOT_MASK];
            f(e0 & SLOT_MASK, x0, so.off[(unsigned)e0 >> SLOT_BITS]);
            f(e1 & SLOT_MASK, x1, so.off[(unsigned)e1 >> SLOT_BITS]);
            f(e2 & SLOT_MASK, x2, so.off[(unsigned)e2 >> SLOT_BITS]);
            f(e3 & SLOT_MASK, x3, so.off[(unsigned)e3 >> SLOT_BITS]);
            r(4);
        }
        if (k < cnt)
        {
            // the last, partial round (1-3 entries)
            const int4 e4 = col[(size_t)(k >> 2) * cap];
            const int ee[3] = {e4.x, e4.y, e4.z};
            for (int q = 0; q < 3 && k + q < cnt; q++)
            {
                const int e = ee[q];
                f(e & SLOT_MASK, g.xl[e & SLOT_MASK], so.off[(unsigned)e >> SLOT_BITS]);
                r(1);
            }
        }
    }
    else
        for_each_slot_overflow<ONE>(g, S, so, t, i, v, V, xi, [&](int js, float4 xj, float4 o) {
            f(js, xj, o);
            r(1);
        });
}

template <bool ONE, typename F, bool DF>
__device__ __forceinline__ void for_each_slot_pair(const Geo &g, const Side &S, const SkinOffT<DF> &so, int t, int i,
                                                   int v, int V, float4 &xi, F &&f)
{
    for_each_slot_pair<ONE>(g, S, so, t, i, v, V, xi, f, NoRound{});
}

// The double-float kernels' walk.  Their pair arithmetic costs hundreds of
// instructions, and a list entry out of range (a fifth to a third of a skin
// list) would idle its lane for all of them, as the lanes of a warp hardly
// ever agree.  So share v of V of slot t's list is first pruned: rounds of
// four entries tested in binary32 against the largest cutoff (widened by
// 2e-5 relative, far above the binary32 error), the entries in range
// written to the share's own compact list (entry m at nbc[m cap V + t V + v]:
// a row over consecutive shares), which the double-float loop then walks.
// The EAM force pass reuses the density pass's compact lists.
__device__ __forceinline__ int prune_share(const Geo &g, const SkinOffT<false> &so, int cnt, int t, int v, int V,
                                           float4 ih)
{
    const int cap = g.cap;
    const size_t row = (size_t)cap * V;
    const float lim = g.rcut2;
    const int4 *col = reinterpret_cast<const int4 *>(g.nbr) + t;
    unsigned *out = g.nbc + (size_t)t * V + v;
    const float3 h3 = make_float3(g.cellh_s[0], g.cellh_s[1], g.cellh_s[2]);
    int m = 0;
    for (int k = 4 * v; k < cnt; k += 4 * V)
    {
        const int4 e4 = col[(size_t)(k >> 2) * cap];
        const int left = cnt - k;
        // (the words behind a list's last entry are not defined)
        const unsigned e[4] = {(unsigned)e4.x, left > 1 ? (unsigned)e4.y : (unsigned)e4.x,
                               left > 2 ? (unsigned)e4.z : (unsigned)e4.x, left > 3 ? (unsigned)e4.w : (unsigned)e4.x};
        float4 x[4];
        for (int w = 0; w < 4; w++) x[w] = g.xl[e[w] & SLOT_MASK];
        for (int w = 0; w < 4; w++)
        {
            const float3 d = rv_steps(ih, x[w], so.steps[e[w] >> SLOT_BITS], h3);
            if (w < left && d.x * d.x + d.y * d.y + d.z * d.z < lim)
            {
                *out = e[w];
                out += row;
                m++;
            }
        }
    }
    return m;
}

// f(neighbour slot, its double-float row, the entry's cell steps) for the m
// entries of a share's compact list.  L1 wavefronts bound the walk, so a
// neighbour is one 32-byte row and its offset one shared word (rv_steps),
// F'(rho_j) rides in the row (LEAN) and the EAM slopes come from one 64-byte
// row (eam_pair_row): 256k EAM density 187 -> 166 us, force 230 -> 177, L1
// wavefronts from 80 % of their peak (the FMA pipe at 38 to 50 %) to 68 and
// 73 % (44 and 62 %); 300 jobs of 600 to 3000 atoms 1464 -> 1160 us a step.
template <typename F>
__device__ __forceinline__ void for_each_pruned(const Geo &g, const SkinOffT<false> &so, int m, int t, int v, int V, F &&f)
{
    const size_t row = (size_t)g.cap * V;
    const unsigned *p = g.nbc + (size_t)t * V + v;
    unsigned next = m > 0 ? *p : 0u;
    for (int k = 0; k < m; k++)
    {
        const unsigned e = next;
        p += row;
        if (k + 1 < m) next = *p;
        float4 jh, jl;
        ld_slot32(g.xr + 2 * (size_t)(e & SLOT_MASK), jh, jl);
        f((int)(e & SLOT_MASK), jh, jl, so.steps[e >> SLOT_BITS]);
    }
}

// sum over the lanes of a group of G (every lane of the warp takes part)
__device__ __forceinline__ dfl group_sum(dfl v, int G)
{
    for (int o = G >> 1; o > 0; o >>= 1)
    {
        const dfl w = {__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
        v = df_add(v, w);
    }
    return v;
}

// ---------------------------------------------------------------- kernels

// Packed systems, every step (one thread per current atom index): the
// velocity-Verlet start step (src/integrators.c:40-75, the operations of
// k_bin_classify), the slot tables that change every step and the
// displacement test; advances the device time by one step.  The cells and
// the remaining slot tables are refreshed on rebuild steps only.
template <class L>
__global__ void k_skin_start(__grid_constant__ const L loc)
{
    step_wait();
    int bx, nb;
    const Geo &g = loc_geo(loc, bx, nb);
    if (loc_idle(loc, g)) return;
    const double dt = g.st.dt;
    const int group = g.st.group, thermostat = g.st.thermostat;
    __shared__ double hk[FMDG_MAXK];
    if (threadIdx.x < g.nkinds) hk[threadIdx.x] = g.st.hk[threadIdx.x];
    __syncthreads();
    Dyn *dyn = g.dyn;
    if (bx == 0 && threadIdx.x == 0) dyn->time += dt;
    const int i = bx * blockDim.x + threadIdx.x;
    if (i >= dyn->n) return;
    const Side S = g.side[dyn->cur];
    const size_t cap = g.cap;
    const int kind = (int)S.kind[i];
    double x[3] = {S.x[i], S.x[cap + i], S.x[2 * cap + i]};
    if (group < 0 || S.group[i] == group)
    {
        const double lam = dyn->lambda;
        const double coef = hk[kind];
        for (int d = 0; d < 3; d++)
        {
            double vv = S.v[d * cap + i];
            if (thermostat) vv = __dmul_rn(vv, lam);
            vv = __dadd_rn(vv, __dmul_rn(coef, g.F[d * cap + i]));
            S.v[d * cap + i] = vv;
            x[d] = __dadd_rn(x[d], __dmul_rn(dt, vv));
            S.x[d * cap + i] = x[d];
        }
    }
    const int t = S.slot[i];
    g.xd[t] = make_double4_32a(x[0], x[1], x[2], 0.0);
    slot_rel_build(g, dyn, t, x, __int_as_float(kind));
}

// The per-atom tables of the current positions (prep_skin_atom), one thread per
// atom, for a force evaluation without a refresh before it
__global__ void __launch_bounds__(128) k_prep_skin(__grid_constant__ const LocOne loc)
{
    const Geo &g = loc.g;
    Dyn *dyn = g.dyn;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= dyn->n) return;
    const Side S = g.side[dyn->cur];
    const int cap = g.cap;
    const double x[3] = {S.x[i], S.x[cap + i], S.x[2 * (size_t)cap + i]};
    prep_skin_atom(g, dyn, i, S.slot[i], S.cell_of[i], (int)S.kind[i], S.group[i], x, !dyn->rebuild);
}

// The stencil walk of a list build: f(code, c, ax, ay, az) for every cell
// of for_each_stencil_cell, with the cell's image offset folded into the
// atom's position once per cell (ax, ay, az).
template <typename F>
__device__ __forceinline__ void for_each_build_cell(const Geo &g, const SkinOffT<false> &so, CellXYZ ci, float4 xi,
                                                    F &&f)
{
    for_each_stencil_cell(g, ci, xi, [&](int code, int c) {
        const float4 o = so.off[code];
        f(code, c, xi.x - o.x, xi.y - o.y, xi.z - o.z);
    });
}

// Per-slot state recorded with a new list: build cell and build-frame
// position (+ its double-float remainder in binary64 mode).  Slot = index:
// packed systems were renumbered by the refresh, a single system is here --
// nothing in a build reads a slot table of another atom, so every thread
// rewrites its own row of them.
template <class L>
__device__ __forceinline__ void record_build(const Geo &g, const Side &S, int t, float4 xi)
{
    const int c = S.cell_of[t];
    g.cb[t] = c;
    g.xl[t] = xi;
    g.xb[t] = xi;
    if (!L::one_system && g.prec != FMDG_PREC_FP64) return;
    const size_t cap = g.cap;
    const double4_32a x = L::one_system ? make_double4_32a(S.x[t], S.x[cap + t], S.x[2 * cap + t], 0.0) : g.xd[t];
    if (L::one_system)
    {
        S.slot[t] = t;
        g.pos[t] = t;
        g.xd[t] = x;
        g.gslot[t] = S.group[t];
    }
    if (g.prec == FMDG_PREC_FP64)
    {
        // (xs is 1 in binary64 mode)
        const double4_32a o = g.corig[c];
        g.xr[2 * (size_t)t] = xi;
        g.xr[2 * (size_t)t + 1] = make_float4((float)(x.x - o.x - (double)xi.x), (float)(x.y - o.y - (double)xi.y),
                                              (float)(x.z - o.z - (double)xi.z), 0.f);
    }
}

// the last block of a build to finish clears the system's rebuild flag
__device__ __forceinline__ void finish_build(Dyn *dyn, int nb)
{
    __shared__ unsigned ticket;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        ticket = atomicAdd(&dyn->nl_done, 1u);
    }
    __syncthreads();
    if (ticket == (unsigned)nb - 1 && threadIdx.x == 0)
    {
        dyn->nl_done = 0;
        dyn->rebuild = 0;
    }
}

// one thread per slot; every block leaves at once when no rebuild is due
template <class L>
__global__ void __launch_bounds__(L::max_threads, L::min_blocks) k_nlist_skin(__grid_constant__ const L loc)
{
    step_wait();
    int bx, nb;
    const Geo &g = loc_geo(loc, bx, nb);
    if (loc_idle(loc, g)) return;
    Dyn *dyn = g.dyn;
    if (!dyn->rebuild) return;
    __shared__ SkinOffT<false> so;
    load_offsets(g, so);
    const int cap = g.cap, maxnb = g.maxnb;
    const int t = bx * blockDim.x + threadIdx.x;
    if (t < cap)
    {
        int cnt = 0;
        const int i = t;        // (slot = index: record_build)
        if (i < dyn->n)
        {
            const Side S = g.side[dyn->cur];
            const float4 *xf = after_wait<true>(g.xf4);
            const float4 xi = xf[i];
            const float rl2 = g.rskin2;
            int4 *row = reinterpret_cast<int4 *>(g.nbr) + t;
            // Up to 32 candidates of a cell give a mask of hits first, then
            // the hits are taken from the mask: a lane hits at 8 % of its
            // candidates but some lane of the warp at nearly all, so a
            // candidate costs what every lane runs for it, and the test
            // alone is 11 instructions where test and entry were 25 (512k
            // atoms, 8 A cutoff: 1020 us a build before, 850 now; 256k EAM 337
            // and 246; 600 jobs of 600 to 3000 atoms 785 and 740 us a step).
            // Entries shift through a four-entry register buffer (in order:
            // x oldest); every fourth writes one 16-byte row.  The radius is
            // widened by 1e-5 relative so the folded rounding of the cell
            // offsets can only add entries.
            const float rb2 = rl2 * 1.00001f;
            int4 buf = make_int4(0, 0, 0, 0);
            const int center = home_code(g);
            for_each_build_cell(g, so, cell_xyz(g, S.cell_of[i]), xi, [&](int code, int c, float ax, float ay, float az) {
                const int jb = S.cell_start[c], je = S.cell_start[c + 1];
                auto near = [&](int j) {
                    const float4 xj = ld_step<L::free_loads>(xf + j);
                    return norm2(make_float3(ax - xj.x, ay - xj.y, az - xj.z)) < rb2;
                };
                for (int j0 = jb; j0 < je; j0 += 32)
                {
                    const int n = min(je - j0, 32);
                    unsigned m = 0;
                    int k = 0;
                    for (; k + 4 <= n; k += 4)
                    {
                        const bool h0 = near(j0 + k), h1 = near(j0 + k + 1), h2 = near(j0 + k + 2), h3 = near(j0 + k + 3);
                        m |= ((h0 ? 1u : 0u) | (h1 ? 2u : 0u) | (h2 ? 4u : 0u) | (h3 ? 8u : 0u)) << k;
                    }
                    for (; k < n; k++) m |= near(j0 + k) ? 1u << k : 0u;
                    // (not the atom itself, in its own cell)
                    if (code == center && (unsigned)(i - j0) < 32u) m &= ~(1u << (i - j0));
                    for (; m; m &= m - 1)
                    {
                        const int j = j0 + __ffs(m) - 1;
                        buf = make_int4(buf.y, buf.z, buf.w, (int)((unsigned)j | ((unsigned)code << SLOT_BITS)));
                        cnt++;
                        if ((cnt & 3) == 0 && cnt <= maxnb) row[(size_t)((cnt >> 2) - 1) * cap] = buf;
                    }
                }
            });
            const int rem = cnt & 3;
            if (rem && cnt <= maxnb)
            {
                const int4 last = (rem == 1) ? make_int4(buf.w, 0, 0, 0)
                                : (rem == 2) ? make_int4(buf.z, buf.w, 0, 0) : make_int4(buf.y, buf.z, buf.w, 0);
                row[(size_t)(cnt >> 2) * cap] = last;
            }
            record_build<L>(g, S, t, xi);
        }
        else
            g.pos[t] = -1;
        g.nbr_count[t] = cnt;
    }
    finish_build(dyn, nb);
}

// The list of slot t built by the G lanes of a group (gl: this lane's
// index in it, gbase: the group's first lane in the warp): the lanes test
// G consecutive candidates of a cell together and place their hits in
// candidate order (ballot + prefix count), so the list is the one-thread
// build's, entry for entry.  Every lane of the group must call it (its
// control flow depends on the slot only).
__device__ __forceinline__ void build_slot_grouped(const Geo &g, const Side &S, const SkinOffT<false> &so, int t, int n,
                                                   int G, int gl, int gbase)
{
    const int cap = g.cap, maxnb = g.maxnb;
    const unsigned gmask = (G == 32) ? 0xffffffffu : ((1u << G) - 1u) << gbase;
    int cnt = 0;
    const int i = t;        // (slot = index: record_build)
    if (i < n)
    {
        const float4 xi = g.xf4[i];
        const float rb2 = g.rskin2 * 1.00001f;   // as in k_nlist_skin
        int *ent = g.nbr;   // entry k of slot t: int4 row (k / 4) * cap + t, component k % 4
        const int center = home_code(g);
        for_each_build_cell(g, so, cell_xyz(g, S.cell_of[i]), xi, [&](int code, int c, float ax, float ay, float az) {
            const int jb = S.cell_start[c], je = S.cell_start[c + 1];
            const bool self = code == center;
            for (int base = jb; base < je; base += G)
            {
                const int j = base + gl;
                bool hit = false;
                if (j < je && !(self && j == i))
                {
                    const float4 xj = g.xf4[j];
                    const float dx = ax - xj.x, dy = ay - xj.y, dz = az - xj.z;
                    hit = dx * dx + dy * dy + dz * dz < rb2;
                }
                const unsigned m = __ballot_sync(gmask, hit) >> gbase;
                if (hit)
                {
                    const int k = cnt + __popc(m & ((1u << gl) - 1u));
                    if (k < maxnb)
                        ent[((size_t)(k >> 2) * cap + t) * 4 + (k & 3)] =
                            (int)((unsigned)j | ((unsigned)code << SLOT_BITS));
                }
                cnt += __popc(m);
            }
        });
        if (gl == 0) record_build<LocOne>(g, S, t, xi);
    }
    else if (gl == 0)
        g.pos[t] = -1;
    if (gl == 0) g.nbr_count[t] = cnt;
}

// Single-system build (a served job's admission, the fmd.h path) with G
// lanes per slot: a system of 10^3-10^5 atoms gives one thread per slot too
// few warps to hide the gather latency of its long candidate walk.
template <int G>
__global__ void __launch_bounds__(128) k_nlist_skin_grp(__grid_constant__ const LocOne loc)
{
    step_wait();
    static_assert(G >= 2 && G <= 32 && (G & (G - 1)) == 0, "G: a power of two up to the warp");
    const Geo &g = loc.g;
    Dyn *dyn = g.dyn;
    if (!dyn->rebuild) return;
    __shared__ SkinOffT<false> so;
    load_offsets(g, so);
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) / G;   // uniform over a group
    if (t < g.cap) build_slot_grouped(g, g.side[dyn->cur], so, t, dyn->n, G, threadIdx.x & (G - 1), threadIdx.x & 31 & ~(G - 1));
    finish_build(dyn, gridDim.x);
}

// Shares and lanes.  A slot's list walk is split into V = 2^share_log shares
// whose partial sums meet in a fixed binary tree (share v with v + V/2
// first), so the result depends on V alone, and V on the system's size alone
// (fmdg_share_log).  A slot is given G = 2^lane_log <= V lanes, each of
// which walks V / G shares: single systems G = V, packed ones fewer while
// enough other atoms run (a served job's arithmetic must not depend on the
// mix).  part_tree: the part of the tree inside one lane; share_log -
// lane_log levels over the lane's M = V / G partial sums.
constexpr int MAX_SHARES = 16;
template <int NV>
__device__ __forceinline__ void part_tree(dfl (&part)[MAX_SHARES][NV], int M, int nv, dfl (&sum)[NV])
{
    for (int h = M >> 1; h > 0; h >>= 1)
        for (int m = 0; m < h; m++)
            for (int q = 0; q < nv; q++) part[m][q] = df_add(part[m][q], part[m + h][q]);
    for (int q = 0; q < nv; q++) sum[q] = part[0][q];
}

// The per-slot epilogues (embedding; finish step and block sums) are
// binary64 work, which issues at 1/64 of the binary32 rate: run by every
// group's first lane they would cost one warp's issue per 32 / G slots.  The
// groups' sums go through shared memory instead (rows of blockDim / G) and
// the block's first blockDim / G threads take one slot each, full warps
// again.  Every thread of the block calls these; the sums meet in a fixed
// tree over the lanes.
extern __shared__ double stage[];

// the slot whose epilogue this thread runs, -1: none
__device__ __forceinline__ int slot_of_thread(const Geo &g, int bx, int gl)
{
    const int apb = blockDim.x >> gl;
    const int t = bx * apb + threadIdx.x;
    return ((int)threadIdx.x < apb && t < g.cap) ? t : -1;
}

// one value per slot: that of this thread's slot
__device__ __forceinline__ double group_value(dfl v, int gl)
{
    if (gl == 0) return df_to_double(v);
    v = group_sum(v, 1 << gl);
    if ((threadIdx.x & ((1 << gl) - 1)) == 0) stage[threadIdx.x >> gl] = df_to_double(v);
    __syncthreads();
    return (int)threadIdx.x < (int)(blockDim.x >> gl) ? stage[threadIdx.x] : 0.0;
}

// The force (3 values), and with `thermo` energy and virial, of this
// thread's slot.  The force values are summed by a transposing butterfly: an
// exchange halves the values a lane carries, 2 + 1 + 1 + ... double-float
// additions instead of three per level.
__device__ __forceinline__ void group_forces(const dfl (&v)[5], int gl, bool thermo, double (&out)[5])
{
    if (gl == 0)
    {
        for (int q = 0; q < 5; q++) out[q] = df_to_double(v[q]);
        return;
    }
    const int G = 1 << gl, lane = threadIdx.x & (G - 1), apb = blockDim.x >> gl, row = threadIdx.x >> gl;
    auto take = [](dfl keep, dfl give, int o) {
        const dfl w = {__shfl_xor_sync(0xffffffffu, give.hi, o), __shfl_xor_sync(0xffffffffu, give.lo, o)};
        return df_add(keep, w);
    };
    int o = G >> 1;
    const bool up = (lane & o) != 0;     // keeps values 2, 3 (else 0, 1); 3: the energy
    const dfl k0 = take(up ? v[2] : v[0], up ? v[0] : v[2], o);
    dfl k1 = take(up ? v[3] : v[1], up ? v[1] : v[3], o);
    o >>= 1;
    if (o == 0)
    {
        stage[(up ? 2 : 0) * apb + row] = df_to_double(k0);
        stage[(up ? 3 : 1) * apb + row] = df_to_double(k1);
    }
    else
    {
        const bool up2 = (lane & o) != 0;
        dfl r = take(up2 ? k1 : k0, up2 ? k0 : k1, o);
        const int q = (up ? 2 : 0) + (up2 ? 1 : 0), low = o - 1;
        for (o >>= 1; o > 0; o >>= 1) r = take(r, r, o);
        if ((lane & low) == 0) stage[q * apb + row] = df_to_double(r);
    }
    if (thermo)
    {
        const dfl e = group_sum(v[4], G);
        if (lane == 0) stage[4 * apb + row] = df_to_double(e);
    }
    __syncthreads();
    const int mine = (int)threadIdx.x < apb ? threadIdx.x : 0;
    for (int q = 0; q < 5; q++) out[q] = (q < 4 || thermo) ? stage[q * apb + mine] : 0.0;
}

// EAM pass 1 + embedding (src/eam.h:270-406, src/eam.c:160-179), a group of
// 2^lane_log lanes per slot (see k_force_skin).  LEAN (one kind, no group): the pair's table
// row and cutoff in registers, no per-entry kind or group lookups; F'(rho)
// goes into the slots' rows.
template <class L, bool MIXED, bool HYBRID, bool LEAN>
__global__ void __launch_bounds__(L::max_threads, MIXED ? L::min_blocks : L::df_min_blocks) k_density_skin(__grid_constant__ const L loc, int rec)
{
    int bx, nb;
    const Geo &g = loc_geo(loc, bx, nb);
    const int group = g.st.group;
    __shared__ SmemPotT<!MIXED, LEAN> sp;
    __shared__ SkinOffT<MIXED && !LEAN> so;   // (lean binary32: no remainders, exact on a cubic grid)
    load_pot<false>(g, sp, skin_params(g));
    load_offsets(g, so);
    step_wait();        // (the tables above were set up before any step)
    if (loc_idle(loc, g)) return;
    Dyn *dyn = g.dyn;
    const Side S = g.side[dyn->cur];
    const int gl = L::one_lane ? 0 : g.lane_log, lane = threadIdx.x & ((1 << gl) - 1);
    double acc[1] = {0.0};
    dfl dens[1] = {{0.f, 0.f}};    // this lane's shares of the density
    auto is_active = [&](int t, int ki) {
        return (group < 0 || g.gslot[t] == group) && sp.elem[ki] >= 0;   // hybrid: EAM kinds only
    };
    {
        const int t = (bx * blockDim.x + threadIdx.x) >> gl;
        const int i = (t < g.cap) ? g.pos[t] : -1;
        float4 xi = i >= 0 ? g.xl[t] : make_float4(0.f, 0.f, 0.f, 0.f);
        const int ki = (LEAN || i < 0) ? 0 : __float_as_int(xi.w);
        const int nk = g.nkinds, nint = g.Nr2 - 1;
        const bool on = i >= 0 && is_active(t, ki);
        const int V = L::one_lane ? 1 : 1 << g.share_log, M = L::split_shares ? V >> gl : 1;
        dfl part[L::split_shares ? MAX_SHARES : 1][1];
        for (int m = 0; m < M; m++)
        {
            const int v = lane + (m << gl);
            dfl acc_rho = {0.f, 0.f};
            if constexpr (!MIXED)
            {
                // double-float pair arithmetic (fmdg_df.cuh)
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 ih = on ? g.xr[2 * (size_t)t] : zero, il = on ? g.xr[2 * (size_t)t + 1] : zero;
                const float3 h3 = make_float3(g.cellh_s[0], g.cellh_s[1], g.cellh_s[2]);
                const float3 hl3 = make_float3(g.cellh_slo[0], g.cellh_slo[1], g.cellh_slo[2]);
                const dfl inv_h = df_of(g.inv_h_df);
                const float kmax = (float)(nint - 1);
                // (LEAN: the rows' w is not the kind)
                auto pair = [&](int js, float w, auto &&geom) {
                    if (!LEAN && group >= 0 && g.gslot[js] != group) return;
                    const int pidx = LEAN ? 0 : ki * nk + __float_as_int(w);
                    const fmdg_pair_t &pp = sp.pairs[pidx];
                    if (HYBRID && pp.cat != FMDG_POT_EAM) return;
                    const GeomDF p = geom();
                    if (within_cut_df_mi(g, t, js, p.r2, sp.pf[pidx][2], pp.p[2]))
                        acc_rho = df_add(acc_rho, df_rho(g, pp, p, inv_h, kmax, nint));
                };
                const int cnt = on ? g.nbr_count[t] : 0;
                const int m_in = prune_share(g, so, cnt <= g.maxnb ? cnt : 0, t, v, V, ih);
                if (on) g.nbc_count[(size_t)t * V + v] = m_in;
                for_each_pruned(g, so, m_in, t, v, V, [&](int js, float4 jh, float4 jl, unsigned w) {
                    pair(js, jh.w, [&]() { return skin_geom_df(ih, il, jh, jl, w, h3, hl3); });
                });
                if (cnt > g.maxnb)
                    for_each_slot_overflow<L::one_system>(g, S, so, t, i, v, V, xi, [&](int js, float4 xj, float4) {
                        pair(js, xj.w, [&]() { return geom_df_of64(geom64_mi(g, g.xd[t], g.xd[js])); });
                    });
            }
            else if (!on)
                ;
            else if constexpr (LEAN)
            {
                // branch-free walk (table rows read for every entry, entries
                // beyond the cutoff add zero), in rounds of four as in the
                // lean force kernel: cutoff decided in binary32, a round with
                // an entry near it gone through again (256k: 84 -> 77 us)
                const float inv_h = g.inv_hi_f;   // (scaled r^2: index only)
                const float kmax = (float)(nint - 1);
                const float4 *trho = g.pkf_rho + (size_t)sp.pairs[0].jloc * nint;
                const float3 h3 = make_float3(g.cellh_s[0], g.cellh_s[1], g.cellh_s[2]);
                const float rc2f = sp.pf[0][2], band = 5e-6f * rc2f;
                const double rc2 = sp.pairs[0].p[2];
                Acc32<1> ac;
                auto value = [&](float r2) {
                    float b;
                    const int ir2 = table_index(r2 * inv_h, kmax, b);
                    return spl_val(trho[ir2], b);
                };
                auto round = [&](int4 e4, int left, auto last) {
                    constexpr bool LAST = decltype(last)::value;
                    const int e[4] = {e4.x, (LAST && left < 2) ? e4.x : e4.y, (LAST && left < 3) ? e4.x : e4.z,
                                      LAST ? e4.x : e4.w};
                    float4 x[4];
                    for (int w = 0; w < 4; w++) x[w] = g.xl[e[w] & SLOT_MASK];
                    float r2[4];
                    for (int w = 0; w < 4; w++)
                    {
                        r2[w] = norm2(rv_steps(xi, x[w], so.steps[(unsigned)e[w] >> SLOT_BITS], h3));
                        if (LAST && w >= left) r2[w] = 4.f * rc2f;
                    }
                    for (int w = 0; w < 4; w++)
                    {
                        const float y = value(r2[w]);
                        ac.part[0] += r2[w] < rc2f ? y : 0.f;
                    }
                    const float near = fminf(fminf(fabsf(r2[0] - rc2f), fabsf(r2[1] - rc2f)),
                                             fminf(fabsf(r2[2] - rc2f), fabsf(r2[3] - rc2f)));
                    if (near <= band)
                        for (int w = 0; w < 4; w++)
                            if (fabsf(r2[w] - rc2f) <= band)
                            {
                                const bool in = geom64_mi(g, g.xd[t], g.xd[e[w] & SLOT_MASK]).r2 < rc2;
                                if (in != (r2[w] < rc2f)) ac.part[0] += in ? value(r2[w]) : -value(r2[w]);
                            }
                    ac.entries(LAST ? left : 4);
                };
                const int cnt = g.nbr_count[t];
                if (cnt <= g.maxnb)
                {
                    const int step = 4 * V;
                    const size_t cap = g.cap;
                    const int4 *col = after_wait<L::free_loads>(reinterpret_cast<const int4 *>(g.nbr)) + t;
                    int k = 4 * v;
                    for (; k + 4 <= cnt; k += step)
                    {
                        if (k + step + 4 <= cnt)
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(col + (size_t)((k + step) >> 2) * cap));
                        round(ld_step<L::free_loads>(col + (size_t)(k >> 2) * cap), 4, std::false_type{});
                    }
                    if (k < cnt) round(ld_step<L::free_loads>(col + (size_t)(k >> 2) * cap), cnt - k, std::true_type{});
                }
                else
                    for_each_slot_overflow<L::one_system>(g, S, so, t, i, v, V, xi, [&](int js, float4 xj, float4 o) {
                        const float r2 = norm2(rv_of(xi, xj, o));
                        bool in = r2 < rc2f;
                        if (fabsf(r2 - rc2f) <= band) in = geom64_mi(g, g.xd[t], g.xd[js]).r2 < rc2;
                        if (in) ac.part[0] += value(r2);
                        ac.entries(1);
                    });
                ac.flush();
                acc_rho = {ac.hi[0], ac.lo[0]};
            }
            else
            {
                const float inv_h = g.inv_hi_f;   // (scaled r^2: index only)
                const float kmax = (float)(nint - 1);
                Acc32<1> ac;
                for_each_slot_pair<L::one_system>(g, S, so, t, i, v, V, xi, [&](int js, float4 xj, float4 o) {
                    if (group >= 0 && g.gslot[js] != group) return;
                    const int pidx = ki * nk + __float_as_int(xj.w);
                    const fmdg_pair_t &pp = sp.pairs[pidx];
                    const float3 rv = rv_lo(so, xi, xj, o);
                    const float r2 = rv.x * rv.x + rv.y * rv.y + rv.z * rv.z;
                    if ((!HYBRID || pp.cat == FMDG_POT_EAM) &&
                        within_cut_skin(g, t, js, r2, sp.pf[pidx][2], pp.p[2]))
                    {
                        float b;
                        const int ir2 = table_index(r2 * inv_h, kmax, b);
                        ac.part[0] += spl_val(g.pkf_rho[(size_t)pp.jloc * nint + ir2], b);
                    }
                    ac.tick();
                });
                ac.flush();
                acc_rho = {ac.hi[0], ac.lo[0]};
            }
            if (L::split_shares && M > 1) part[m][0] = acc_rho;
            else dens[0] = acc_rho;
        }
        if constexpr (L::split_shares)
            if (M > 1) part_tree(part, M, 1, dens);
    }
    step_trigger();
    // binary64 mode: F'(rho) as a double-float, in the w of the slot's row
    // where the rows need no kind (as below in binary32)
    auto store_fp = [&](int t, float2 fp) {
        if (LEAN)
        {
            float *w = reinterpret_cast<float *>(g.xr + 2 * (size_t)t);
            w[3] = fp.x;
            w[7] = fp.y;
        }
        else
            g.fpdf[t] = fp;
    };
    // embedding, one thread per slot
    const double rho = group_value(dens[0], gl);
    const int t = slot_of_thread(g, bx, gl);
    const int i = (t >= 0) ? g.pos[t] : -1;
    if (i >= 0)
    {
        const int ki = LEAN ? 0 : (int)S.kind[i];
        if (is_active(t, ki))
        {
            const int ei = sp.elem[ki];
            const double qr = rho * g.inv_drho;
            int irho = (int)qr;
            if (irho >= g.Nrho - 1 || irho < 0)
            {
                atomic_or_err(dyn, FMDG_ERRBIT_RHO_RANGE);
                irho = irho < 0 ? 0 : g.Nrho - 2;
            }
            const int nrint = g.Nrho - 1;
            double fp;
            if (!MIXED)
            {
                const double b = qr - irho;
                const double4_32a tf = g.pk_F[(size_t)ei * nrint + irho];
                fp = spl_der(tf, b, g.inv_drho);
                acc[0] = spl_val(tf, b);
            }
            else
            {
                const float b = (float)(qr - irho);
                const float4 tf = g.pkf_F[(size_t)ei * nrint + irho];
                const float f32 = spl_der(tf, b, (float)g.inv_drho);
                g.fpb[t] = f32;
                // lean (one kind: the kind bits are unused): F'(rho) also
                // rides in the w of the slot's list position, so the force
                // walk reads it with the neighbour's position (one gather
                // per pair instead of two); the next step start rewrites w
                if (LEAN) reinterpret_cast<float *>(g.xl + t)[3] = f32;
                fp = (double)f32;
                acc[0] = (double)spl_val(tf, b);
            }
            g.vaream[i] = fp;
            g.fpd[t] = fp;
            if (!MIXED) store_fp(t, df_split(fp));
        }
        else
        {
            g.vaream[i] = 0.0;
            g.fpd[t] = 0.0;
            g.fpb[t] = 0.f;
            if (MIXED && LEAN) reinterpret_cast<float *>(g.xl + t)[3] = 0.f;
            if (!MIXED) store_fp(t, make_float2(0.f, 0.f));
        }
    }
    if (rec == REC_FULL && loc_thermo(loc, g)) block_reduce_store<1>(acc, g.partials + (size_t)nb * 8 + bx, blockDim.x >> gl);
}

// Pair forces + velocity-Verlet finish step (src/integrators.c:94-126) and
// the thermo record, 2^lane_log lanes per slot (shares and lanes, above);
// the forces are stored in the current order for the next start step.  LEAN
// (one kind, no group; the density pass of the same step ran LEAN too): pair
// parameters in registers, no per-entry kind or group lookups; in binary32
// hardware exp2 / rsqrt / rcp approximations.
template <class L, int CAT, bool MIXED, bool LEAN>
__global__ void __launch_bounds__(L::max_threads, !MIXED ? L::df_min_blocks : (LEAN ? L::lean_min_blocks : L::min_blocks)) k_force_skin(__grid_constant__ const L loc, int finish, int rec)
{
    int bx, nb;
    const Geo &g = loc_geo(loc, bx, nb);
    const int group = g.st.group;
    const double dt = g.st.dt;
    __shared__ SmemPotT<!MIXED, LEAN> sp;
    __shared__ SkinOffT<MIXED && !LEAN> so;   // (lean binary32: no remainders, exact on a cubic grid)
    load_pot<false>(g, sp, skin_params(g));
    load_offsets(g, so);
    step_wait();        // (the tables above were set up before any step)
    if (loc_idle(loc, g)) return;
    Dyn *dyn = g.dyn;
    const Side S = g.side[dyn->cur];
    const int cap = g.cap;
    const int gl = L::one_lane ? 0 : g.lane_log, lane = threadIdx.x & ((1 << gl) - 1);
    const bool thermo = rec == REC_FULL && loc_thermo(loc, g);
    const bool sums = thermo || (L::one_system && rec == REC_LAMBDA);      // kinetic sums
    // pe, m v^2, m v (3), count, pair virial
    double acc[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    // this lane's shares of the force (3), energy and virial
    dfl sum[5] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
    {
        const int t = (bx * blockDim.x + threadIdx.x) >> gl;
        const int i = (t < cap) ? g.pos[t] : -1;
        float4 xi = i >= 0 ? g.xl[t] : make_float4(0.f, 0.f, 0.f, 0.f);
        const int ki = LEAN ? 0 : __float_as_int(xi.w);   // (lean EAM: w holds F'(rho))
        const int nk = g.nkinds;
        const int nint = g.Nr2 - 1;
        const size_t ne = g.nelem;
        const bool on = i >= 0 && (group < 0 || g.gslot[t] == group);
        const int V = L::one_lane ? 1 : 1 << g.share_log, M = L::split_shares ? V >> gl : 1;
        dfl part[L::split_shares ? MAX_SHARES : 1][5];
        for (int m = 0; m < M; m++)
        {
            const int v = lane + (m << gl);
            for (int q = 0; q < 5; q++) sum[q] = {0.f, 0.f};
            if constexpr (!MIXED)
            {
                // double-float pair arithmetic (fmdg_df.cuh, df_pair)
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 ih = on ? g.xr[2 * (size_t)t] : zero, il = on ? g.xr[2 * (size_t)t + 1] : zero;
                const float3 h3 = make_float3(g.cellh_s[0], g.cellh_s[1], g.cellh_s[2]);
                const float3 hl3 = make_float3(g.cellh_slo[0], g.cellh_slo[1], g.cellh_slo[2]);
                dfl fpi = {0.f, 0.f};
                if (LEAN) fpi = {ih.w, il.w};
                else if ((CAT == CAT_EAM || CAT == CAT_HYBRID) && on) fpi = df_of(g.fpdf[t]);
                const dfl inv_h = df_of(g.inv_h_df);
                const float kmax = (float)(nint - 1);
                auto pair = [&](auto with_e, int js, float w, auto &&geom, auto &&fpj) {
                    if (!LEAN && group >= 0 && g.gslot[js] != group) return;
                    const int pidx = LEAN ? 0 : ki * nk + __float_as_int(w);
                    const fmdg_pair_t &pp = sp.pairs[pidx];
                    const int cat = (CAT == CAT_HYBRID) ? pp.cat : CAT;
                    const int rci = (cat == FMDG_POT_MORSE) ? 3 : 2;
                    const GeomDF p = geom();
                    if (!within_cut_df_mi(g, t, js, p.r2, sp.pf[pidx][rci], pp.p[rci])) return;
                    dfl fa, eh;
                    df_pair(g, sp, pidx, pp, cat, p, fpi, inv_h, kmax, nint, ne, fpj, fa, eh);
                    for (int d = 0; d < 3; d++) sum[d] = df_add(sum[d], df_mul(fa, p.rv[d]));
                    if constexpr (decltype(with_e)::value)
                    {
                        sum[3] = df_add(sum[3], eh);
                        sum[4] = df_add(sum[4], df_mul(fa, p.r2));     // rv . (fa rv), both sides of the pair
                    }
                };
                // F'(rho_j): in the row, or (kinds in the rows, overflow) in a table
                auto listed = [&](auto with_e) {
                    return [&, with_e](int js, float4 jh, float4 jl, unsigned w) {
                        pair(with_e, js, jh.w, [&]() { return skin_geom_df(ih, il, jh, jl, w, h3, hl3); },
                             [&]() { return LEAN ? dfl{jh.w, jl.w} : df_of(g.fpdf[js]); });
                    };
                };
                const int cnt = on ? g.nbr_count[t] : 0;
                const int m_in = (CAT == CAT_EAM) ? (on ? g.nbc_count[(size_t)t * V + v] : 0)
                                                  : prune_share(g, so, cnt <= g.maxnb ? cnt : 0, t, v, V, ih);
                if (thermo) for_each_pruned(g, so, m_in, t, v, V, listed(std::true_type{}));
                else for_each_pruned(g, so, m_in, t, v, V, listed(std::false_type{}));
                if (cnt > g.maxnb)
                    for_each_slot_overflow<L::one_system>(g, S, so, t, i, v, V, xi, [&](int js, float4 xj, float4) {
                        pair(std::true_type{}, js, xj.w, [&]() { return geom_df_of64(geom64_mi(g, g.xd[t], g.xd[js])); },
                             [&]() {
                                 const float4 *r = g.xr + 2 * (size_t)js;
                                 return LEAN ? dfl{r[0].w, r[1].w} : df_of(g.fpdf[js]);
                             });
                    });
            }
            else if (!on)
                ;
            else if constexpr (LEAN)
            {
                const float4 pq = make_float4(sp.pf[0][0], sp.pf[0][1], sp.pf[0][2], sp.pf[0][3]);
                const float rc2f = (CAT == CAT_MORSE) ? pq.w : pq.z;
                const double rc2 = (CAT == CAT_MORSE) ? sp.pairs[0].p[3] : sp.pairs[0].p[2];
                // scaled frame (Geo::xs; pq holds scaled parameters): real
                // force factors from scaled geometry.  Morse: 2^((r0' - r')
                // alpha' log2 e) with alpha' = alpha / xs, r0' = r0 xs, factor
                // 2 alpha D0 xs = 2 alpha' D0 xs^2; LJ: 12 eps4 xs^2 / r'^2
                const float xs2 = g.xs2_f;
                const float m_c1 = pq.y * 1.44269504f, m_c2 = 2.f * pq.y * pq.x * xs2;
                const float lj_c = 12.f * pq.x * xs2;
                const float fpi = (CAT == CAT_EAM) ? g.fpb[t] : 0.f;
                const float inv_h = g.inv_h_df.x;         // derivatives with respect to the real r^2
                const float inv_hi = g.inv_hi_f;  // table index of the scaled r^2
                const float kmax = (float)(nint - 1);
                const int ee = sp.pairs[0].iloc;
                const float4 *tpr = g.pkf_pr + (size_t)ee * nint * 2;
                // LJ / Morse pair: force factor and half energy (explicitly
                // rounded operations in the forces: the walks with and without
                // the energy give the same bits)
                auto pair_lm = [&](float r2, float &fa, float &e) {
                    if (CAT == CAT_LJ)
                    {
                        const float inv_r2 = rcp_approx(r2);
                        const float s2 = __fmul_rn(pq.y, inv_r2);
                        const float s6 = __fmul_rn(__fmul_rn(s2, s2), s2);
                        fa = __fmul_rn(__fmul_rn(lj_c, inv_r2), __fmul_rn(s6, __fsub_rn(s6, 0.5f)));
                        e = 0.5f * (pq.x * (s6 * s6 - s6));
                    }
                    else
                    {
                        const float inv_r = rsqrt_approx(r2);
                        // (r0 - r in one rounding: a rounded r would cost
                        // up to 3e-7 of the exponential)
                        const float e1 = ex2_approx(__fmul_rn(__fmaf_rn(-r2, inv_r, pq.z), m_c1));
                        fa = __fmul_rn(__fmul_rn(m_c2, inv_r), __fmaf_rn(e1, e1, -e1));
                        e = 0.5f * (pq.x * (e1 * e1 - 2.f * e1));
                    }
                };
                // E: the walk sums the energy, W: the pair virial (rv . F =
                // fa r^2); both on steps that form the thermo record only
                auto walk = [&](auto with_e, auto with_v) {
                    constexpr bool E = decltype(with_e)::value;
                    constexpr bool W = decltype(with_v)::value;
                    constexpr int NA = W ? 5 : (E ? 4 : 3);
                    Acc32<NA> ac;
                    // adds a pair's force (times sign), energy and virial
                    auto add = [&](float sign, float3 rv, float r2, float fpj) {
                        float fa, e;
                        if constexpr (CAT == CAT_EAM)
                        {
                            float b;
                            const int ir2 = table_index(r2 * inv_hi, kmax, b);
                            float4 tph, trh;
                            ld_row32(tpr + 2 * ir2, tph, trh);
                            const float phi_d = spl_der_rn(tph, b, inv_h);
                            const float rho_d = spl_der_rn(trh, b, inv_h);
                            fa = __fmul_rn(-2.f, __fmaf_rn(__fadd_rn(fpi, fpj), rho_d, phi_d));
                            if constexpr (E) e = 0.5f * spl_val(tph, b);
                        }
                        else
                            pair_lm(r2, fa, e);
                        fa = __fmul_rn(fa, sign);
                        ac.part[0] = __fmaf_rn(fa, rv.x, ac.part[0]);
                        ac.part[1] = __fmaf_rn(fa, rv.y, ac.part[1]);
                        ac.part[2] = __fmaf_rn(fa, rv.z, ac.part[2]);
                        if constexpr (E) ac.part[3] += sign * e;
                        if constexpr (W) ac.part[NA - 1] += fa * r2;
                    };
                    // A round of four entries (LAST: the first `left` of
                    // them).  The cutoff is decided in binary32; when an
                    // entry of the round lies within `band` of it, the round
                    // is gone through again and an entry that binary64 decides
                    // otherwise is added or taken back: one test a round
                    // instead of several instructions an entry.  (Error of the
                    // binary32 r^2: coordinates and offsets below 2 rc, three
                    // roundings each of 1.2e-7 rc and the subtractions' own:
                    // 5e-7 rc a component, 2e-6 rc^2 at most.)  L1 throughput
                    // and issue bound the walk;
                    // against a flag per entry and a second walk, without the
                    // record: EAM 256k 142 -> 112 us, Morse 512k 256 -> 250,
                    // LJ 32k 18.0 -> 16.5.
                    const float band = 5e-6f * rc2f;
                    const float3 h3 = make_float3(g.cellh_s[0], g.cellh_s[1], g.cellh_s[2]);
                    auto round = [&](int4 e4, int left, auto last) {
                        constexpr bool LAST = decltype(last)::value;
                        const int e[4] = {e4.x, (LAST && left < 2) ? e4.x : e4.y, (LAST && left < 3) ? e4.x : e4.z,
                                          LAST ? e4.x : e4.w};
                        float4 x[4];
                        for (int w = 0; w < 4; w++) x[w] = g.xl[e[w] & SLOT_MASK];
                        float3 rv[4];
                        float r2[4];
                        for (int w = 0; w < 4; w++)
                        {
                            rv[w] = rv_steps(xi, x[w], so.steps[(unsigned)e[w] >> SLOT_BITS], h3);
                            r2[w] = norm2(rv[w]);
                            if (LAST && w >= left) r2[w] = 4.f * rc2f;
                        }
                        for (int w = 0; w < 4; w++)
                        {
                            if constexpr (CAT == CAT_EAM)
                            {
                                if (r2[w] < rc2f) add(1.f, rv[w], r2[w], x[w].w);
                            }
                            else
                            {
                                float fa, e;
                                pair_lm(r2[w], fa, e);
                                const bool in = r2[w] < rc2f;
                                fa = in ? fa : 0.f;
                                ac.part[0] = __fmaf_rn(fa, rv[w].x, ac.part[0]);
                                ac.part[1] = __fmaf_rn(fa, rv[w].y, ac.part[1]);
                                ac.part[2] = __fmaf_rn(fa, rv[w].z, ac.part[2]);
                                if constexpr (E) ac.part[3] += in ? e : 0.f;
                                if constexpr (W) ac.part[NA - 1] += fa * r2[w];
                            }
                        }
                        const float near = fminf(fminf(fabsf(r2[0] - rc2f), fabsf(r2[1] - rc2f)),
                                                 fminf(fabsf(r2[2] - rc2f), fabsf(r2[3] - rc2f)));
                        if (near <= band)
                        {
                            for (int w = 0; w < 4; w++)
                                if (fabsf(r2[w] - rc2f) <= band)
                                {
                                    const bool in = geom64_mi(g, g.xd[t], g.xd[e[w] & SLOT_MASK]).r2 < rc2;
                                    if (in != (r2[w] < rc2f)) add(in ? 1.f : -1.f, rv[w], r2[w], x[w].w);
                                }
                        }
                        ac.entries(LAST ? left : 4);
                    };
                    const int cnt = g.nbr_count[t];
                    if (cnt <= g.maxnb)
                    {
                        constexpr bool PF = CAT != CAT_EAM;      // prefetch of the next list row
                        const int step = 4 * V;
                        const int4 *col = after_wait<L::free_loads>(reinterpret_cast<const int4 *>(g.nbr)) + t;
                        int k = 4 * v;
                        for (; k + 4 <= cnt; k += step)
                        {
                            if (PF && k + step + 4 <= cnt)
                                asm volatile("prefetch.global.L1 [%0];" ::"l"(col + (size_t)((k + step) >> 2) * cap));
                            round(ld_step<L::free_loads>(col + (size_t)(k >> 2) * cap), 4, std::false_type{});
                        }
                        if (k < cnt) round(ld_step<L::free_loads>(col + (size_t)(k >> 2) * cap), cnt - k, std::true_type{});
                    }
                    else
                        for_each_slot_overflow<L::one_system>(g, S, so, t, i, v, V, xi, [&](int js, float4 xj, float4 o) {
                            const float3 rv = rv_of(xi, xj, o);
                            const float r2 = norm2(rv);
                            bool in = r2 < rc2f;
                            if (fabsf(r2 - rc2f) <= band) in = geom64_mi(g, g.xd[t], g.xd[js]).r2 < rc2;
                            // (xj.w: kind bits here)
                            if (in) add(1.f, rv, r2, CAT == CAT_EAM ? g.fpb[js] : 0.f);
                            ac.entries(1);
                        });
                    ac.flush();
                    for (int d = 0; d < 3; d++) sum[d] = {ac.hi[d], ac.lo[d]};
                    if constexpr (E) sum[3] = {ac.hi[3], ac.lo[3]};
                    if constexpr (W) sum[4] = {ac.hi[NA - 1], ac.lo[NA - 1]};
                };
                if (thermo)
                    walk(std::true_type{}, std::true_type{});
                else
                    walk(std::false_type{}, std::false_type{});
            }
            else
            {
                const float fpi = (CAT == CAT_EAM || CAT == CAT_HYBRID) ? g.fpb[t] : 0.f;
                const float inv_h = g.inv_h_df.x;         // derivatives with respect to the real r^2
                const float inv_hi = g.inv_hi_f;  // table index of the scaled r^2
                const float kmax = (float)(nint - 1);
                const float xs2 = g.xs2_f;
                Acc32<5> ac;
                for_each_slot_pair<L::one_system>(g, S, so, t, i, v, V, xi, [&](int js, float4 xj, float4 o) {
                    if (group >= 0 && g.gslot[js] != group) return;
                    const int pidx = ki * nk + __float_as_int(xj.w);
                    const fmdg_pair_t &pp = sp.pairs[pidx];
                    const int cat = (CAT == CAT_HYBRID) ? pp.cat : CAT;
                    const float3 rv = rv_lo(so, xi, xj, o);
                    const float r2 = rv.x * rv.x + rv.y * rv.y + rv.z * rv.z;
                    if (cat == FMDG_POT_LJ)
                    {
                        if (within_cut_skin(g, t, js, r2, sp.pf[pidx][2], pp.p[2]))
                        {
                            float fa, e;
                            lj_pair(r2, sp.pf[pidx][0], sp.pf[pidx][1], fa, e);
                            fa *= xs2;         // the real force factor (scaled frame)
                            ac.part[0] += rv.x * fa;
                            ac.part[1] += rv.y * fa;
                            ac.part[2] += rv.z * fa;
                            ac.part[3] += e;
                            ac.part[4] += fa * r2;
                        }
                    }
                    else if (cat == FMDG_POT_MORSE)
                    {
                        if (within_cut_skin(g, t, js, r2, sp.pf[pidx][3], pp.p[3]))
                        {
                            float fa, e;
                            morse_pair(r2, sp.pf[pidx][0], sp.pf[pidx][1], sp.pf[pidx][2], fa, e);
                            fa *= xs2;         // the real force factor (scaled frame)
                            ac.part[0] += fa * rv.x;
                            ac.part[1] += fa * rv.y;
                            ac.part[2] += fa * rv.z;
                            ac.part[3] += e;
                            ac.part[4] += fa * r2;
                        }
                    }
                    else if (cat == FMDG_POT_EAM)
                    {
                        if (within_cut_skin(g, t, js, r2, sp.pf[pidx][2], pp.p[2]))
                        {
                            float b;
                            const int ir2 = table_index(r2 * inv_hi, kmax, b);
                            const int ei = pp.iloc, ej = pp.jloc;
                            const float4 tph = g.pkf_phi[((size_t)ei * ne + ej) * nint + ir2];
                            const float phi_d = spl_der(tph, b, inv_h);
                            const float rho_ip = spl_der(g.pkf_rho[(size_t)ei * nint + ir2], b, inv_h);
                            const float rho_jp = (ei == ej) ? rho_ip
                                               : spl_der(g.pkf_rho[(size_t)ej * nint + ir2], b, inv_h);
                            const float mag = 2.f * (fpi * rho_jp + g.fpb[js] * rho_ip + phi_d);
                            ac.part[0] -= mag * rv.x;
                            ac.part[1] -= mag * rv.y;
                            ac.part[2] -= mag * rv.z;
                            ac.part[3] += 0.5f * spl_val(tph, b);
                            ac.part[4] -= mag * r2;
                        }
                    }
                    ac.tick();
                });
                ac.flush();
                for (int q = 0; q < 5; q++) sum[q] = {ac.hi[q], ac.lo[q]};
            }
            if (L::split_shares && M > 1)
            {
                for (int q = 0; q < 3; q++) part[m][q] = sum[q];
                if (thermo)
                    for (int q = 3; q < 5; q++) part[m][q] = sum[q];
            }
        }
        if constexpr (L::split_shares)
            if (M > 1) part_tree(part, M, thermo ? 5 : 3, sum);
    }
    step_trigger();
    // the group's sums, then one thread per slot
    double fin[5];
    group_forces(sum, gl, thermo, fin);
    const int t = slot_of_thread(g, bx, gl);
    const int i = (t >= 0) ? g.pos[t] : -1;
    if (i >= 0)
    {
        const int ki = LEAN ? 0 : (int)S.kind[i];
        const bool active = (group < 0 || g.gslot[t] == group);
        double f[3] = {fin[0], fin[1], fin[2]};
        double pe = fin[3], vir = 0.5 * fin[4];
        if (MIXED)
        {
            // binary32 pairs were summed in the scaled frame (Geo::xs): the
            // real force is the sum over xs, the real virial over xs^2
            for (int d = 0; d < 3; d++) f[d] *= g.inv_xs;
            vir *= g.inv_xs * g.inv_xs;
        }
        if (active && g.ttm_on)
        {
            // TTM friction (src/forces.c:292-330, 1-D): F_z += xi m (v_z - vcm_z)
            const double time = dyn->time, hdt = dyn->dt / 2.0;
            if ((time >= g.ttm_start - hdt) && ((time < g.ttm_stop + hdt) || g.ttm_stop < g.ttm_start))
            {
                const double z = S.x[2 * (size_t)cap + i];
                const double q = z * g.ttm_inv_tcellh_z;
                const double r = rint(q);
                int it = (fabs(q - r) <= 1e-9 * fmax(1.0, fabs(q))) ? (int)__ddiv_rn(z, g.ttm_tcellh_z) : (int)q;
                it += g.ttm_g2l_z;
                if (it >= 0 && it < g.ttm_nz)
                    f[2] += g.ttm_xi[it] * sp.mass[ki] * (S.v[2 * (size_t)cap + i] - g.ttm_vcm[3 * it + 2]);
                else
                    atomic_or_err(dyn, FMDG_ERRBIT_TTM);
            }
        }
        for (int d = 0; d < 3; d++) g.F[(size_t)d * cap + i] = f[d];
        acc[0] = pe;
        acc[6] = vir;
        if (active)
        {
            const double m = sp.mass[ki];
            double v[3] = {S.v[i], S.v[cap + i], S.v[2 * (size_t)cap + i]};
            if (finish)
            {
                const double coef = sp.hk[ki];   // dt * 0.5 / m, as the reference forms it
                for (int d = 0; d < 3; d++)
                {
                    v[d] = __dadd_rn(v[d], __dmul_rn(coef, f[d]));
                    S.v[(size_t)d * cap + i] = v[d];
                }
            }
            if (sums)
            {
                acc[1] = m * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
                acc[2] = m * v[0];
                acc[3] = m * v[1];
                acc[4] = m * v[2];
                acc[5] = 1.0;
            }
        }
    }
    __shared__ double blk[7];
    __shared__ unsigned ticket;
    if (sums) block_reduce_store<7>(acc, blk, blockDim.x >> gl);
    else if (L::one_system)
        return;     // (nothing for the last block to do)
    if (threadIdx.x == 0)
    {
        if (sums)
            for (int k = 0; k < 7; k++) g.partials[(size_t)k * nb + bx] = blk[k];
        __threadfence();
        ticket = atomicAdd(&dyn->blocks_done, 1u);
    }
    __syncthreads();
    if (ticket == (unsigned)nb - 1)
    {
        __threadfence();
        if (thermo) final_reduce(g, nb, 0, g.has_eam, g.st.thermostat, dt, g.st.tau, g.st.T0);
        else if (sums) final_lambda(g, nb, dt, g.st.tau, g.st.T0);
        if (threadIdx.x == 0)
        {
            dyn->blocks_done = 0;
            if (finish && dyn->steps_left > 0) dyn->steps_left--;
        }
    }
}

// dynamic shared bytes of slot_of_thread for NV values per slot
size_t stage_bytes(const LocOne &L, int blk, int nv) { return L.g.lane_log ? (size_t)nv * 8 * (blk >> L.g.lane_log) : 0; }
size_t stage_bytes(const LocPack &L, int blk, int nv)
{
    size_t most = 0;
    for (int k = 0; k < L.nsys; k++)
        if (const int gl = L.geos[k].lane_log) most = std::max(most, (size_t)nv * 8 * (blk >> gl));
    return most;
}

template <class L, bool MIXED>
void launch_force_skin(const L &loc, int cats, int finish, int rec, int nb, int blk, cudaStream_t st, bool lean, bool overlap)
{
    const size_t sh = stage_bytes(loc, blk, 5);
    const int ncat = __builtin_popcount(cats);
    if (ncat > 1) fmdg_launch(k_force_skin<L, CAT_HYBRID, MIXED, false>, nb, blk, sh, st, overlap, 1, loc, finish, rec);
    else if (lean)
    {
        if (cats == (1 << FMDG_POT_LJ)) fmdg_launch(k_force_skin<L, CAT_LJ, MIXED, true>, nb, blk, sh, st, overlap, 1, loc, finish, rec);
        else if (cats == (1 << FMDG_POT_MORSE)) fmdg_launch(k_force_skin<L, CAT_MORSE, MIXED, true>, nb, blk, sh, st, overlap, 1, loc, finish, rec);
        else fmdg_launch(k_force_skin<L, CAT_EAM, MIXED, true>, nb, blk, sh, st, overlap, 1, loc, finish, rec);
    }
    else if (cats == (1 << FMDG_POT_LJ)) fmdg_launch(k_force_skin<L, CAT_LJ, MIXED, false>, nb, blk, sh, st, overlap, 1, loc, finish, rec);
    else if (cats == (1 << FMDG_POT_MORSE)) fmdg_launch(k_force_skin<L, CAT_MORSE, MIXED, false>, nb, blk, sh, st, overlap, 1, loc, finish, rec);
    else fmdg_launch(k_force_skin<L, CAT_EAM, MIXED, false>, nb, blk, sh, st, overlap, 1, loc, finish, rec);
}

template <class L>
void launch_density_skin(const L &loc, bool mixed, bool hyb, int rec, int nb, int blk, cudaStream_t st, bool lean, bool overlap)
{
    const size_t sh = stage_bytes(loc, blk, 1);
    if (mixed)
    {
        if (hyb) fmdg_launch(k_density_skin<L, true, true, false>, nb, blk, sh, st, overlap, 1, loc, rec);
        else if (lean) fmdg_launch(k_density_skin<L, true, false, true>, nb, blk, sh, st, overlap, 1, loc, rec);
        else fmdg_launch(k_density_skin<L, true, false, false>, nb, blk, sh, st, overlap, 1, loc, rec);
    }
    else
    {
        if (hyb) fmdg_launch(k_density_skin<L, false, true, false>, nb, blk, sh, st, overlap, 1, loc, rec);
        else if (lean) fmdg_launch(k_density_skin<L, false, false, true>, nb, blk, sh, st, overlap, 1, loc, rec);
        else fmdg_launch(k_density_skin<L, false, false, false>, nb, blk, sh, st, overlap, 1, loc, rec);
    }
}

} // namespace

int fmdg_pack_launch_start(const fmdg_pack_launch &P)
{
    const cudaError_t e = fmdg_launch(k_skin_start<LocPack>, P.la.bstart[P.nsys], 128, 0, P.stream, P.overlap, 1, P.la);
    if (e != cudaSuccess) return -fmdg_fail("pack start", e);
    return 1;
}

// phases: bit 0 list (re)build, bit 1 EAM density, bit 2
// pair forces + finish step (all three for a step).  Returns the kernels
// launched, or minus a status.
int fmdg_pack_launch_forces(const fmdg_pack_launch &P, int phases)
{
    cudaStream_t st = P.stream;
    const int nab = P.la.bstart[P.nsys], nfb = P.lf.bstart[P.nsys];
    int n = 0;
    if (phases & 1)
    {
        fmdg_launch(k_nlist_skin<LocPack>, nab, 128, 0, st, P.overlap, 1, P.la);
        n++;
    }
    if ((phases & 2) && (P.cats & (1 << FMDG_POT_EAM)))
    {
        if (P.shares) launch_density_skin(LocPackShares{P.lf}, P.mixed != 0, __builtin_popcount(P.cats) > 1, REC_FULL, nfb, P.fblk, st, P.lean != 0, P.overlap);
        else launch_density_skin(P.lf, P.mixed != 0, __builtin_popcount(P.cats) > 1, REC_FULL, nfb, P.fblk, st, P.lean != 0, P.overlap);
        n++;
    }
    if (phases & 4)
    {
        if (P.shares)
        {
            const LocPackShares L{P.lf};
            if (P.mixed) launch_force_skin<LocPackShares, true>(L, P.cats, 1, REC_FULL, nfb, P.fblk, st, P.lean != 0, P.overlap);
            else launch_force_skin<LocPackShares, false>(L, P.cats, 1, REC_FULL, nfb, P.fblk, st, P.lean != 0, P.overlap);
        }
        else if (P.mixed) launch_force_skin<LocPack, true>(P.lf, P.cats, 1, REC_FULL, nfb, P.fblk, st, P.lean != 0, P.overlap);
        else launch_force_skin<LocPack, false>(P.lf, P.cats, 1, REC_FULL, nfb, P.fblk, st, P.lean != 0, P.overlap);
        n++;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return -fmdg_fail("pack forces", e);
    return n;
}

// The single-system path on a skin list (fmdg_launch_nlist/density/
// pair_forces dispatch here when the system has one): slot tables + list
// (re)build; EAM density; pair forces (+ finish step).
// prepped: a refresh has just written the per-atom tables.
int fmdg_skin_launch_nlist(fmdg_sys_t *s, bool prepped)
{
    const LocOne L{s->g};
    if (!prepped)
    {
        k_prep_skin<<<fmdg_grid(s->g.cap, 128), 128, 0, s->stream>>>(L);
        s->launches++;
    }
    // lanes per slot by size, from build times measured on GB300 (LJ,
    // Morse, EAM jobs of 2k-190k atoms): 16 up to 2^14 slots, 8 up to 2^16,
    // then one thread per slot (enough warps; a group's ballots cost more
    // than they hide).  Groups of 2 or 4 lanes never won: the lanes of
    // different groups in a warp diverge and serialise.
    const int cap = s->g.cap;
    int G = s->build_lanes;
    if (G == 0) G = cap <= (1 << 14) ? 16 : (cap <= (1 << 16) ? 8 : 1);
    const int nbg = fmdg_grid(cap > 0 ? cap * G : 1, 128);
    switch (G)
    {
    case 2: fmdg_launch(k_nlist_skin_grp<2>, nbg, 128, 0, s->stream, s->overlap, 1, L); break;
    case 4: fmdg_launch(k_nlist_skin_grp<4>, nbg, 128, 0, s->stream, s->overlap, 1, L); break;
    case 8: fmdg_launch(k_nlist_skin_grp<8>, nbg, 128, 0, s->stream, s->overlap, 1, L); break;
    case 16: fmdg_launch(k_nlist_skin_grp<16>, nbg, 128, 0, s->stream, s->overlap, 1, L); break;
    case 32: fmdg_launch(k_nlist_skin_grp<32>, nbg, 128, 0, s->stream, s->overlap, 1, L); break;
    default: fmdg_launch(k_nlist_skin<LocOne>, nbg, 128, 0, s->stream, s->overlap, 1, L); break;
    }
    s->launches++;
    FMDG_CK(cudaGetLastError());
    return FMDG_OK;
}

// one kind and every atom in the step's group: the lean kernels
static bool lean_system(const fmdg_sys_t *s) { return s->nkinds == 1 && s->g.st.group < 0; }

int fmdg_skin_launch_density(fmdg_sys_t *s)
{
    launch_density_skin(LocOne{s->g}, s->g.prec == FMDG_PREC_MIXED, __builtin_popcount(s->cats) > 1,
                        s->rec, fmdg_force_blocks(s), s->fblk, s->stream, lean_system(s), s->overlap);
    s->launches++;
    FMDG_CK(cudaGetLastError());
    return FMDG_OK;
}

int fmdg_skin_launch_pair_forces(fmdg_sys_t *s, int finish)
{
    const LocOne L{s->g};
    const int nb = fmdg_force_blocks(s);
    if (s->g.prec == FMDG_PREC_MIXED)
        launch_force_skin<LocOne, true>(L, s->cats, finish, s->rec, nb, s->fblk, s->stream, lean_system(s), s->overlap);
    else launch_force_skin<LocOne, false>(L, s->cats, finish, s->rec, nb, s->fblk, s->stream, lean_system(s), s->overlap);
    s->launches++;
    FMDG_CK(cudaGetLastError());
    return FMDG_OK;
}
