// Cell-list refresh on the GPU with the reference's cell assignment and
// in-cell atom order.
//
// Reference behaviour being reproduced (FMD 0.4.0, one subdomain):
//  * src/misc.c:268-308 `_fmd_refreshGrid`: interior cells are visited in
//    storage order; inside a cell, atom i is re-binned with
//    floor(x/cellh)+1 (local index incl. the one-cell ghost margin); a
//    departing atom is appended to its destination cell and removed from
//    its source by swap-with-last (src/cell.c:151-160, src/cell.h:84-95), so
//    the atom moved into slot i is examined next.
//  * src/md-ghost.c:827-869 `_fmd_particles_migrate`: for d = 0,1,2, the
//    lower ghost layer then the upper one hand their whole lists (appended,
//    x[d] -/+ l[d]) to the opposite interior layer (periodic) or are
//    discarded (open boundary).
//
// Parallel restatement.  Destinations do not depend on order, so they are
// computed per atom first.  The order then follows from three facts:
//  (1) a cell's departure sequence depends only on its own list and on the
//      NUMBER A of atoms that arrived from lower-index cells before it was
//      visited (arrivals never depart again) -- one warp per cell replays
//      the swap-remove walk with A placeholder tokens in O(1) state, because
//      only the scan position can hold a moved element;
//  (2) arrivals into a cell D are ordered by (source cell, departure rank);
//      the first A of them fill the placeholder slots, the rest are appended;
//  (3) atoms that passed through ghost cells arrive after all interior
//      arrivals, ordered by the pass of their last hop, then by their
//      position in that ghost cell's list, which is itself (direct arrivals
//      by (source, rank)) followed by earlier-pass arrivals -- a fixed-width
//      key of the pass sequence read from the last hop backwards.
// Each destination cell sorts its (few) arrivals by that key, after which
// every atom knows its new index and one scatter writes the next side.
//
// Kernels.  A single system of more than CLUSTER_ATOMS atoms runs the phases
// as grid kernels (k_bin_classify, k_bin_scan, k_bin_cells, k_bin_arrivals,
// k_bin_place).  A smaller one runs all of them in one kernel: one cluster of
// blocks, a cluster barrier between the phases (k_refresh_cluster) -- launches
// and their gaps were most of a small system's step.  Packed systems refresh
// on the steps that rebuild their list only, on a cluster each, or, in packs
// of systems above PACK_CLUSTER_ATOMS, by grid kernels (k_pack_*).
#include <cooperative_groups.h>

#include "fmdg_perdev.h"
#include "fmdg_prep.cuh"

namespace cg = cooperative_groups;

namespace {

// largest system of the cluster kernel: 4000 atoms refresh in 12 us against
// 24 for the separate kernels, 32 000 atoms in 61 (eight blocks) against 21
constexpr int CLUSTER_ATOMS = 1 << 13;
// Largest packed system of the cluster kernel.  Its eight SMs a system refresh
// 186 624 LJ atoms in 390 us, the grid kernels in 150, but each of their five
// launches costs a little on every step, also the nine in ten that refresh
// nothing: fleets of 186 624-atom jobs, us a step with the cluster -> grid
// kernels, LJ 479 -> 438, EAM 939 -> 911, Morse 734 -> 706; sixteen LJ jobs of
// 32 000 atoms 285 -> 279 but Morse 393 -> 400; 2048 jobs of 500 to 200 000
// atoms (1.762e9 atom-steps/s on clusters alone) 1.750e9 with the line at
// 2^14, 1.758e9 at 2^16.
constexpr int PACK_CLUSTER_ATOMS = 1 << 16;
// blocks of a pack's grid kernels: one per SM (two: 0.2 % less in that fleet)
constexpr int PACK_GRID = 152;

__device__ __forceinline__ int cell_flat(const Geo &g, int x, int y, int z)
{
    return z + g.nc[2] * (y + g.nc[1] * x);
}

// Phase 1, one atom: start-of-step update fused with the binning decision.
//  mode VV: src/integrators.c:40-75 (v *= lambda; v += dt*0.5/m*F; x += dt*v)
//  mode SE: src/integrators.c:129-152 (v += dt*F/m; x += dt*v)
// Explicit _rn intrinsics keep the reference's operation order with no
// fused multiply-add, so positions and velocities match bit for bit given
// the same forces.  hk: half kick dt * 0.5 / m per kind, formed on the host
// (set_step_dt) with the reference's operations.
__device__ __forceinline__ void classify_atom(const Geo &g, Dyn *dyn, const Side &S, int i, int mode, const double *hk)
{
    const double dt = g.st.dt;
    const int group = g.st.group, thermostat = g.st.thermostat;
    const int cap = g.cap;

    double x[3], v[3];
    for (int d = 0; d < 3; d++) { x[d] = S.x[d * cap + i]; v[d] = S.v[d * cap + i]; }

    if (mode != FMDG_REFRESH_ONLY && (group < 0 || S.group[i] == group))
    {
        const int k = S.kind[i];
        const double m = g.mass[k];
        if (mode == FMDG_REFRESH_VV)
        {
            const double lam = dyn->lambda;
            const double coef = hk[k];
            for (int d = 0; d < 3; d++)
            {
                double vv = v[d];
                if (thermostat) vv = __dmul_rn(vv, lam);
                vv = __dadd_rn(vv, __dmul_rn(coef, g.F[d * cap + i]));
                v[d] = vv;
                x[d] = __dadd_rn(x[d], __dmul_rn(dt, vv));
            }
        }
        else
        {
            for (int d = 0; d < 3; d++)
            {
                double vv = __dadd_rn(v[d], __ddiv_rn(__dmul_rn(dt, g.F[d * cap + i]), m));
                v[d] = vv;
                x[d] = __dadd_rn(x[d], __dmul_rn(dt, vv));
            }
        }
        for (int d = 0; d < 3; d++) S.v[d * cap + i] = v[d];
    }

    const int c = S.cell_of[i];
    const int cc[3] = { c / (g.nc[1] * g.nc[2]), (c / g.nc[2]) % g.nc[1], c % g.nc[2] };
    int jc[3];
    bool departs = false, outside = false;
    for (int d = 0; d < 3; d++)
    {
        const int q = cell_floor(x[d], g.cellh[d], g.inv_cellh[d], g.inv_cellh_f[d]);
        // local index including the ghost margin (ic_start = 1)
        if (!(q >= -1 && q <= g.nc[d])) outside = true;
        jc[d] = outside ? 0 : q + 1;
        if (jc[d] - 1 != cc[d]) departs = true;
    }
    if (outside)
    {
        // src/misc.c:286-290 raises FMD_ERR_UNEXPECTED_POSITION; the atom is
        // left where it is so no index leaves the grid
        atomic_or_err(dyn, FMDG_ERRBIT_POSITION);
        for (int d = 0; d < 3; d++) S.x[d * cap + i] = x[d];
        g.bdest[i] = -2;
        return;
    }
    if (!departs)
    {
        for (int d = 0; d < 3; d++) S.x[d * cap + i] = x[d];
        g.bdest[i] = -2;
        return;
    }

    // migration path through the ghost margin (src/md-ghost.c:827-869)
    int q[3] = {0, 0, 0};
    int nq = 0;
    bool deleted = false;
    for (int d = 0; d < 3; d++)
    {
        if (jc[d] == 0 || jc[d] == g.nc[d] + 1)
        {
            const bool upper = (jc[d] != 0);
            if (!g.pbc[d]) deleted = true;
            q[nq++] = 1 + 2 * d + (upper ? 1 : 0);
            if (upper) { jc[d] = 1;          x[d] = __dadd_rn(x[d], -g.l[d]); }
            else       { jc[d] = g.nc[d];    x[d] = __dadd_rn(x[d],  g.l[d]); }
        }
    }
    atomicAdd(&g.dep_count[c], 1);
    dyn->any_move = 1;
    if (deleted)
    {
        g.bdest[i] = -1;
        if (g.skin_on)
        {
            // the slot is gone: out of reach of the lists that hold it (a
            // position beyond every cutoff) until the next build leaves it
            // out.  What the branch-free walks form from so large an r^2 may
            // be infinite or not a number (the cubic of a table's interval):
            // they select zero instead of it, and must not multiply by a mask.
            const int t = S.slot[i];
            const float far = 1e8f;
            g.pos[t] = -1;
            g.xl[t] = make_float4(far, far, far, 0.f);
            g.xd[t] = make_double4_32a(1e8, 1e8, 1e8, 0.0);
            if (g.prec == FMDG_PREC_FP64)
            {
                g.xr[2 * (size_t)t] = make_float4(far, far, far, 0.f);
                g.xr[2 * (size_t)t + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        return;
    }
    for (int d = 0; d < 3; d++) S.x[d * cap + i] = x[d];
    const int D = cell_flat(g, jc[0] - 1, jc[1] - 1, jc[2] - 1);
    // key bits: [9] migrated, [8:6] last pass, [5:3] previous, [2:0] first
    int path = 0;
    if (nq > 0)
    {
        path = 1 << 9;
        int shift = 6;
        for (int k = nq - 1; k >= 0; k--, shift -= 3) path |= q[k] << shift;
    }
    g.bpath[i] = path;
    g.bdest[i] = D;
    atomicAdd(&g.arr_total[D], 1);
    if (nq == 0 && c < D) atomicAdd(&g.arr_lower[D], 1);
}

// Exclusive scans over the cells by the blocks of one cluster: arrival bases
// and the next side's cell_start, plus the atom count after the refresh.
// Each block takes a run of cells: first its totals, which the blocks read
// from one another's shared memory, then tiles of blockDim cells scanned by
// warp shuffles on top of the totals before them.  Coalesced: the 17 576
// cells of the 256 000-atom EAM system take 9.8 us (launch included), a
// single block with consecutive cells per thread took 36.
struct ScanSmem
{
    int2 total;          // this block's sums
    int2 warp[32];
};

__device__ __forceinline__ int2 warp_inclusive(int2 v, int lane)
{
    for (int o = 1; o < 32; o <<= 1)
    {
        const int a = __shfl_up_sync(0xffffffffu, v.x, o), b = __shfl_up_sync(0xffffffffu, v.y, o);
        if (lane >= o) { v.x += a; v.y += b; }
    }
    return v;
}

// inclusive scan over the block; every thread must call it
__device__ __forceinline__ int2 block_inclusive(int2 v, ScanSmem &sm, int2 &sum)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_inclusive(v, lane);
    if (lane == 31) sm.warp[w] = v;
    __syncthreads();
    if (w == 0)
    {
        const int2 t = warp_inclusive(lane < nw ? sm.warp[lane] : make_int2(0, 0), lane);
        __syncwarp();
        if (lane < nw) sm.warp[lane] = t;
    }
    __syncthreads();
    if (w > 0) { v.x += sm.warp[w - 1].x; v.y += sm.warp[w - 1].y; }
    sum = sm.warp[nw - 1];
    __syncthreads();
    return v;
}

__device__ __forceinline__ void scan_cells(const Geo &g, Dyn *dyn, const Side &S, const Side &T, ScanSmem &sm,
                                           cg::cluster_group &cl)
{
    const int nc = g.ncell, rank = cl.block_rank(), nblk = cl.num_blocks();
    const int per = (nc + nblk - 1) / nblk;
    const int lo = min(nc, rank * per), hi = min(nc, lo + per);
    auto cell = [&](int c) {
        if (c >= hi) return make_int2(0, 0);
        const int a = g.arr_total[c];
        return make_int2(a, S.cell_start[c + 1] - S.cell_start[c] - g.dep_count[c] + a);
    };
    int2 sum = make_int2(0, 0), tile;
    for (int c = lo + threadIdx.x; c < hi; c += blockDim.x)
    {
        const int2 v = cell(c);
        sum.x += v.x;
        sum.y += v.y;
    }
    block_inclusive(sum, sm, tile);
    if (threadIdx.x == 0) sm.total = tile;
    cl.sync();
    int2 base = make_int2(0, 0);
    for (int r = 0; r < rank; r++)
    {
        const int2 t = cl.map_shared_rank(&sm, r)->total;
        base.x += t.x;
        base.y += t.y;
    }
    for (int c0 = lo; c0 < hi; c0 += blockDim.x)
    {
        const int c = c0 + threadIdx.x;
        const int2 v = cell(c);
        const int2 in = block_inclusive(v, sm, tile);
        if (c < hi)
        {
            g.arr_base[c] = base.x + in.x - v.x;
            T.cell_start[c] = base.y + in.y - v.y;
        }
        base.x += tile.x;
        base.y += tile.y;
    }
    if (rank == nblk - 1 && threadIdx.x == 0)
    {
        g.arr_base[nc] = base.x;
        T.cell_start[nc] = base.y;
        dyn->n_next = base.y;
    }
    // (no block leaves while another still reads its totals)
    cl.sync();
}

// Replay of the swap-remove walk of one source cell (src/misc.c:276-303)
// with A placeholder tokens for the atoms that arrived from lower-index
// cells.  Emits the departure rank of each leaving atom (and queues it in
// its destination's bucket), the final slot of each stayer, and the slot of
// each placeholder.  By one warp: lane w holds the departures among tokens
// 32 w .. 32 w + 31 as a mask, tokens keep their place unless the walk moves
// them, and the walk steps from departure to departure (one or two a cell)
// instead of from token to token behind a dependent load each: half of a
// small system's refresh (4004 atoms in 160 cells: 33.6 us, 22.3 with this
// and twice the blocks).
constexpr int REPLAY_TOKENS = 1024;
__device__ __forceinline__ void replay_cell(const Geo &g, const Side &S, int c, int lane)
{
    const int start = S.cell_start[c];
    const int n0 = S.cell_start[c + 1] - start;
    const int base = g.arr_base[c];
    int len = n0 + g.arr_lower[c];
    unsigned leaving = 0;
    for (int k = 0; k < len; k += 32)
    {
        const int tok = k + lane;
        const bool d = tok < n0 && g.bdest[start + tok] != -2;
        const unsigned m = __ballot_sync(0xffffffffu, d);
        if (lane == k >> 5) leaving = m;
        if (tok < n0) g.bslot[start + tok] = tok;
        else if (tok < len) g.arr_slot[base + (tok - n0)] = tok;
    }
    __syncwarp();
    int i = 0, rank = 0;
    auto leave = [&](int tok) {
        if (lane == 0)
        {
            const int a = start + tok, D = g.bdest[a];
            g.brank[a] = rank;
            if (D >= 0) g.bucket[g.arr_base[D] + atomicAdd(&g.bucket_fill[D], 1)] = a;
        }
        rank++;
    };
    for (;;)
    {
        // the next departure at i or behind it
        const int low = i - 32 * lane;
        const unsigned mine = low <= 0 ? leaving : (low < 32 ? leaving & (0xffffffffu << low) : 0u);
        const unsigned any = __ballot_sync(0xffffffffu, mine != 0);
        if (!any) break;
        const int w = __ffs(any) - 1;
        i = 32 * w + __ffs(__shfl_sync(0xffffffffu, mine, w)) - 1;
        if (i >= len) break;
        leave(i);
        // the last element moves into slot i, unless it leaves as well
        for (len--; len > i; len--)
        {
            const bool gone = len < n0 && (__shfl_sync(0xffffffffu, leaving, len >> 5) >> (len & 31) & 1u);
            if (!gone) break;
            leave(len);
        }
        if (len > i && lane == 0)
        {
            if (len < n0) g.bslot[start + len] = i;
            else g.arr_slot[base + (len - n0)] = i;
        }
        i++;
    }
}

// the same of a cell of more tokens, by one thread
__device__ __noinline__ void replay_long_cell(const Geo &g, const Side &S, int c)
{
    const int start = S.cell_start[c];
    const int n0 = S.cell_start[c + 1] - start;
    const int base = g.arr_base[c];
    int len = n0 + g.arr_lower[c], i = 0, moved = -1, rank = 0;
    while (i < len)
    {
        const int tok = (moved >= 0) ? moved : i;
        const int a = start + tok;
        if (tok < n0 && g.bdest[a] != -2)
        {
            const int D = g.bdest[a];
            g.brank[a] = rank++;
            if (D >= 0)
            {
                const int pos = atomicAdd(&g.bucket_fill[D], 1);
                g.bucket[g.arr_base[D] + pos] = a;
            }
            len--;
            // the old last element (never overwritten: only the scan
            // position is) moves into slot i
            moved = (len != i) ? len : -1;
        }
        else
        {
            if (tok < n0) g.bslot[a] = i;
            else g.arr_slot[base + (tok - n0)] = i;
            i++;
            moved = -1;
        }
    }
}

// The cells first .. first + count - 1 (at most 32) by one warp.
__device__ __forceinline__ void replay_cells(const Geo &g, const Side &S, int first, int count, int lane)
{
    const int c = first + lane;
    int kind = 0;       // 1: departures; 2: the same, too many tokens for the masks
    if (lane < count && c < g.ncell)
    {
        const int n0 = S.cell_start[c + 1] - S.cell_start[c], A = g.arr_lower[c];
        if (g.dep_count[c] != 0) kind = n0 + A <= REPLAY_TOKENS ? 1 : 2;
        else
            for (int k = 0; k < A; k++) g.arr_slot[g.arr_base[c] + k] = n0 + k;
    }
    for (unsigned m = __ballot_sync(0xffffffffu, kind == 1); m; m &= m - 1) replay_cell(g, S, first + __ffs(m) - 1, lane);
    if (kind == 2) replay_long_cell(g, S, c);
}

// Order the arrivals of destination cell D and give them new indexes.
__device__ __forceinline__ void order_arrivals(const Geo &g, const Side &S, const Side &T, int D)
{
    const int total = g.arr_total[D];
    if (total == 0) return;
    const int base = g.arr_base[D];
    int *b = g.bucket + base;
    auto key = [&](int a) -> unsigned long long {
        return ((unsigned long long)g.bpath[a] << 44) |
               ((unsigned long long)S.cell_of[a] << 20) |
               (unsigned long long)g.brank[a];
    };
    for (int k = 1; k < total; k++)
    {
        const int a = b[k];
        const unsigned long long ka = key(a);
        int j = k - 1;
        while (j >= 0 && key(b[j]) > ka) { b[j + 1] = b[j]; j--; }
        b[j + 1] = a;
    }
    const int A = g.arr_lower[D];
    const int nstay = S.cell_start[D + 1] - S.cell_start[D] - g.dep_count[D];
    const int ns = T.cell_start[D];
    for (int k = 0; k < total; k++)
    {
        const int a = b[k];
        g.bnewidx[a] = ns + (k < A ? g.arr_slot[base + k] : nstay + A + (k - A));
    }
}

// Last phase, one atom: its place on the next side (moved: some atom moved,
// so the sides are swapped after this), and the per-atom tables the force
// kernels read, formed from the position in hand.  PACK: the slots are
// renumbered in the new order -- slot = index, so a list build walks and
// writes consecutive atoms of a cell together, and until the next rebuild
// (no refresh in between) every slot-to-index map is the identity.
template <bool PACK>
__device__ __forceinline__ void place_atom(const Geo &g, Dyn *dyn, const Side &S, const Side &T, int i, bool moved,
                                           int n_next)
{
    const int cap = g.cap;
    const int c = S.cell_of[i];
    int idx = i, D = c;
    if (moved)
    {
        const int d = g.bdest[i];
        if (d == -1) return;
        if (d == -2) idx = T.cell_start[c] + (g.dep_count[c] == 0 ? (i - S.cell_start[c]) : g.bslot[i]);
        else
        {
            D = d;
            idx = g.bnewidx[i];
        }
        if (idx < 0 || idx >= n_next)
        {
            // cannot happen for a consistent refresh; recorded instead of writing
            atomic_or_err(dyn, FMDG_ERRBIT_INTERNAL);
            return;
        }
    }
    const double x[3] = {S.x[i], S.x[cap + i], S.x[2 * (size_t)cap + i]};
    const unsigned kind = S.kind[i];
    const int group = S.group[i];
    const int t = PACK ? idx : (g.skin_on ? S.slot[i] : 0);
    if (moved)
    {
        for (int k = 0; k < 3; k++)
        {
            T.x[k * cap + idx] = x[k];
            T.v[k * cap + idx] = S.v[k * cap + i];
        }
        T.kind[idx] = kind;
        T.group[idx] = group;
        T.atomid[idx] = S.atomid[i];
        T.cell_of[idx] = D;
        if (g.skin_on) T.slot[idx] = t;
    }
    else if (PACK)
        S.slot[i] = t;
    if (g.skin_on) prep_skin_atom(g, dyn, idx, t, D, (int)kind, group, x, !PACK && !dyn->rebuild);
    else prep_local_atom(g, idx, D, (int)kind, x);
}

// swaps sides after a refresh that moved atoms; advances the device copy of
// the simulation time by one step (src/integrators.c:203, :256)
__device__ __forceinline__ void flip_sides(const Geo &g, Dyn *dyn, int mode)
{
    dyn->time += (mode == FMDG_REFRESH_ONLY) ? 0.0 : g.st.dt;
    if (dyn->any_move)
    {
        dyn->cur ^= 1;
        dyn->n = dyn->n_next;
        dyn->any_move = 0;
    }
}

__device__ __forceinline__ void load_half_kicks(const Geo &g, double *hk)
{
    if (threadIdx.x < g.nkinds) hk[threadIdx.x] = g.st.hk[threadIdx.x];
    __syncthreads();
}

// ------------------------------------------------- grid kernels (one system)

__global__ void __launch_bounds__(256) k_bin_classify(__grid_constant__ const LocOne loc, int mode)
{
    step_wait();
    const Geo &g = loc.g;
    __shared__ double hk[FMDG_MAXK];
    load_half_kicks(g, hk);
    Dyn *dyn = g.dyn;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < dyn->n) classify_atom(g, dyn, g.side[dyn->cur], i, mode, hk);
}

// cells a warp of k_bin_cells looks at
constexpr int WARP_CELLS = 8;

// (one cluster)
constexpr int SCAN_BLOCKS = 8;
__global__ void __launch_bounds__(1024) k_bin_scan(__grid_constant__ const LocOne loc)
{
    step_wait();
    const Geo &g = loc.g;
    Dyn *dyn = g.dyn;
    if (!dyn->any_move) return;
    __shared__ ScanSmem sm;
    cg::cluster_group cl = cg::this_cluster();
    scan_cells(g, dyn, g.side[dyn->cur], g.side[dyn->cur ^ 1], sm, cl);
}

__global__ void __launch_bounds__(128) k_bin_cells(__grid_constant__ const LocOne loc)
{
    step_wait();
    const Geo &g = loc.g;
    const Dyn *dyn = g.dyn;
    if (!dyn->any_move) return;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    replay_cells(g, g.side[dyn->cur], warp * WARP_CELLS, WARP_CELLS, threadIdx.x & 31);
}

__global__ void __launch_bounds__(128) k_bin_arrivals(__grid_constant__ const LocOne loc)
{
    step_wait();
    const Geo &g = loc.g;
    const Dyn *dyn = g.dyn;
    const int D = blockIdx.x * blockDim.x + threadIdx.x;
    if (dyn->any_move && D < g.ncell) order_arrivals(g, g.side[dyn->cur], g.side[dyn->cur ^ 1], D);
}

// the last block to finish swaps the sides
__global__ void __launch_bounds__(256) k_bin_place(__grid_constant__ const LocOne loc, int mode)
{
    step_wait();
    const Geo &g = loc.g;
    Dyn *dyn = g.dyn;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int cur = dyn->cur;
    if (i < dyn->n) place_atom<false>(g, dyn, g.side[cur], g.side[cur ^ 1], i, dyn->any_move != 0, dyn->n_next);
    __shared__ unsigned ticket;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        ticket = atomicAdd(&dyn->place_done, 1u);
        if (ticket == gridDim.x - 1)
        {
            dyn->place_done = 0;
            flip_sides(g, dyn, mode);
        }
    }
}

// --------------------------------------------- grid kernels (large, packed)
//
// The same phases for a pack of large systems, on the steps that rebuild a
// member's skin list.  A bounded grid goes from one due member to the next,
// so on the other steps a launch is a block per SM that reads the members'
// flags and leaves (a block per 128 atoms, idle on most steps, cost 1.2 % of
// the 2048-job fleet's rate).

// the members (bits) that rebuild their list this step; every lane of the
// warp takes part
__device__ __forceinline__ unsigned due_members(const LocPack &L)
{
    const int s = threadIdx.x & 31;
    bool due = false;
    if (s < L.nsys)
    {
        const Dyn *d = L.geos[s].dyn;
        due = d->steps_left > 0 && d->rebuild != 0;
    }
    return __ballot_sync(0xffffffffu, due);
}

__global__ void __launch_bounds__(256) k_pack_classify(__grid_constant__ const LocPack loc)
{
    step_wait();
    __shared__ double hk[FMDG_MAXK];
    for (unsigned m = due_members(loc); m; m &= m - 1)
    {
        const Geo &g = loc.geos[__ffs(m) - 1];
        __syncthreads();
        load_half_kicks(g, hk);
        Dyn *dyn = g.dyn;
        const int n = dyn->n;
        const Side S = g.side[dyn->cur];
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
            classify_atom(g, dyn, S, i, FMDG_REFRESH_ONLY, hk);
    }
}

// (one cluster of SCAN_BLOCKS per system)
__global__ void __launch_bounds__(512) k_pack_scan(__grid_constant__ const LocPack loc)
{
    step_wait();
    const Geo &g = loc.geos[blockIdx.x / SCAN_BLOCKS];
    Dyn *dyn = g.dyn;
    if (dyn->steps_left <= 0 || !dyn->rebuild || !dyn->any_move) return;
    __shared__ ScanSmem sm;
    cg::cluster_group cl = cg::this_cluster();
    scan_cells(g, dyn, g.side[dyn->cur], g.side[dyn->cur ^ 1], sm, cl);
}

__global__ void __launch_bounds__(256) k_pack_cells(__grid_constant__ const LocPack loc)
{
    step_wait();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (unsigned m = due_members(loc); m; m &= m - 1)
    {
        const Geo &g = loc.geos[__ffs(m) - 1];
        const Dyn *dyn = g.dyn;
        if (!dyn->any_move) continue;
        const Side S = g.side[dyn->cur];
        for (int c = warp * WARP_CELLS; c < g.ncell; c += nw * WARP_CELLS) replay_cells(g, S, c, WARP_CELLS, threadIdx.x & 31);
    }
}

__global__ void __launch_bounds__(128) k_pack_arrivals(__grid_constant__ const LocPack loc)
{
    step_wait();
    for (unsigned m = due_members(loc); m; m &= m - 1)
    {
        const Geo &g = loc.geos[__ffs(m) - 1];
        const Dyn *dyn = g.dyn;
        if (!dyn->any_move) continue;
        const Side S = g.side[dyn->cur], T = g.side[dyn->cur ^ 1];
        for (int D = blockIdx.x * blockDim.x + threadIdx.x; D < g.ncell; D += gridDim.x * blockDim.x) order_arrivals(g, S, T, D);
    }
}

// The last block to finish a member swaps its sides and leaves the cells'
// counters at zero for its next refresh.
__global__ void __launch_bounds__(256) k_pack_place(__grid_constant__ const LocPack loc)
{
    step_wait();
    __shared__ unsigned ticket;
    for (unsigned m = due_members(loc); m; m &= m - 1)
    {
        const Geo &g = loc.geos[__ffs(m) - 1];
        Dyn *dyn = g.dyn;
        const int cur = dyn->cur, n = dyn->n;
        const bool moved = dyn->any_move != 0;
        const int n_next = moved ? dyn->n_next : n;
        const Side S = g.side[cur], T = g.side[cur ^ 1];
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.cap; i += gridDim.x * blockDim.x)
        {
            if (i < n) place_atom<true>(g, dyn, S, T, i, moved, n_next);
            if (i >= n_next) g.pos[i] = -1;
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            __threadfence();
            ticket = atomicAdd(&dyn->place_done, 1u);
        }
        __syncthreads();
        if (ticket != gridDim.x - 1) continue;
        // (dep_count, arr_lower, arr_total, bucket_fill are contiguous)
        if (moved)
            for (int c = threadIdx.x; c < 4 * g.ncell; c += blockDim.x) g.dep_count[c] = 0;
        if (threadIdx.x == 0)
        {
            dyn->place_done = 0;
            flip_sides(g, dyn, FMDG_REFRESH_ONLY);
        }
    }
}

// ----------------------------------------------------------- cluster kernel

__device__ __forceinline__ const Geo &cluster_geo(const LocOne &L, int) { return L.g; }
__device__ __forceinline__ const Geo &cluster_geo(const LocPack &L, int s) { return L.geos[s]; }

// All phases of one system's refresh by one cluster.  Packed systems
// (LocPack): only on a step that rebuilds the system's skin list (between
// rebuilds an atom stays within skin/2 of its build position, less than a
// cell, and the packed kernels address atoms by slot); the conditions are
// uniform over a cluster.
template <class L>
__global__ void __launch_bounds__(512) k_refresh_cluster(__grid_constant__ const L loc, int mode)
{
    step_wait();
    constexpr bool PACK = !L::one_system;
    cg::cluster_group cl = cg::this_cluster();
    const int nblk = cl.num_blocks(), rank = cl.block_rank();
    const Geo &g = cluster_geo(loc, blockIdx.x / nblk);
    if (loc_idle(loc, g)) return;
    Dyn *dyn = g.dyn;
    if (PACK && !dyn->rebuild) return;
    __shared__ double hk[FMDG_MAXK];
    __shared__ ScanSmem sm;
    load_half_kicks(g, hk);
    const int n = dyn->n, cur = dyn->cur, ncell = g.ncell;
    const Side S = g.side[cur], T = g.side[cur ^ 1];
    const int tid = rank * blockDim.x + threadIdx.x, nt = nblk * blockDim.x;
    // (the cells' counters are zero between refreshes: cleared below)
    for (int i = tid; i < n; i += nt) classify_atom(g, dyn, S, i, mode, hk);
    cl.sync();
    const bool moved = *(volatile int *)&dyn->any_move != 0;
    int n_next = n;
    if (moved)
    {
        scan_cells(g, dyn, S, T, sm, cl);
        const int nw = nt >> 5, each = min(32, (ncell + nw - 1) / nw);
        for (int c = (tid >> 5) * each; c < ncell; c += nw * each) replay_cells(g, S, c, each, tid & 31);
        cl.sync();
        for (int c = tid; c < ncell; c += nt) order_arrivals(g, S, T, c);
        cl.sync();
        n_next = *(volatile int *)&dyn->n_next;
    }
    for (int i = tid; i < n; i += nt) place_atom<PACK>(g, dyn, S, T, i, moved, n_next);
    if (PACK)
        for (int i = n_next + tid; i < g.cap; i += nt) g.pos[i] = -1;
    cl.sync();
    // (dep_count, arr_lower, arr_total, bucket_fill are contiguous)
    if (moved)
        for (int c = tid; c < 4 * ncell; c += nt) g.dep_count[c] = 0;
    if (tid == 0) flip_sides(g, dyn, mode);
}

// Blocks of as few threads as give every atom one: the phases are binary64
// work, which an SM issues for one warp at a time, so few warps on many SMs.
// A pack's systems (up to PACK_CLUSTER_ATOMS) take eight blocks each (the
// portable cluster size).
constexpr int REFRESH_BLOCKS = 8;
int refresh_threads(int n, int blocks)
{
    const int t = (fmdg_grid(n, blocks) + 31) & ~31;
    return t < 64 ? 64 : (t > 512 ? 512 : t);
}

// A single system takes sixteen, where its device has room for such a
// cluster: 4000 atoms refresh in 11.6 us against 14.0 with eight.  Both the
// permission for a cluster of more than eight and the answer belong to the
// device.
int single_refresh_blocks(const fmdg_sys_t *s)
{
    static PerDevice kept;
    if (s->refresh_blocks) return s->refresh_blocks;
    return kept.get(s->device, [s] {
        int current = s->device;
        cudaGetDevice(&current);
        if (current != s->device) cudaSetDevice(s->device);
        const auto kernel = k_refresh_cluster<LocOne>;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(16);
        cfg.blockDim = dim3(512);
        cudaLaunchAttribute at = {};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 16;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int room = 0, blocks = 16;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&room, kernel, &cfg) != cudaSuccess || room < 1)
        {
            cudaGetLastError();
            blocks = REFRESH_BLOCKS;
        }
        if (current != s->device) cudaSetDevice(current);
        return blocks;
    });
}

} // namespace

// One refresh: optional integrator start step, then re-binning and the
// per-atom tables.  All launches go to the system's stream; graph-capturable
// (no host reads).
int fmdg_launch_refresh(fmdg_sys_t *s, int mode, double dt, int group, int thermostat)
{
    Geo &g = s->g;
    cudaStream_t st = s->stream;
    set_step_dt(s, dt);
    g.st.group = group;
    g.st.thermostat = thermostat;
    const LocOne L{g};
    if (g.cap <= CLUSTER_ATOMS)
    {
        const int nb = single_refresh_blocks(s);
        FMDG_CK(fmdg_launch(k_refresh_cluster<LocOne>, nb, refresh_threads(g.cap, nb), 0, st, s->overlap, nb, L, mode));
        s->launches++;
        return FMDG_OK;
    }
    // dep_count, arr_lower, arr_total, bucket_fill are contiguous
    FMDG_CK(cudaMemsetAsync(g.dep_count, 0, sizeof(int) * 4 * (size_t)g.ncell, st));
    const bool ov = s->overlap;
    FMDG_CK(fmdg_launch(k_bin_classify, fmdg_grid(g.cap, 256), 256, 0, st, false, 1, L, mode));
    FMDG_CK(fmdg_launch(k_bin_scan, SCAN_BLOCKS, 1024, 0, st, ov, SCAN_BLOCKS, L));
    FMDG_CK(fmdg_launch(k_bin_cells, fmdg_grid(g.ncell, 4 * WARP_CELLS), 128, 0, st, ov, 1, L));
    FMDG_CK(fmdg_launch(k_bin_arrivals, fmdg_grid(g.ncell, 128), 128, 0, st, ov, 1, L));
    FMDG_CK(fmdg_launch(k_bin_place, fmdg_grid(g.cap, 256), 256, 0, st, ov, 1, L, mode));
    s->launches += 5;
    return FMDG_OK;
}

bool fmdg_pack_large(int n) { return n > PACK_CLUSTER_ATOMS; }

// Step start of every system of a pack: velocity-Verlet start step, slot
// tables and displacement test (k_skin_start), then the cell refresh of the
// systems that rebuild their skin list this step: a cluster each, or, in a
// pack of large systems, the grid kernels.  Returns the kernels launched, or
// minus a status.
int fmdg_pack_launch_refresh(const fmdg_pack_launch &P)
{
    cudaStream_t st = P.stream;
    const bool ov = P.overlap;
    const int mode = FMDG_REFRESH_ONLY;
    int n = fmdg_pack_launch_start(P);
    if (n < 0) return n;
    if (P.large)
    {
        const int grid = PACK_GRID;
        fmdg_launch(k_pack_classify, grid, 256, 0, st, ov, 1, P.la);
        fmdg_launch(k_pack_scan, SCAN_BLOCKS * P.nsys, 512, 0, st, ov, SCAN_BLOCKS, P.la);
        fmdg_launch(k_pack_cells, grid, 256, 0, st, ov, 1, P.la);
        fmdg_launch(k_pack_arrivals, grid, 128, 0, st, ov, 1, P.la);
        fmdg_launch(k_pack_place, grid, 256, 0, st, ov, 1, P.la);
        n += 5;
    }
    else
    {
        int most = 1;
        for (int k = 0; k < P.nsys; k++) most = P.la.geos[k].cap > most ? P.la.geos[k].cap : most;
        fmdg_launch(k_refresh_cluster<LocPack>, REFRESH_BLOCKS * P.nsys, refresh_threads(most, REFRESH_BLOCKS), 0, st, ov,
                    REFRESH_BLOCKS, P.la, mode);
        n++;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return -fmdg_fail("pack refresh", e);
    return n;
}
