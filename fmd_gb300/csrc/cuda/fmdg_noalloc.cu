// Pair forces without any allocation by the library.
//
// Some callers cannot let a library call cudaMalloc: code that records the
// call into a CUDA graph (allocation is not a capturable stream operation),
// hosts that own all device memory through their own pool or arena, and
// serving loops where the implicit device synchronisation of cudaMalloc
// would stall work queued by other streams.  fmdg_pair_forces_noalloc gives
// them the binary64 LJ / Morse force evaluation of fmdg_compute_forces with
// every input and output supplied by the caller.  The only scratch it needs,
// the per-block energy partials of the deterministic two-level reduction,
// lives in a fixed file-scope device array (FMDG_NOALLOC_MAX_BLOCKS blocks
// of up to 128 atoms, i.e. at most FMDG_NOALLOC_MAX_ATOMS atoms per call; 512 KiB
// held by every GPU that loads the library until the process exits).
//
// Host code cannot use the array's name as a device address, so the first
// call on each device (with that device current) looks the address up with
// cudaGetSymbolAddress and keeps it; that first call should be made before
// any stream capture begins.  All calls share the one array and each call
// overwrites it completely, so calls that overlap on the GPU (different
// streams, no ordering between them) race and must be serialised by the
// caller.
//
// The first look-up is made under a lock, so first calls from several host
// threads are safe.  A cudaDeviceReset of a device invalidates the address
// kept for it: this entry point must not be called on that device again in
// the same process.  Atom kinds must lie in [0, nkinds): an atom whose kind,
// or a neighbour's kind, lies outside gets NaN forces (and the energy is
// NaN), the pair table is never read out of range.
#include <math.h>
#include <mutex>
#include <stdio.h>
#include <string.h>
#include "fmdg_internal.cuh"

#define FMDG_NOALLOC_MAX_BLOCKS 8192
#define FMDG_NOALLOC_MAX_ATOMS (FMDG_NOALLOC_MAX_BLOCKS * 128)
#define FMDG_NOALLOC_MAX_KINDS 4
#define FMDG_NOALLOC_MAX_DEVICES 64

static __device__ __align__(256) double g_noalloc_partials[FMDG_NOALLOC_MAX_BLOCKS];

namespace {

struct NoallocArgs   // passed by value: no device copy of the parameters
{
    int n, nkinds;
    int atoms;          // per block
    int nc[3], pbc[3];
    double l[3];
    float lf[3], rcf;   // binary32: box lengths, largest cutoff (rounded up)
    fmdg_pair_t pairs[FMDG_NOALLOC_MAX_KINDS * FMDG_NOALLOC_MAX_KINDS];
};

__device__ __forceinline__ int wrap_axis(const NoallocArgs &a, int d, int h, int o)
{
    int j = h + o;
    if (j < 0) return a.pbc[d] ? j + a.nc[d] : -1;
    if (j >= a.nc[d]) return a.pbc[d] ? j - a.nc[d] : -1;
    return j;
}

// box lengths the neighbour cell at offset o along axis d of home cell h is
// shifted by: -1, 0 or 1
__device__ __forceinline__ int axis_sign(const NoallocArgs &a, int d, int h, int o)
{
    const int j = h + o;
    return j < 0 ? -1 : (j >= a.nc[d] ? 1 : 0);
}

// its image shift
__device__ __forceinline__ double axis_shift(const NoallocArgs &a, int d, int h, int o)
{
    const int j = h + o;
    return j < 0 ? -a.l[d] : (j >= a.nc[d] ? a.l[d] : 0.0);
}

// binary64 as binary32 truncated towards zero, in integer operations
// (conversion instructions issue at the binary64 rate); below the binary32
// range 0, beyond it (and NaN) infinity
__device__ __forceinline__ float trunc_f(double x)
{
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned e = (hi >> 20) & 0x7ffu;
    unsigned m = (((hi & 0x7fffffffu) - 0x38000000u) << 3) | (lo >> 29);
    m = e < 897u ? 0u : m;
    m = e > 1150u ? 0x7f800000u : m;
    return __uint_as_float(m | (hi & 0x80000000u));
}

// Binary64 gather over the 27-cell stencil (same pair arithmetic as the
// binary64 path of fmdg_force.cu's formulas: src/lj.h:26-58,
// src/morse.h:26-58), one warp per atom.
//
// GB300 issues binary64 at 1/64 of the binary32 rate, so the binary64 work
// per pair (~50 instructions) bounds this kernel.  Five candidates in six
// of the stencil are out of range: one thread per atom spent more on their
// distances, and on warps whose lanes were in range one by one, than on the
// pairs.  Here the lanes test 32 candidates in binary32 (a conservative
// filter), the hits are queued in shared memory by ballot, and whenever the
// queue holds 32 every lane evaluates one pair: full warps of binary64
// work, none on candidates the filter drops.  62 100 Morse atoms: 7.50 ->
// 1.26 ms.
constexpr int NOALLOC_WARPS = 16;      // per block

template <bool MORSE, bool LJ>
__global__ void __launch_bounds__(32 * NOALLOC_WARPS) k_pair_noalloc(
    __grid_constant__ const NoallocArgs a, const double *__restrict__ x, const unsigned *__restrict__ kind,
    const int *__restrict__ cell_start, const int *__restrict__ cell_of, double *__restrict__ F, double *partials)
{
    __shared__ int queue[NOALLOC_WARPS][64];
    __shared__ double red[NOALLOC_WARPS];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int n = a.n;
    int *q = queue[w];
    double pe_warp = 0.0;
    for (int i = blockIdx.x * a.atoms + w; i < min(n, (blockIdx.x + 1) * a.atoms); i += NOALLOC_WARPS)
    {
        const int c = cell_of[i];
        const int cx = c / (a.nc[1] * a.nc[2]), cy = (c / a.nc[2]) % a.nc[1], cz = c % a.nc[2];
        const double xi[3] = {x[i], x[n + i], x[2 * (size_t)n + i]};
        const unsigned ki = kind[i];
        bool bad = ki >= (unsigned)a.nkinds;
        double f[3] = {0.0, 0.0, 0.0}, pe = 0.0;
        // Filter: a pair in range has |x_j| <= |x_i| + rc + |shift|, and the
        // binary32 difference of its truncated coordinates is off by at most
        // 2^-21 of the magnitudes involved along each axis; beyond the
        // cutoff plus that (doubled) no pair is in range
        float xf[3], slack = 0.f;
        for (int d = 0; d < 3; d++)
        {
            xf[d] = trunc_f(xi[d]);
            slack = fmaxf(slack, 2.f * fabsf(xf[d]) + 2.f * a.lf[d] + a.rcf);
        }
        const float lim = a.rcf + 4.f * 4.8e-7f * slack;
        const float lim2 = lim * lim * 1.000001f;

        // one pair per lane (have: lanes with one)
        auto evaluate = [&](int e, bool have) {
            if (!have) return;
            const int j = e & 0xfffff, code = e >> 20;
            const unsigned kj = kind[j];
            const fmdg_pair_t &pp = a.pairs[ki * a.nkinds + kj];
            const int o[3] = {code / 9 - 1, (code / 3) % 3 - 1, code % 3 - 1}, h[3] = {cx, cy, cz};
            double rv[3];
            for (int d = 0; d < 3; d++)
            {
                double x2 = x[(size_t)d * n + j];
                const double s = axis_shift(a, d, h[d], o[d]);
                if (s != 0.0) x2 = __dadd_rn(x2, s);
                rv[d] = __dsub_rn(xi[d], x2);
            }
            const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(rv[0], rv[0]), __dmul_rn(rv[1], rv[1])),
                                        __dmul_rn(rv[2], rv[2]));
            if (LJ && (!MORSE || pp.cat == FMDG_POT_LJ))
            {
                if (!(r2 < pp.p[2])) return;
                const double inv_r2 = 1.0 / r2;
                const double inv_rs2 = pp.p[1] * inv_r2;
                const double inv_rs6 = inv_rs2 * inv_rs2 * inv_rs2;
                const double inv_rs12 = inv_rs6 * inv_rs6;
                const double factor = 12.0 * pp.p[0] * inv_r2 * (inv_rs12 - 0.5 * inv_rs6);
                for (int d = 0; d < 3; d++) f[d] += rv[d] * factor;
                pe += 0.5 * (pp.p[0] * (inv_rs12 - inv_rs6));
            }
            else if (MORSE)
            {
                if (!(r2 < pp.p[3])) return;
                // 1/r, and r from it by one Newton step to the rounding of a
                // square root: one special function instead of two (1371 ->
                // 1264 us), error against 64 bits unchanged; coincident
                // atoms have r = 0
                const double inv_r = rsqrt(r2);
                const double r1 = r2 * inv_r;
                const double r = __double_as_longlong(r2) ? fma(0.5 * inv_r, fma(-r1, r1, r2), r1) : 0.0;
                const double e1 = exp(-pp.p[1] * (r - pp.p[2]));
                const double e2 = e1 * e1;
                const double factor = 2.0 * pp.p[1] * pp.p[0] * inv_r * (e2 - e1);
                for (int d = 0; d < 3; d++) f[d] += factor * rv[d];
                pe += 0.5 * (pp.p[0] * (e2 - 2.0 * e1));
            }
        };

        int qn = 0;
        for (int col = 0; col < 9; col++)
        {
            const int ox = col / 3 - 1, oy = col % 3 - 1;
            const int jx = wrap_axis(a, 0, cx, ox), jy = wrap_axis(a, 1, cy, oy);
            if (jx < 0 || jy < 0) continue;
            const int c0 = a.nc[2] * (jy + a.nc[1] * jx);
            const float px = xf[0] - (float)axis_sign(a, 0, cx, ox) * a.lf[0];
            const float py = xf[1] - (float)axis_sign(a, 1, cy, oy) * a.lf[1];
            for (int oz = -1; oz <= 1; oz++)
            {
                const int jz = wrap_axis(a, 2, cz, oz);
                if (jz < 0) continue;
                const float pz = xf[2] - (float)axis_sign(a, 2, cz, oz) * a.lf[2];
                const int code = col * 3 + oz + 1;
                const int je = cell_start[c0 + jz + 1];
                for (int j0 = cell_start[c0 + jz]; j0 < je; j0 += 32)
                {
                    const int j = j0 + lane;
                    bool hit = false;
                    if (j < je && !(code == 13 && j == i))
                    {
                        const float dx = px - trunc_f(x[j]), dy = py - trunc_f(x[n + j]);
                        const float dz = pz - trunc_f(x[2 * (size_t)n + j]);
                        bad = bad || kind[j] >= (unsigned)a.nkinds;     // outside the pair table: no table read
                        // (a coordinate that is not a number is infinity here and
                        // dropped, as the exact test drops it)
                        hit = !bad && !(dx * dx + dy * dy + dz * dz >= lim2);
                    }
                    const unsigned m = __ballot_sync(FULL, hit);
                    if (hit) q[qn + __popc(m & ((1u << lane) - 1u))] = j | (code << 20);
                    qn += __popc(m);
                    __syncwarp();
                    if (qn >= 32)
                    {
                        const int e = q[lane], rest = q[32 + lane];
                        __syncwarp();
                        qn -= 32;
                        if (lane < qn) q[lane] = rest;
                        __syncwarp();
                        evaluate(e, true);
                    }
                }
            }
        }
        evaluate(lane < qn ? q[lane] : 0, lane < qn);
        __syncwarp();
        // fixed tree over the lanes
        for (int off = 16; off > 0; off >>= 1)
        {
            for (int d = 0; d < 3; d++) f[d] += __shfl_down_sync(FULL, f[d], off);
            pe += __shfl_down_sync(FULL, pe, off);
        }
        if (__any_sync(FULL, bad))
        {
            for (int d = 0; d < 3; d++) f[d] = __longlong_as_double(0x7ff8000000000000ll);
            pe = f[0];
        }
        if (lane == 0)
        {
            for (int d = 0; d < 3; d++) F[(size_t)d * n + i] = f[d];
            pe_warp += pe;
        }
    }
    // deterministic block sum -> this block's slot of the static partials
    if (lane == 0) red[w] = pe_warp;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double t = 0.0;
        for (int k = 0; k < NOALLOC_WARPS; k++) t += red[k];
        partials[blockIdx.x] = t;
    }
}

__global__ void k_pair_noalloc_final(const double *partials, int nblocks, double *pe_out)
{
    __shared__ double red[256];
    double s = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) s += partials[b];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1)
    {
        if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) *pe_out = red[0];
}

double *g_partials_addr[FMDG_NOALLOC_MAX_DEVICES];
std::mutex g_partials_lock;   // guards the first look-up on each device

} // namespace

extern "C" int fmdg_pair_forces_noalloc(int n, const int nc[3], const int pbc[3], const double l[3], int nkinds,
                                        const fmdg_pair_t *pairs, const double *x, const unsigned *kind,
                                        const int *cell_start, const int *cell_of, double *F, double *pe,
                                        void *stream)
{
    if (n < 0 || n > FMDG_NOALLOC_MAX_ATOMS)
    {
        char msg[160];
        snprintf(msg, sizeof msg, "fmdg_pair_forces_noalloc: %d atoms exceed the fixed scratch limit of %d",
                 n, FMDG_NOALLOC_MAX_ATOMS);
        return fmdg_set_error(msg);
    }
    if (nkinds < 1 || nkinds > FMDG_NOALLOC_MAX_KINDS)
        return fmdg_set_error("fmdg_pair_forces_noalloc: 1..4 atom kinds");
    NoallocArgs a;
    memset(&a, 0, sizeof a);
    a.n = n;
    a.nkinds = nkinds;
    for (int d = 0; d < 3; d++)
    {
        if (nc[d] < 1) return fmdg_set_error("fmdg_pair_forces_noalloc: bad cell grid");
        a.nc[d] = nc[d];
        a.pbc[d] = pbc[d] ? 1 : 0;
        a.l[d] = l[d];
    }
    double rc2max = 0.0;
    int cats = 0;
    for (int k = 0; k < nkinds * nkinds; k++)
    {
        if (pairs[k].cat != FMDG_POT_LJ && pairs[k].cat != FMDG_POT_MORSE)
            return fmdg_set_error("fmdg_pair_forces_noalloc: LJ and Morse pairs only");
        a.pairs[k] = pairs[k];
        cats |= 1 << pairs[k].cat;
        const double rc2 = pairs[k].cat == FMDG_POT_MORSE ? pairs[k].p[3] : pairs[k].p[2];
        if (rc2 > rc2max) rc2max = rc2;
    }
    for (int d = 0; d < 3; d++) a.lf[d] = (float)fabs(l[d]);
    a.rcf = (float)(sqrt(rc2max) * (1.0 + 1e-6));
    int dev = 0;
    FMDG_CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= FMDG_NOALLOC_MAX_DEVICES) return fmdg_set_error("fmdg_pair_forces_noalloc: device id");
    double *partials = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_partials_lock);
        if (g_partials_addr[dev] == nullptr)
        {
            void *p = nullptr;
            FMDG_CK(cudaGetSymbolAddress(&p, g_noalloc_partials));
            g_partials_addr[dev] = (double *)p;
        }
        partials = g_partials_addr[dev];
    }
    cudaStream_t st = (cudaStream_t)stream;
    // one atom per warp while the partials hold a slot per block
    a.atoms = NOALLOC_WARPS;
    while ((n + a.atoms - 1) / a.atoms > FMDG_NOALLOC_MAX_BLOCKS) a.atoms *= 2;
    const int nb = n > 0 ? (n + a.atoms - 1) / a.atoms : 1;
    const int threads = 32 * NOALLOC_WARPS;
    if (cats == (1 << FMDG_POT_LJ))
        k_pair_noalloc<false, true><<<nb, threads, 0, st>>>(a, x, kind, cell_start, cell_of, F, partials);
    else if (cats == (1 << FMDG_POT_MORSE))
        k_pair_noalloc<true, false><<<nb, threads, 0, st>>>(a, x, kind, cell_start, cell_of, F, partials);
    else k_pair_noalloc<true, true><<<nb, threads, 0, st>>>(a, x, kind, cell_start, cell_of, F, partials);
    k_pair_noalloc_final<<<1, 256, 0, st>>>(partials, nb, pe);
    FMDG_CK(cudaGetLastError());
    return FMDG_OK;
}
