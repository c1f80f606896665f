// mdg_pme.cu -- smooth particle-mesh Ewald reciprocal space.
//
// mdpy v0.2.1 only names a long-range solver (LONG_RANGE_SOLVER = ['PME',
// 'PPPM'], mdpy/constraint/__init__.py:22; CharmmForcefield(long_range_solver,
// ewald_error), mdpy/forcefield/charmm_forcefield.py:23,30-31) and never
// implements one; this file is new.  Method: Essmann et al., J. Chem. Phys.
// 103 (1995) 8577 -- order-p cardinal B-spline charge assignment, the
// influence function exp(-pi^2 m^2/beta^2)/(pi V m^2) |b(m)|^2 applied in
// Fourier space, and analytic-derivative force interpolation.
//
// Per evaluation:
//   k_spread_rows  one warp per cluster, an atom at a time: p^3 int64 fixed-
//              point adds, whole rows of z points per instruction (k_spread,
//              on request: one thread per atom into a shared-memory tile of the
//              block's grid patch; the same sums);
//   mdg_fft.cu the transforms of small grids, influence function included, in
//              three launches for a whole batch; larger grids:
//   k_grid_convert  int64 grid -> float grid, and re-zeroes the int64 grid;
//   cuFFT R2C  (the only library call of the path);
//   k_convolve multiply by the influence function; optional energy sum;
//   cuFFT C2R  gives the potential on the grid (unnormalised inverse);
//   k_gather   one thread per atom (on request the block's patch of the
//              potential staged in shared memory; k_gather_rows where clusters
//              are few); -q grad(theta) . phi into the fixed-point force
//              accumulators.
// Charges enter pre-scaled by sqrt(k_e), so the Coulomb constant needs no
// extra multiply anywhere.
#include <algorithm>
#include <cmath>
#include <vector>

#include "mdg_internal.cuh"

namespace mdg {
namespace {

long long round_up(long long v, long long m) { return (v + m - 1) / m * m; }

// th[i] = M_p(w + p - 1 - i), dth = d th / dw (same recursion as the oracle)
template <int P>
__device__ __forceinline__ void spline(float w, float *th, float *dth) {
    float a[P];
#pragma unroll
    for (int i = 0; i < P; ++i) a[i] = 0.f;
    a[0] = 1.f - w;
    a[1] = w;
#pragma unroll
    for (int n = 3; n <= P; ++n) {
        if (n == P) {
            dth[0] = -a[0];
#pragma unroll
            for (int i = 1; i < P; ++i) dth[i] = a[i - 1] - a[i];
        }
        const float div = 1.0f / (float)(n - 1);
        float b[P];
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float left = i >= 1 ? a[i - 1] : 0.f;
            const float right = i <= n - 2 ? a[i] : 0.f;
            b[i] = div * ((w + (float)(n - 1 - i)) * left + ((float)(i + 1) - w) * right);
        }
#pragma unroll
        for (int i = 0; i < n; ++i) a[i] = b[i];
    }
#pragma unroll
    for (int i = 0; i < P; ++i) th[i] = a[i];
}

struct PmeArgs {
    const float4 *__restrict__ xq;
    const SysDev *__restrict__ sys;
    const int *__restrict__ cl_sys;
    int n_pad;
    unsigned long long *grid_i;
    const float *__restrict__ phi;
    unsigned long long *f;
    int tile_gather;               // stage the block's grid patch in shared memory
    float weight;                  // force weight (multiple time steps)
};

// grid coordinate u = x K / L wrapped into [0, K) with fmodf (exact), so the
// first stencil point g0 is a valid index for any finite or non-finite x
template <int P>
__device__ __forceinline__ void frac(float x, float kl, int K, int &g0, float &w) {
    const float Kf = (float)K;
    float u = fmodf(x * kl, Kf);
    if (u < 0.f) u += Kf;
    if (!(u >= 0.f && u < Kf)) u = 0.f;  // NaN, or -tiny + K rounding to K
    int m = (int)u;
    if (m > K - 1) m = K - 1;
    w = u - (float)m;
    g0 = m - P + 1;
    if (g0 < 0) g0 += K;
}

// grid points of shared-memory tile per spreading / gathering thread
// (dynamic shared memory)
constexpr int kTilePerThread = 40;

// The grid patch a block's atoms touch.  Every thread of the block calls it
// (it holds block barriers).  g: the atom's first stencil point (wrapped);
// rel: its offset from the block's first charged atom, unwrapped to the
// nearest periodic copy.  Returns 0 when no atom of the block is charged, 1
// when the patch (ex x ey x ez points from lo) fits `cap` points and all
// charged atoms share one system, 2 otherwise.
struct Patch {
    int first, sys, ok, ref[3], lo[3], hi[3];
};

template <int P>
__device__ __forceinline__ int block_patch(Patch &sp, bool active, int sys, const int (&g)[3],
                                           const int (&K)[3], int (&rel)[3], long long cap,
                                           int &ex, int &ey, int &ez) {
    if (threadIdx.x == 0) {
        sp.first = 0x7fffffff;
        sp.ok = 1;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            sp.lo[d] = 0x7fffffff;
            sp.hi[d] = -0x7fffffff;
        }
    }
    __syncthreads();
    if (active) atomicMin(&sp.first, (int)threadIdx.x);
    __syncthreads();
    if (sp.first == 0x7fffffff) return 0;
    if ((int)threadIdx.x == sp.first) {
        sp.sys = sys;
#pragma unroll
        for (int d = 0; d < 3; ++d) sp.ref[d] = g[d];
    }
    __syncthreads();
    if (active) {
        if (sys != sp.sys) sp.ok = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            int r = g[d] - sp.ref[d];
            if (2 * r > K[d]) r -= K[d];
            if (2 * r < -K[d]) r += K[d];
            rel[d] = r;
            atomicMin(&sp.lo[d], r);
            atomicMax(&sp.hi[d], r);
        }
    }
    __syncthreads();
    ex = sp.hi[0] - sp.lo[0] + P;
    ey = sp.hi[1] - sp.lo[1] + P;
    ez = sp.hi[2] - sp.lo[2] + P;
    return (sp.ok && (long long)ex * ey * ez <= cap) ? 1 : 2;
}

// grid index of patch point t (x-major, z fastest), wrapped into the box
__device__ __forceinline__ size_t patch_point(const Patch &sp, int t, int ey, int ez, int K0,
                                              int K1, int K2) {
    const int lz = t % ez, ly = (t / ez) % ey, lx = t / (ez * ey);
    int gx = sp.ref[0] + sp.lo[0] + lx, gy = sp.ref[1] + sp.lo[1] + ly,
        gz = sp.ref[2] + sp.lo[2] + lz;
    gx += gx < 0 ? K0 : 0;
    gx -= gx >= K0 ? K0 : 0;
    gy += gy < 0 ? K1 : 0;
    gy -= gy >= K1 ? K1 : 0;
    gz += gz < 0 ? K2 : 0;
    gz -= gz >= K2 ? K2 : 0;
    return ((size_t)gx * K1 + gy) * K2 + gz;
}

// Charge spreading through tiles.  Atoms arrive in cluster order, so a block's atoms sit in
// a compact patch of the grid: the block accumulates its p^3 contributions per
// atom into an int64 tile in shared memory (shared atomics) and then adds each
// nonzero tile point to the system's grid with one global atomic -- about 30
// instead of 64 global atomics per atom at order 4.  A block whose patch does
// not fit the tile, or that spans two systems, adds straight to the grid.  All
// sums are of the same int64 contributions, so both paths give the same grid
// bit for bit.
template <int P>
__global__ void __launch_bounds__(256) k_spread(PmeArgs a) {
    extern __shared__ unsigned long long tile[];
    __shared__ Patch sp;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const float4 p = k < a.n_pad ? a.xq[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const bool active = k < a.n_pad && p.w != 0.f;  // padding slots and uncharged atoms add nothing
    int sys = -1, g[3] = {0, 0, 0}, K[3] = {1, 1, 1};
    float th[3][P];
    if (active) {
        sys = a.cl_sys[k / kCluster];
        const SysDev &sd = a.sys[sys];
        const float xs[3] = {p.x, p.y, p.z};
        float dth[P], w;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            K[d] = sd.K[d];
            frac<P>(xs[d], sd.kl[d], K[d], g[d], w);
            spline<P>(w, th[d], dth);
        }
    }
    int rel[3] = {0, 0, 0}, ex = 0, ey = 0, ez = 0;
    const int mode = block_patch<P>(sp, active, sys, g, K, rel,
                                    (long long)kTilePerThread * blockDim.x, ex, ey, ez);
    if (mode == 0) return;  // nothing charged in this block
    const int npts = ex * ey * ez;
    const bool tiled = mode == 1;
    if (!tiled) {
        if (!active) return;
        unsigned long long *grid = a.grid_i + a.sys[sys].grid_off;
        int iz[P];
#pragma unroll
        for (int c = 0; c < P; ++c) iz[c] = (g[2] + c) >= K[2] ? g[2] + c - K[2] : g[2] + c;
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const int ga = (g[0] + i) >= K[0] ? g[0] + i - K[0] : g[0] + i;
            const float qa = p.w * th[0][i];
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const int gb = (g[1] + j) >= K[1] ? g[1] + j - K[1] : g[1] + j;
                const float qab = qa * th[1][j];
                unsigned long long *row = grid + ((size_t)ga * K[1] + gb) * K[2];
#pragma unroll
                for (int c = 0; c < P; ++c) fix_red(&row[iz[c]], to_fix(qab * th[2][c]));
            }
        }
        return;
    }
    for (int t = threadIdx.x; t < npts; t += blockDim.x) tile[t] = 0ull;
    __syncthreads();
    if (active) {
        const int bx = rel[0] - sp.lo[0], by = rel[1] - sp.lo[1], bz = rel[2] - sp.lo[2];
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const float qa = p.w * th[0][i];
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const float qab = qa * th[1][j];
                unsigned long long *row = tile + ((size_t)(bx + i) * ey + (by + j)) * ez + bz;
#pragma unroll
                for (int c = 0; c < P; ++c)
                    atomicAdd(&row[c], (unsigned long long)to_fix(qab * th[2][c]));
            }
        }
    }
    __syncthreads();
    const SysDev &sd = a.sys[sp.sys];
    unsigned long long *grid = a.grid_i + sd.grid_off;
    for (int t = threadIdx.x; t < npts; t += blockDim.x) {
        const unsigned long long v = tile[t];
        if (v != 0ull) fix_red(&grid[patch_point(sp, t, ey, ez, sd.K[0], sd.K[1], sd.K[2])], (long long)v);
    }
}

// Charge spreading without tiles.  A warp takes a cluster (or a half, a quarter
// of one where clusters are few): each lane works out its atom's spline weights
// and wrapped grid indices into shared memory, then the warp adds one atom at a
// time, 32 / P rows of P neighbouring z points per instruction.  A row's points
// share one or two 32-byte sectors, so an instruction's adds reach L2 as 8 to 16
// sector updates instead of the 32 of a thread per atom, which is what bounds
// spreading; the conversions to fixed point come from FP32 adds (to_fix_alu), the
// next bound.  The contributions are those of k_spread, bit for bit.  Order 4:
// 1M atoms 266 -> 130 us, 88k 36 -> 18, 40 boxes of 1.5k-12k 62 -> 30, 2,700 atoms
// 11.3 -> 5.5.
constexpr int kRowWarps = 4;  // warps per block

template <int P>
__global__ void __launch_bounds__(32 * kRowWarps) k_spread_rows(PmeArgs a, int n_warps, int sub) {
    constexpr int kStride = 6 * P + 1;  // odd: the lanes' stores hit distinct banks
    constexpr int kRows = 32 / P;       // rows per instruction
    __shared__ float s_w[kRowWarps][32 * kStride];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warp = blockIdx.x * kRowWarps + w;
    if (warp >= n_warps) return;  // whole warps leave: no block barrier below
    const int n_at = 32 / sub, cluster = warp / sub;
    const int k = cluster * kCluster + (warp % sub) * n_at + lane;
    const float4 p = lane < n_at ? a.xq[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    unsigned active = __ballot_sync(0xffffffffu, p.w != 0.f);  // padding and uncharged atoms add nothing
    if (active == 0u) return;
    const SysDev &sd = a.sys[a.cl_sys[cluster]];
    if (p.w != 0.f) {
        float *const mine = s_w[w] + lane * kStride;
        int *const at = (int *)(mine + 3 * P);
        const float xs[3] = {p.x, p.y, p.z};
        const int stride[3] = {sd.K[1] * sd.K[2], sd.K[2], 1};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float th[P], dth[P], f;
            int g;
            const int K = sd.K[d];
            frac<P>(xs[d], sd.kl[d], K, g, f);
            spline<P>(f, th, dth);
#pragma unroll
            for (int c = 0; c < P; ++c) {
                mine[d * P + c] = d == 0 ? p.w * th[c] : th[c];
                at[d * P + c] = (g + c >= K ? g + c - K : g + c) * stride[d];
            }
        }
    }
    __syncwarp();
    unsigned long long *const grid = a.grid_i + sd.grid_off;
    const int r = lane / P, c = lane % P;
    while (active) {
        const int t = __ffs(active) - 1;
        active &= active - 1;
        const float *const wt = s_w[w] + t * kStride;
        const int *const at = (const int *)(wt + 3 * P);
        const float wz = wt[2 * P + c];
        const int oz = at[2 * P + c];
#pragma unroll
        for (int r0 = 0; r0 < P * P; r0 += kRows) {
            const int row = r0 + r;
            if (r < kRows && row < P * P) {
                const int i = row / P, j = row % P;
                fix_red(&grid[at[i] + at[P + j] + oz], to_fix_alu(wt[i] * wt[P + j] * wz));
            }
        }
    }
}

__global__ void k_grid_convert(long long *__restrict__ gi, float *__restrict__ gr,
                               long long total) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    gr[i] = __ll2float_rn(gi[i]) * (1.0f / kFixScaleF);
    gi[i] = 0;
}

// one size group: `count` complex grids starting nc elements apart (the
// padded stride; padding carries G = 0); grid g belongs to system sys_ids[g]
template <bool ENERGY>
__global__ void __launch_bounds__(256) k_convolve(float2 *__restrict__ gc,
                                                  const float *__restrict__ G, long long total,
                                                  long long nc, int Kh, int K2,
                                                  const int *__restrict__ sys_ids,
                                                  long long *__restrict__ energy) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double e = 0.0;
    int q = -1;
    if (i < total) {
        const float2 c = gc[i];
        const float g = G[i];
        // G = 0 (k = 0 and the padding between members): the element is
        // dropped whatever it holds
        const bool live = g != 0.f;
        if (ENERGY) {
            const int kz = (int)((i % nc) % Kh);
            const float wgt = (kz == 0 || (2 * kz == K2)) ? 1.0f : 2.0f;
            e = live ? (double)(0.5f * wgt * g * (c.x * c.x + c.y * c.y)) : 0.0;
            q = sys_ids[i / nc];
        }
        gc[i] = live ? make_float2(c.x * g, c.y * g) : make_float2(0.f, 0.f);
    }
    if (ENERGY) {
        const double v[1] = {e};
        const int slot[1] = {MDG_TERM_COUL_RECIP};
        block_energy_add<1>(energy, q, v, slot);
    }
}

// Force gathering where clusters are few.  A warp takes 8 atoms: it reads the
// potential around one after the other, 32 / P rows of P neighbouring z points per
// load, into shared memory, and then 8 lanes sum an atom each from there, in
// k_gather's order: the same forces bit for bit.  Bound by latency, which four
// times the warps and independent loads shorten: 2,700 atoms 8.6 -> 6.2 us.  A
// thread per atom has more loads in flight per SM once it fills the GPU: 88k atoms
// 12.3 against 16.2 us here, 1M 73 against 134, 40 boxes of 1.5k-12k 22 against 26;
// the line lies where a warp per 8 atoms fills every SM with about 32 warps.
constexpr int kGatherAtoms = 8;        // per warp
constexpr int kGatherRowsBelow = 1200; // clusters

template <int P>
__global__ void __launch_bounds__(32 * kRowWarps) k_gather_rows(PmeArgs a, int n_warps) {
    constexpr int n_at = kGatherAtoms;
    constexpr int kVal = P * P * P | 1;   // odd strides: a lane per atom is conflict-free
    constexpr int kIdx = 3 * P | 1;
    constexpr int kRows = 32 / P;         // rows per load
    constexpr int kIts = (P * P + kRows - 1) / kRows;
    constexpr int kUnroll = P == 4 ? 4 : 1;  // atoms whose loads are in flight together
    extern __shared__ float s_gather[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *const val = s_gather + w * n_at * (kVal + kIdx);
    int *const idx = (int *)(val + n_at * kVal);
    const int warp = blockIdx.x * kRowWarps + w, per = kCluster / n_at;
    const int cluster = warp / per;
    const int k = cluster * kCluster + (warp % per) * n_at + lane;
    const bool mine = warp < n_warps && lane < n_at;
    const float4 p = mine ? a.xq[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const bool active = p.w != 0.f;  // not a padding slot or an uncharged atom
    const unsigned todo = __ballot_sync(0xffffffffu, active);
    const SysDev &sd = a.sys[warp < n_warps ? a.cl_sys[cluster] : 0];
    float th[3][P], dth[3][P];
    if (active) {
        const float xs[3] = {p.x, p.y, p.z};
        const int stride[3] = {sd.K[1] * sd.K[2], sd.K[2], 1};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float f;
            int g;
            const int K = sd.K[d];
            frac<P>(xs[d], sd.kl[d], K, g, f);
            spline<P>(f, th[d], dth[d]);
#pragma unroll
            for (int c = 0; c < P; ++c)
                idx[lane * kIdx + d * P + c] = (g + c >= K ? g + c - K : g + c) * stride[d];
        }
    }
    __syncwarp();
    wait_for_previous();  // (the positions are older than the chain of transforms)
    if (todo == 0u) return;
    const float *const phi = a.phi + sd.grid_off;
    const int r = lane / P, c = lane % P;
    for (int t0 = 0; t0 < n_at; t0 += kUnroll) {
        float v[kUnroll][kIts];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const int t = t0 + u;
            const int *const at = idx + t * kIdx;
#pragma unroll
            for (int q = 0; q < kIts; ++q) {
                const int row = q * kRows + r;
                if (((todo >> t) & 1u) && r < kRows && row < P * P)
                    v[u][q] = __ldg(&phi[at[row / P] + at[P + row % P] + at[2 * P + c]]);
            }
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
#pragma unroll
            for (int q = 0; q < kIts; ++q) {
                const int row = q * kRows + r;
                if (r < kRows && row < P * P) val[(t0 + u) * kVal + row * P + c] = v[u][q];
            }
    }
    __syncwarp();
    if (!active) return;
    const float *const mv = val + lane * kVal;
    float fx = 0.f, fy = 0.f, fz = 0.f;
#pragma unroll
    for (int i = 0; i < P; ++i) {
#pragma unroll
        for (int j = 0; j < P; ++j) {
            float sz = 0.f, sdz = 0.f;
#pragma unroll
            for (int q = 0; q < P; ++q) {
                const float u = mv[(i * P + j) * P + q];
                sz = fmaf(th[2][q], u, sz);
                sdz = fmaf(dth[2][q], u, sdz);
            }
            fx = fmaf(dth[0][i] * th[1][j], sz, fx);
            fy = fmaf(th[0][i] * dth[1][j], sz, fy);
            fz = fmaf(th[0][i] * th[1][j], sdz, fz);
        }
    }
    fx *= -p.w * sd.kl[0] * a.weight;
    fy *= -p.w * sd.kl[1] * a.weight;
    fz *= -p.w * sd.kl[2] * a.weight;
    fix_red(&a.f[k], to_fix(fx));
    fix_red(&a.f[a.n_pad + k], to_fix(fy));
    fix_red(&a.f[2 * a.n_pad + k], to_fix(fz));
}

// Force gathering, a thread per atom; with tiles a block first copies the
// potential on its grid patch into shared memory (row by row), then every atom
// reads its p^3 values from there; a block whose patch does not fit reads the grid
// directly.  The arithmetic is the same either way, so both paths give the same
// forces.
template <int P>
__global__ void __launch_bounds__(256) k_gather(PmeArgs a) {
    extern __shared__ float ptile[];
    __shared__ Patch sp;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const float4 p = k < a.n_pad ? a.xq[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const bool active = k < a.n_pad && p.w != 0.f;  // padding slots and uncharged atoms
    int sys = -1, g[3] = {0, 0, 0}, K[3] = {1, 1, 1};
    float th[3][P], dth[3][P];
    float kl[3] = {0.f, 0.f, 0.f};
    size_t goff = 0;
    if (active) {
        sys = a.cl_sys[k / kCluster];
        const SysDev &sd = a.sys[sys];
        const float xs[3] = {p.x, p.y, p.z};
        float w;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            K[d] = sd.K[d];
            kl[d] = sd.kl[d];
            frac<P>(xs[d], sd.kl[d], K[d], g[d], w);
            spline<P>(w, th[d], dth[d]);
        }
        goff = sd.grid_off;
    }
    int rel[3] = {0, 0, 0}, ex = 0, ey = 0, ez = 0;
    const int mode = a.tile_gather ? block_patch<P>(sp, active, sys, g, K, rel,
                                                    (long long)2 * kTilePerThread * blockDim.x,
                                                    ex, ey, ez)
                                   : 2;
    if (mode == 0) return;
    const bool tiled = mode == 1;
    if (tiled) {
        const SysDev &sd = a.sys[sp.sys];
        const float *phi = a.phi + sd.grid_off;
        const int npts = ex * ey * ez;
        for (int t = threadIdx.x; t < npts; t += blockDim.x)
            ptile[t] = __ldg(&phi[patch_point(sp, t, ey, ez, sd.K[0], sd.K[1], sd.K[2])]);
        __syncthreads();
    }
    if (!active) return;
    const float *phi = a.phi + goff;
    const int bx = tiled ? rel[0] - sp.lo[0] : 0, by = tiled ? rel[1] - sp.lo[1] : 0,
              bz = tiled ? rel[2] - sp.lo[2] : 0;
    int iz[P];
#pragma unroll
    for (int c = 0; c < P; ++c) iz[c] = (g[2] + c) >= K[2] ? g[2] + c - K[2] : g[2] + c;
    float fx = 0.f, fy = 0.f, fz = 0.f;
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const int ga = (g[0] + i) >= K[0] ? g[0] + i - K[0] : g[0] + i;
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const int gb = (g[1] + j) >= K[1] ? g[1] + j - K[1] : g[1] + j;
            float v[P];
            if (tiled) {
                const float *trow = ptile + ((size_t)(bx + i) * ey + (by + j)) * ez + bz;
#pragma unroll
                for (int c = 0; c < P; ++c) v[c] = trow[c];
            } else {
                const float *row = phi + ((size_t)ga * K[1] + gb) * K[2];
#pragma unroll
                for (int c = 0; c < P; ++c) v[c] = __ldg(&row[iz[c]]);
            }
            float sz = 0.f, sdz = 0.f;
#pragma unroll
            for (int c = 0; c < P; ++c) {
                sz = fmaf(th[2][c], v[c], sz);
                sdz = fmaf(dth[2][c], v[c], sdz);
            }
            fx = fmaf(dth[0][i] * th[1][j], sz, fx);
            fy = fmaf(th[0][i] * dth[1][j], sz, fy);
            fz = fmaf(th[0][i] * th[1][j], sdz, fz);
        }
    }
    fx *= -p.w * kl[0] * a.weight;
    fy *= -p.w * kl[1] * a.weight;
    fz *= -p.w * kl[2] * a.weight;
    fix_red(&a.f[k], to_fix(fx));
    fix_red(&a.f[a.n_pad + k], to_fix(fy));
    fix_red(&a.f[2 * a.n_pad + k], to_fix(fz));
}

// host FP64 B-spline values, same recursion as the device
void spline_host(double w, int P, double *th) {
    std::vector<double> a(P + 1, 0.0), b(P + 1, 0.0);
    a[0] = 1 - w;
    a[1] = w;
    for (int n = 3; n <= P; ++n) {
        double div = 1.0 / (n - 1);
        for (int i = 0; i < n; ++i) {
            double left = i >= 1 ? a[i - 1] : 0.0, right = i <= n - 2 ? a[i] : 0.0;
            b[i] = div * ((w + n - 1 - i) * left + (i + 1 - w) * right);
        }
        for (int i = 0; i < n; ++i) a[i] = b[i];
    }
    for (int i = 0; i < P; ++i) th[i] = a[i];
}

std::vector<double> bspline_moduli(int K, int P) {
    std::vector<double> th(P), mod(K);
    spline_host(0.0, P, th.data());
    const double pi = 3.14159265358979323846;
    for (int m = 0; m < K; ++m) {
        double sr = 0, si = 0;
        for (int k = 0; k <= P - 2; ++k) {
            double mk = th[P - 2 - k];  // M_p(k+1)
            sr += mk * std::cos(2 * pi * m * k / K);
            si += mk * std::sin(2 * pi * m * k / K);
        }
        mod[m] = sr * sr + si * si;
    }
    for (int m = 0; m < K; ++m)
        if (mod[m] < 1e-10) mod[m] = 0.5 * (mod[(m - 1 + K) % K] + mod[(m + 1) % K]);
    return mod;
}

}  // namespace

void pme_free(mdg_system *s) {
    Pme &p = s->pme;
    for (PmeGroup &g : p.groups) {
        if (g.plan_f) cufftDestroy(g.plan_f);
        if (g.plan_b) cufftDestroy(g.plan_b);
        if (g.sys_ids) cudaFree(g.sys_ids);
    }
    p.groups.clear();
    fft_free(p.fft);
    cudaFree(p.grid_i);
    cudaFree(p.grid_r);
    cudaFree(p.grid_c);
    cudaFree(p.influence);
    p.grid_i = nullptr;
    p.grid_r = nullptr;
    p.grid_c = nullptr;
    p.influence = nullptr;
    p.grid_total = p.cgrid_total = 0;
}

// Grids, cuFFT plans and influence functions of every system.  grids holds
// (K0, K1, K2) per system.  Systems with the same grid share one batched plan
// pair (a size group); the grids of a group lie back to back, so one R2C and
// one C2R transform the whole group.  The influence function is built in FP64
// on the host from each system's own box and stored as float.
int pme_setup(mdg_system *s, const int *grids) {
    Pme &p = s->pme;
    pme_free(s);
    const int ns = s->n_sys;
    std::vector<std::vector<int>> members;
    std::vector<int> gk;
    for (int q = 0; q < ns; ++q) {
        size_t g = 0;
        for (; g < members.size(); ++g)
            if (gk[3 * g] == grids[3 * q] && gk[3 * g + 1] == grids[3 * q + 1] &&
                gk[3 * g + 2] == grids[3 * q + 2])
                break;
        if (g == members.size()) {
            members.emplace_back();
            gk.insert(gk.end(), grids + 3 * q, grids + 3 * q + 3);
        }
        members[g].push_back(q);
    }
    long long roff = 0, coff = 0;
    for (size_t g = 0; g < members.size(); ++g) {
        PmeGroup grp;
        for (int d = 0; d < 3; ++d) grp.K[d] = gk[3 * g + d];
        grp.count = (int)members[g].size();
        // every grid starts on a 256-byte boundary (cuFFT rejects misaligned
        // pointers): member strides are rounded up, the gaps stay zero
        const long long nr = round_up((long long)grp.K[0] * grp.K[1] * grp.K[2], 64);
        const long long nc = round_up((long long)grp.K[0] * grp.K[1] * (grp.K[2] / 2 + 1), 32);
        grp.nr_stride = nr;
        grp.nc_stride = nc;
        grp.grid_off = roff;
        grp.cgrid_off = coff;
        for (int m = 0; m < grp.count; ++m) {
            SysDev &d = s->sys_h[members[g][m]];
            for (int k = 0; k < 3; ++k) {
                d.K[k] = grp.K[k];
                d.kl[k] = (float)(grp.K[k] / d.Ld[k]);
            }
            d.grid_off = roff + m * nr;
            d.cgrid_off = coff + m * nc;
        }
        roff += grp.count * nr;
        coff += grp.count * nc;
        p.groups.push_back(grp);
    }
    p.grid_total = roff;
    p.cgrid_total = coff;
    // the spreading tile of a 256-thread block is above the 48 KB default
    const int tile_max = (int)(sizeof(unsigned long long) * kTilePerThread * 256);
    if (cudaFuncSetAttribute(k_spread<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_max) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_spread<5>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_max) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_spread<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_max) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_gather<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_max) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_gather<5>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_max) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_gather<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_max) !=
            cudaSuccess)
        return MDG_ERR_CUDA;
    if (cudaMalloc(&p.grid_i, roff * sizeof(long long)) != cudaSuccess) return MDG_ERR_NOMEM;
    if (cudaMalloc(&p.grid_r, roff * sizeof(float)) != cudaSuccess) return MDG_ERR_NOMEM;
    if (cudaMalloc(&p.grid_c, coff * sizeof(float2)) != cudaSuccess) return MDG_ERR_NOMEM;
    if (cudaMalloc(&p.influence, coff * sizeof(float)) != cudaSuccess) return MDG_ERR_NOMEM;
    // the padding between members' grids is never written by cuFFT: zero it
    // once (and the convolution keeps it zero), so no stale bits of a freed
    // buffer reach the energy sum
    if (cudaMemset(p.grid_i, 0, roff * sizeof(long long)) != cudaSuccess ||
        cudaMemset(p.grid_r, 0, roff * sizeof(float)) != cudaSuccess ||
        cudaMemset(p.grid_c, 0, coff * sizeof(float2)) != cudaSuccess)
        return MDG_ERR_CUDA;
    const double pi = 3.14159265358979323846;
    const double b2 = p.beta * p.beta;
    std::vector<float> G(coff);
    std::vector<int> own;  // systems whose transforms run in mdg_fft.cu
    for (size_t g = 0; g < members.size(); ++g) {
        PmeGroup &grp = p.groups[g];
        const int K0 = grp.K[0], K1 = grp.K[1], K2 = grp.K[2], Kh = K2 / 2 + 1;
        int n[3] = {K0, K1, K2}, nh[3] = {K0, K1, Kh};
        grp.own = fft_supported(grp.K);
        if (grp.own) own.insert(own.end(), members[g].begin(), members[g].end());
        else if (cufftPlanMany(&grp.plan_f, 3, n, n, 1, (int)grp.nr_stride, nh, 1, (int)grp.nc_stride,
                          CUFFT_R2C, grp.count) != CUFFT_SUCCESS ||
            cufftPlanMany(&grp.plan_b, 3, n, nh, 1, (int)grp.nc_stride, n, 1, (int)grp.nr_stride,
                          CUFFT_C2R, grp.count) != CUFFT_SUCCESS)
            return MDG_ERR_CUFFT;
        if (cudaMalloc(&grp.sys_ids, sizeof(int) * grp.count) != cudaSuccess) return MDG_ERR_NOMEM;
        if (cudaMemcpy(grp.sys_ids, members[g].data(), sizeof(int) * grp.count,
                       cudaMemcpyHostToDevice) != cudaSuccess)
            return MDG_ERR_CUDA;
        auto m0 = bspline_moduli(K0, p.order), m1 = bspline_moduli(K1, p.order),
             m2 = bspline_moduli(K2, p.order);
        for (int q : members[g]) {
            const SysDev &d = s->sys_h[q];
            const double *L = d.Ld;
            const double V = L[0] * L[1] * L[2];
            float *Gs = G.data() + d.cgrid_off;
            for (int a = 0; a < K0; ++a) {
                const double fa = (a <= K0 / 2 ? a : a - K0) / L[0];
                for (int b = 0; b < K1; ++b) {
                    const double fb = (b <= K1 / 2 ? b : b - K1) / L[1];
                    for (int c = 0; c < Kh; ++c) {
                        const double fc = c / L[2];
                        const double msq = fa * fa + fb * fb + fc * fc;
                        double gv = 0.0;
                        if (msq > 0)
                            gv = std::exp(-pi * pi * msq / b2) / (pi * V * msq) /
                                 (m0[a] * m1[b] * m2[c]);
                        Gs[((size_t)a * K1 + b) * Kh + c] = (float)gv;
                    }
                }
            }
        }
    }
    if (cudaMemcpy(p.influence, G.data(), coff * sizeof(float), cudaMemcpyHostToDevice) !=
        cudaSuccess)
        return MDG_ERR_CUDA;
    const int rc = fft_setup(p.fft, s->sys_h, own);
    return rc ? rc : upload_sys_table(s);
}

cudaError_t launch_pme(mdg_system *s, int energy, int *cufft_status) {
    Pme &p = s->pme;
    *cufft_status = CUFFT_SUCCESS;
    PmeArgs a;
    a.xq = s->xq;
    a.sys = s->sys_dev;
    a.cl_sys = s->cl_sys;
    a.n_pad = s->n_pad;
    a.grid_i = (unsigned long long *)p.grid_i;
    a.phi = p.grid_r;
    a.f = s->slow_target ? s->slow_target : s->f;  // the learned form's outer steps: apart
    const bool tile_spread = s->pme_tiles & 1;
    a.tile_gather = (s->pme_tiles >> 1) & 1;
    a.weight = s->recip_weight;
    const int tb = 256;
    const int ab = s->pme_block, nb = (s->n_pad + ab - 1) / ab;  // per-atom kernels
    // dynamic shared memory only for the kernels that stage a tile (it limits
    // their occupancy otherwise for nothing)
    const size_t tile_bytes = sizeof(unsigned long long) * kTilePerThread * ab;
    const size_t spread_smem = tile_spread ? tile_bytes : 0;
    const size_t gather_smem = a.tile_gather ? tile_bytes : 0;
    cudaStream_t st = s->stream;
    if (!tile_spread) {
        // enough warps for every SM: clusters split in up to four where few
        const int sub = s->n_clusters < 1200 ? 4 : s->n_clusters < 4800 ? 2 : 1;
        const int nw = s->n_clusters * sub, nbr = (nw + kRowWarps - 1) / kRowWarps;
        switch (p.order) {
            case 4: k_spread_rows<4><<<nbr, 32 * kRowWarps, 0, st>>>(a, nw, sub); break;
            case 5: k_spread_rows<5><<<nbr, 32 * kRowWarps, 0, st>>>(a, nw, sub); break;
            case 6: k_spread_rows<6><<<nbr, 32 * kRowWarps, 0, st>>>(a, nw, sub); break;
            default: return cudaErrorInvalidValue;
        }
    } else {
        switch (p.order) {
            case 4: k_spread<4><<<nb, ab, spread_smem, st>>>(a); break;
            case 5: k_spread<5><<<nb, ab, spread_smem, st>>>(a); break;
            case 6: k_spread<6><<<nb, ab, spread_smem, st>>>(a); break;
            default: return cudaErrorInvalidValue;
        }
    }
    s->launches += 1;
    // weight 0 (an impulse inner step that only reports the energy): the
    // potential grid is never gathered, so the way back is skipped
    cudaError_t fe = fft_convolve(s, p.fft, energy, a.weight != 0.f);
    if (fe != cudaSuccess) return fe;
    for (PmeGroup &g : p.groups) {
        if (g.own) continue;
        const long long n = g.nr_stride * g.count;
        k_grid_convert<<<(unsigned)((n + tb - 1) / tb), tb, 0, st>>>(p.grid_i + g.grid_off,
                                                                     p.grid_r + g.grid_off, n);
        s->launches += 1;
    }
    for (PmeGroup &g : p.groups) {
        if (g.own) continue;
        cufftResult r = cufftSetStream(g.plan_f, st);
        if (r == CUFFT_SUCCESS)
            r = cufftExecR2C(g.plan_f, p.grid_r + g.grid_off, (cufftComplex *)(p.grid_c + g.cgrid_off));
        if (r != CUFFT_SUCCESS) {
            *cufft_status = r;
            return cudaGetLastError();
        }
    }
    for (PmeGroup &g : p.groups) {
        if (g.own) continue;
        const int Kh = g.K[2] / 2 + 1;
        const long long nc = g.nc_stride;  // padding elements carry G = 0
        const long long totc = nc * g.count;
        const unsigned nbc = (unsigned)((totc + tb - 1) / tb);
        if (energy)
            k_convolve<true><<<nbc, tb, 0, st>>>(p.grid_c + g.cgrid_off, p.influence + g.cgrid_off,
                                                 totc, nc, Kh, g.K[2], g.sys_ids, s->energy);
        else
            k_convolve<false><<<nbc, tb, 0, st>>>(p.grid_c + g.cgrid_off,
                                                  p.influence + g.cgrid_off, totc, nc, Kh, g.K[2],
                                                  g.sys_ids, s->energy);
        s->launches += 1;
    }
    for (PmeGroup &g : p.groups) {
        if (a.weight == 0.f) break;
        if (g.own) continue;
        cufftResult r = cufftSetStream(g.plan_b, st);
        if (r == CUFFT_SUCCESS)
            r = cufftExecC2R(g.plan_b, (cufftComplex *)(p.grid_c + g.cgrid_off), p.grid_r + g.grid_off);
        if (r != CUFFT_SUCCESS) {
            *cufft_status = r;
            return cudaGetLastError();
        }
    }
    if (a.weight != 0.f) {  // weight 0: the energy alone
        // behind this file's transforms alone: an ordinary launch waits for
        // everything before it
        const bool chained = std::all_of(p.groups.begin(), p.groups.end(),
                                         [](const PmeGroup &g) { return g.own; });
        auto launch = [&](auto rows, auto direct, int P) -> cudaError_t {
            if (a.tile_gather || s->n_clusters >= kGatherRowsBelow) {
                direct<<<nb, ab, gather_smem, st>>>(a);
                return cudaGetLastError();
            }
            const int nw = s->n_clusters * (kCluster / kGatherAtoms);
            const int blocks = (nw + kRowWarps - 1) / kRowWarps;
            const size_t smem = sizeof(float) * kRowWarps * kGatherAtoms *
                                ((P * P * P | 1) + (3 * P | 1));
            if (chained) return launch_after(rows, blocks, 32 * kRowWarps, smem, st, a, nw);
            rows<<<blocks, 32 * kRowWarps, smem, st>>>(a, nw);
            return cudaGetLastError();
        };
        cudaError_t ge = cudaSuccess;
        switch (p.order) {
            case 4: ge = launch(k_gather_rows<4>, k_gather<4>, 4); break;
            case 5: ge = launch(k_gather_rows<5>, k_gather<5>, 5); break;
            case 6: ge = launch(k_gather_rows<6>, k_gather<6>, 6); break;
            default: break;
        }
        if (ge != cudaSuccess) return ge;
        s->launches += 1;
    }
    return cudaGetLastError();
}

}  // namespace mdg
