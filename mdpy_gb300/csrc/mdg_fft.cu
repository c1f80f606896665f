// mdg_fft.cu -- the PME grids' Fourier transforms, for every system of a batch
// in three launches.
//
// The convolution phi = IFFT(G FFT(rho)) of a grid K0 x K1 x K2 (x slowest)
// needs 8 dependent kernels with a transform library (int64 -> float, three
// passes forward, the influence function, three passes back), and as many
// again for every other grid size of a batch.  At 30^3 to 100^3 points each
// takes 3 to 6 us, nearly all of it launch and drain.  Here:
//
//   k_fft_planes<fwd>  one block per x plane: int64 charges -> float (and the
//                      int64 grid zeroed), real transform along z, complex
//                      along y, all in shared memory; the half spectrum's
//                      plane out
//   k_fft_columns      one block per 8 columns along x: forward, times G (with
//                      the energy sum), back
//   k_fft_planes<inv>  back along y and z: the potential's plane out
//
// Each line is a mixed-radix Stockham transform (radices 4, 2, 3, 5) between
// two shared-memory buffers; two real z lines share one complex transform.
// Bound by latency at these sizes (10 barriers a plane, one plane per SM up to
// 152 planes), by shared-memory throughput on larger planes.  Grids with other
// prime factors, and larger planes (fft_supported), keep the library's plans.
#include <algorithm>
#include <cmath>
#include <vector>

#include "mdg_internal.cuh"

namespace mdg {
namespace {

constexpr int kCols = 8;             // columns per block of k_fft_columns
constexpr int kPlaneThreads = 128;
constexpr int kPlaneMax = 1300;      // points of the largest plane taken
constexpr size_t kSmemMax = 200 * 1024;
constexpr int kLoad = 8;             // charges (of each of two lines) a thread loads at once

constexpr int kMaxPasses = 8;  // of a length up to 1024

struct FftArgs {
    const FftBlock *__restrict__ blocks;
    const int4 *__restrict__ plan;       // passes of each length: radix, m, magic_of(N / R), magic_of(m)
    const float2 *__restrict__ tw;       // exp(-2 pi i t / K), t < K
    long long *gi;
    float *gr;
    float2 *gc;
    const float *__restrict__ G;
    long long *energy;
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a * (-i) forward, a * i backward
template <bool INV>
__device__ __forceinline__ float2 rot(float2 a) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <int R, bool INV>
__device__ __forceinline__ void butterfly(float2 (&a)[R]) {
    if constexpr (R == 2) {
        const float2 t = csub(a[0], a[1]);
        a[0] = cadd(a[0], a[1]);
        a[1] = t;
    } else if constexpr (R == 3) {
        const float2 s = cadd(a[1], a[2]), d = rot<INV>(csub(a[1], a[2]));
        const float2 m = make_float2(fmaf(-0.5f, s.x, a[0].x), fmaf(-0.5f, s.y, a[0].y));
        const float h = 0.866025403784438647f;  // sin(2 pi / 3)
        a[0] = cadd(a[0], s);
        a[1] = make_float2(fmaf(h, d.x, m.x), fmaf(h, d.y, m.y));
        a[2] = make_float2(fmaf(-h, d.x, m.x), fmaf(-h, d.y, m.y));
    } else if constexpr (R == 4) {
        const float2 s02 = cadd(a[0], a[2]), d02 = csub(a[0], a[2]);
        const float2 s13 = cadd(a[1], a[3]), d13 = rot<INV>(csub(a[1], a[3]));
        a[0] = cadd(s02, s13);
        a[1] = cadd(d02, d13);
        a[2] = csub(s02, s13);
        a[3] = csub(d02, d13);
    } else {
        // cos and sin of 2 pi / 5 and 4 pi / 5
        const float c1 = 0.309016994374947424f, c2 = -0.809016994374947424f,
                    s1 = 0.951056516295153572f, s2 = 0.587785252292473129f;
        const float2 p = cadd(a[1], a[4]), q = cadd(a[2], a[3]);
        const float2 u = rot<INV>(csub(a[1], a[4])), v = rot<INV>(csub(a[2], a[3]));
        const float2 m1 = make_float2(fmaf(c1, p.x, fmaf(c2, q.x, a[0].x)),
                                      fmaf(c1, p.y, fmaf(c2, q.y, a[0].y)));
        const float2 m2 = make_float2(fmaf(c2, p.x, fmaf(c1, q.x, a[0].x)),
                                      fmaf(c2, p.y, fmaf(c1, q.y, a[0].y)));
        const float2 n1 = make_float2(fmaf(s1, u.x, s2 * v.x), fmaf(s1, u.y, s2 * v.y));
        const float2 n2 = make_float2(fmaf(s2, u.x, -s1 * v.x), fmaf(s2, u.y, -s1 * v.y));
        a[0] = cadd(a[0], cadd(p, q));
        a[1] = cadd(m1, n1);
        a[2] = cadd(m2, n2);
        a[3] = csub(m2, n2);
        a[4] = csub(m1, n1);
    }
}

// idx / d for idx * d < 2^32, magic = floor((2^32 - 1) / d) + 1 (0 for d = 1)
__host__ __device__ __forceinline__ unsigned magic_of(unsigned d) { return 0xffffffffu / d + 1u; }
__device__ __forceinline__ unsigned divide(unsigned idx, unsigned magic) {
    return magic == 0u ? idx : __umulhi(idx, magic);
}

// One radix-R pass of `lines` transforms of length N, m = the product of the
// radices before it: y[g R m + k + p m] = sum_q W_R^{pq} W_{Rm}^{qk} x[j + q N / R],
// j = g m + k.  Element e of line l sits at l ls + e es.  JFAST: neighbouring
// threads take neighbouring j of one line (contiguous lines), else neighbouring
// lines (lines beside each other).
template <int R, bool INV, bool JFAST>
__device__ __forceinline__ void fft_pass(const float2 *__restrict__ src, float2 *__restrict__ dst,
                                         const float2 *__restrict__ tw, int N, int m,
                                         unsigned mg_j, unsigned mg_m, int lines, unsigned mg_l,
                                         int ls, int es) {
    const unsigned nj = divide(N, magic_of(R)), step = divide(nj, mg_m);
    for (unsigned idx = threadIdx.x; idx < nj * lines; idx += blockDim.x) {
        unsigned l, j;
        if (JFAST) {
            l = divide(idx, mg_j);
            j = idx - l * nj;
        } else {
            j = divide(idx, mg_l);
            l = idx - j * lines;
        }
        const unsigned g = divide(j, mg_m), k = j - g * m;
        const float2 *s = src + l * ls + j * es;
        float2 a[R];
#pragma unroll
        for (int q = 0; q < R; ++q) a[q] = s[q * nj * es];
        if (m > 1) {
#pragma unroll
            for (int q = 1; q < R; ++q) {
                float2 w = tw[q * k * step];
                if (INV) w.y = -w.y;
                a[q] = cmul(a[q], w);
            }
        }
        butterfly<R, INV>(a);
        float2 *d = dst + l * ls + (g * R * m + k) * es;
#pragma unroll
        for (int p = 0; p < R; ++p) d[p * m * es] = a[p];
    }
    __syncthreads();
}

// `lines` transforms of length N (2^a 3^b 5^c) from `a`, with `b` as the other
// buffer; returns the buffer that holds the result.  plan: the length's passes
// (in shared memory), ended by radix 0.  The caller has synchronised the block
// after writing `a`.
template <bool INV, bool JFAST>
__device__ __forceinline__ float2 *fft_lines(float2 *a, float2 *b, const float2 *tw,
                                             const int4 *plan, int N, int lines, unsigned mg_l,
                                             int ls, int es) {
    for (int p = 0; p < kMaxPasses && plan[p].x != 0; ++p) {
        const int4 q = plan[p];
        switch (q.x) {
            case 4: fft_pass<4, INV, JFAST>(a, b, tw, N, q.y, q.z, q.w, lines, mg_l, ls, es); break;
            case 2: fft_pass<2, INV, JFAST>(a, b, tw, N, q.y, q.z, q.w, lines, mg_l, ls, es); break;
            case 3: fft_pass<3, INV, JFAST>(a, b, tw, N, q.y, q.z, q.w, lines, mg_l, ls, es); break;
            default: fft_pass<5, INV, JFAST>(a, b, tw, N, q.y, q.z, q.w, lines, mg_l, ls, es);
        }
        float2 *t = a;
        a = b;
        b = t;
    }
    return a;
}

// the fixed-point charge as float, rounded once.  A 64-bit conversion takes 16
// cycles a warp; below 2^32 (a charge of 1 e at a grid point is 1.6e9) a 32-bit
// one gives the same value.
__device__ __forceinline__ float grid_value(long long v) {
    const unsigned long long u = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    if (u >> 32) return __ll2float_rn(v) * (1.0f / kFixScaleF);
    const float f = __uint2float_rn((unsigned)u) * (1.0f / kFixScaleF);
    return v < 0 ? -f : f;
}

__host__ __device__ inline int plane_points(int K1, int K2) {
    const int z = (K1 + 1) / 2 * K2, y = K1 * (K2 / 2 + 1);  // packed z lines; half spectrum
    return z > y ? z : y;
}

template <bool INV>
__global__ void __launch_bounds__(kPlaneThreads) k_fft_planes(FftArgs a) {
    extern __shared__ float2 s_fft[];
    __shared__ int4 s_plan[2][kMaxPasses];
    const FftBlock b = a.blocks[blockIdx.x];
    const int K1 = b.K[1], K2 = b.K[2], Kh = K2 / 2 + 1, pairs = (K1 + 1) / 2;
    float2 *const tw1 = s_fft, *const tw2 = tw1 + K1;
    float2 *A = tw2 + K2, *B = A + plane_points(K1, K2);
    for (int t = threadIdx.x; t < K1; t += blockDim.x) tw1[t] = a.tw[b.tw[1] + t];
    for (int t = threadIdx.x; t < K2; t += blockDim.x) tw2[t] = a.tw[b.tw[2] + t];
    if (threadIdx.x < kMaxPasses) {
        s_plan[0][threadIdx.x] = a.plan[kMaxPasses * b.plan[1] + threadIdx.x];
        s_plan[1][threadIdx.x] = a.plan[kMaxPasses * b.plan[2] + threadIdx.x];
    }
    const int4 *const p1 = s_plan[0], *const p2 = s_plan[1];
    const unsigned mg_h = magic_of(Kh);
    const size_t real0 = b.grid_off + (size_t)b.index * K1 * K2;
    float2 *const gc = a.gc + b.cgrid_off + (size_t)b.index * K1 * Kh;
    wait_for_previous();  // (the tables above do not change)
    if constexpr (!INV) {
        // two z lines (y = 2 p and 2 p + 1) as one complex line
        long long *const gi = a.gi + real0;
        const unsigned mg = magic_of(K2);
        // (kLoad points' loads in flight together: one after another, each
        // waits out the memory latency)
        const unsigned total = pairs * K2;
        for (unsigned t0 = threadIdx.x; t0 < total; t0 += kLoad * blockDim.x) {
            long long u[kLoad], w[kLoad];
#pragma unroll
            for (int i = 0; i < kLoad; ++i) {
                const unsigned t = t0 + i * blockDim.x, p = divide(t, mg);
                const unsigned e = 2 * p * K2 + (t - p * K2);
                u[i] = t < total ? gi[e] : 0;
                w[i] = t < total && 2 * p + 1 < (unsigned)K1 ? gi[e + K2] : 0;
            }
#pragma unroll
            for (int i = 0; i < kLoad; ++i) {
                const unsigned t = t0 + i * blockDim.x, p = divide(t, mg);
                const unsigned e = 2 * p * K2 + (t - p * K2);
                if (t >= total) break;
                gi[e] = 0;
                if (2 * p + 1 < (unsigned)K1) gi[e + K2] = 0;
                A[t] = make_float2(grid_value(u[i]), grid_value(w[i]));
            }
        }
        __syncthreads();
        float2 *r = fft_lines<false, true>(A, B, tw2, p2, K2, pairs, 0u, K2, 1);
        float2 *o = r == A ? B : A;
        // the two lines' half spectra: (Z[k] +- conj Z[K2 - k]) / 2
        for (unsigned t = threadIdx.x; t < (unsigned)(pairs * Kh); t += blockDim.x) {
            const unsigned p = divide(t, mg_h), k = t - p * Kh;
            const float2 u = r[p * K2 + k], w = r[p * K2 + (k == 0 ? 0 : K2 - k)];
            o[2 * p * Kh + k] = make_float2(0.5f * (u.x + w.x), 0.5f * (u.y - w.y));
            if (2 * p + 1 < (unsigned)K1)
                o[(2 * p + 1) * Kh + k] = make_float2(0.5f * (u.y + w.y), 0.5f * (w.x - u.x));
        }
        __syncthreads();
        float2 *res = fft_lines<false, false>(o, r, tw1, p1, K1, Kh, mg_h, 1, Kh);
        for (int t = threadIdx.x; t < K1 * Kh; t += blockDim.x) gc[t] = res[t];
    } else {
        for (int t = threadIdx.x; t < K1 * Kh; t += blockDim.x) A[t] = gc[t];
        __syncthreads();
        float2 *r = fft_lines<true, false>(A, B, tw1, p1, K1, Kh, mg_h, 1, Kh);
        float2 *o = r == A ? B : A;
        // two half spectra as one full complex line (lines of a real grid: the
        // mean and the Nyquist term are real)
        const unsigned mg = magic_of(K2);
        for (unsigned t = threadIdx.x; t < (unsigned)(pairs * K2); t += blockDim.x) {
            const unsigned p = divide(t, mg), z = t - p * K2;
            const bool up = z >= (unsigned)Kh;
            const unsigned k = up ? K2 - z : z;
            const float2 zero = make_float2(0.f, 0.f);
            float2 u = r[2 * p * Kh + k], w = 2 * p + 1 < (unsigned)K1 ? r[(2 * p + 1) * Kh + k] : zero;
            if (up || k == 0 || 2 * k == (unsigned)K2) {
                const float s = up ? -1.f : 0.f;
                u.y *= s;
                w.y *= s;
            }
            o[t] = make_float2(u.x - w.y, u.y + w.x);
        }
        __syncthreads();
        float2 *res = fft_lines<true, true>(o, r, tw2, p2, K2, pairs, 0u, K2, 1);
        float *const gr = a.gr + real0;
        for (unsigned t = threadIdx.x; t < (unsigned)(pairs * K2); t += blockDim.x) {
            const unsigned p = divide(t, mg), z = t - p * K2;
            const size_t e = (size_t)2 * p * K2 + z;
            gr[e] = res[t].x;
            if (2 * p + 1 < (unsigned)K1) gr[e + K2] = res[t].y;
        }
    }
}

// kCols neighbouring (y, z) columns along x: forward, times the influence
// function, and back (BACK: the potential is wanted, else the energy alone).
// Elements with G = 0 (k = 0) are dropped whatever they hold.
template <bool ENERGY, bool BACK>
__global__ void __launch_bounds__(128) k_fft_columns(FftArgs a) {
    extern __shared__ float2 s_fft[];
    __shared__ int4 s_plan[kMaxPasses];
    const FftBlock b = a.blocks[blockIdx.x];
    const int K0 = b.K[0], K2 = b.K[2], Kh = K2 / 2 + 1, plane = b.K[1] * Kh;
    const int c0 = b.index * kCols, nc = min(kCols, plane - c0);
    float2 *const tw = s_fft, *A = tw + K0, *B = A + kCols * K0;
    float *const sG = (float *)(B + kCols * K0);
    for (int t = threadIdx.x; t < K0; t += blockDim.x) tw[t] = a.tw[b.tw[0] + t];
    if (threadIdx.x < kMaxPasses) s_plan[threadIdx.x] = a.plan[kMaxPasses * b.plan[0] + threadIdx.x];
    float2 *const gc = a.gc + b.cgrid_off + c0;
    const float *const G = a.G + b.cgrid_off + c0;
    constexpr unsigned mg_c = (unsigned)(0x100000000ull / kCols);
#pragma unroll 4
    for (int t = threadIdx.x; t < kCols * K0; t += blockDim.x) {
        const int x = t / kCols, c = t % kCols;
        sG[t] = c < nc ? G[(size_t)x * plane + c] : 0.f;
    }
    wait_for_previous();  // (tables and influence function do not change)
#pragma unroll 4
    for (int t = threadIdx.x; t < kCols * K0; t += blockDim.x) {
        const int x = t / kCols, c = t % kCols;
        A[t] = c < nc ? gc[(size_t)x * plane + c] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    float2 *r = fft_lines<false, false>(A, B, tw, s_plan, K0, kCols, mg_c, 1, kCols);
    double e = 0.0;
    for (int t = threadIdx.x; t < kCols * K0; t += blockDim.x) {
        const int c = t % kCols;
        const float g = sG[t];
        const float2 v = r[t];
        const bool live = g != 0.f;
        if (ENERGY && live) {
            const int kz = (c0 + c) % Kh;
            const float wgt = (kz == 0 || 2 * kz == K2) ? 1.0f : 2.0f;
            e += (double)(0.5f * wgt * g * (v.x * v.x + v.y * v.y));
        }
        r[t] = live ? make_float2(v.x * g, v.y * g) : make_float2(0.f, 0.f);
    }
    if (ENERGY) {
        const double v[1] = {e};
        const int slot[1] = {MDG_TERM_COUL_RECIP};
        block_energy_add<1>(a.energy, b.sys, v, slot);
    }
    if (!BACK) return;
    __syncthreads();
    float2 *res = fft_lines<true, false>(r, r == A ? B : A, tw, s_plan, K0, kCols, mg_c, 1, kCols);
    for (int t = threadIdx.x; t < kCols * K0; t += blockDim.x) {
        const int x = t / kCols, c = t % kCols;
        if (c < nc) gc[(size_t)x * plane + c] = res[t];
    }
}

bool smooth(int n) {
    for (int p : {2, 3, 5})
        while (n % p == 0) n /= p;
    return n == 1;
}

size_t plane_smem(const int *K) {
    return sizeof(float2) * ((size_t)K[1] + K[2] + 2 * (size_t)plane_points(K[1], K[2]));
}
size_t column_smem(const int *K) {
    return (size_t)K[0] * (sizeof(float2) * (1 + 2 * kCols) + sizeof(float) * kCols);
}

}  // namespace

// Planes of up to kPlaneMax points (about 50 x 50).  All transforms of an
// evaluation, library's -> this file's kernels, us: 30^3 33 -> 20, 40 grids of 25^3
// to 48^3 in 8 sizes 300 -> 45 (one launch sequence after another -> three launches),
// 48 x 64 x 90 39 -> 36, 100^3 44 -> 47: large planes leave SMs idle here.
bool fft_supported(const int *K) {
    return smooth(K[0]) && smooth(K[1]) && smooth(K[2]) && plane_points(K[1], K[2]) <= kPlaneMax &&
           column_smem(K) <= kSmemMax;
}

void fft_free(FftPlan &f) {
    cudaFree(f.planes);
    cudaFree(f.tiles);
    cudaFree(f.tw);
    cudaFree(f.plan);
    f = FftPlan{};
}

// Block tables and twiddle factors (FP64 on the host) of the listed systems.
int fft_setup(FftPlan &f, const std::vector<SysDev> &sys, const std::vector<int> &ids) {
    fft_free(f);
    if (ids.empty()) return MDG_OK;
    std::vector<FftBlock> planes, tiles;
    std::vector<int> start(1025, -1), plan_of(1025, -1);
    std::vector<float2> tw;
    std::vector<int4> plan;
    for (int q : ids) {
        FftBlock b{};
        b.sys = q;
        b.grid_off = sys[q].grid_off;
        b.cgrid_off = sys[q].cgrid_off;
        for (int d = 0; d < 3; ++d) {
            const int K = b.K[d] = sys[q].K[d];
            if (start[K] < 0) {
                start[K] = (int)tw.size();
                for (int t = 0; t < K; ++t) {
                    const double w = -2.0 * 3.14159265358979323846 * t / K;
                    tw.push_back(make_float2((float)std::cos(w), (float)std::sin(w)));
                }
                plan_of[K] = (int)(plan.size() / kMaxPasses);
                int m = 1, passes = 0;
                for (int left = K; left > 1; ++passes) {
                    const int r = left % 4 == 0 ? 4 : left % 2 == 0 ? 2 : left % 3 == 0 ? 3 : 5;
                    plan.push_back(make_int4(r, m, (int)magic_of(K / r), (int)magic_of(m)));
                    m *= r;
                    left /= r;
                }
                for (; passes < kMaxPasses; ++passes) plan.push_back(make_int4(0, 0, 0, 0));
            }
            b.tw[d] = start[K];
            b.plan[d] = plan_of[K];
        }
        const int nt = (b.K[1] * (b.K[2] / 2 + 1) + kCols - 1) / kCols;
        for (b.index = 0; b.index < b.K[0]; ++b.index) planes.push_back(b);
        for (b.index = 0; b.index < nt; ++b.index) tiles.push_back(b);
        f.plane_smem = std::max(f.plane_smem, plane_smem(b.K));
        f.column_smem = std::max(f.column_smem, column_smem(b.K));
    }
    f.n_planes = (int)planes.size();
    f.n_tiles = (int)tiles.size();
    auto put = [](auto **p, const auto &v) {
        const size_t bytes = sizeof(v[0]) * v.size();
        return cudaMalloc((void **)p, bytes) == cudaSuccess &&
               cudaMemcpy(*p, v.data(), bytes, cudaMemcpyHostToDevice) == cudaSuccess;
    };
    if (!put(&f.planes, planes) || !put(&f.tiles, tiles) || !put(&f.tw, tw) || !put(&f.plan, plan))
        return MDG_ERR_NOMEM;
    const int pm = (int)kSmemMax;
    auto grow = [&](auto kernel) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, pm) ==
               cudaSuccess;
    };
    if (!grow(k_fft_planes<false>) || !grow(k_fft_planes<true>) || !grow(k_fft_columns<false, true>) ||
        !grow(k_fft_columns<true, true>) || !grow(k_fft_columns<true, false>))
        return MDG_ERR_CUDA;
    return MDG_OK;
}

// rho (int64, left zeroed) -> phi in the real grids of the plan's systems.
// back = 0: the energy alone.
cudaError_t fft_convolve(mdg_system *s, const FftPlan &f, int energy, int back) {
    if (!f.n_planes) return cudaSuccess;
    FftArgs a;
    a.plan = f.plan;
    a.tw = f.tw;
    a.gi = s->pme.grid_i;
    a.gr = s->pme.grid_r;
    a.gc = s->pme.grid_c;
    a.G = s->pme.influence;
    a.energy = s->energy;
    cudaStream_t st = s->stream;
    a.blocks = f.planes;
    cudaError_t e = launch_after(k_fft_planes<false>, f.n_planes, kPlaneThreads, f.plane_smem, st, a);
    FftArgs c = a;
    c.blocks = f.tiles;
    if (e == cudaSuccess)
        e = launch_after(!back    ? k_fft_columns<true, false>
                         : energy ? k_fft_columns<true, true>
                                  : k_fft_columns<false, true>,
                         f.n_tiles, 128, f.column_smem, st, c);
    s->launches += 2;
    if (back && e == cudaSuccess) {
        e = launch_after(k_fft_planes<true>, f.n_planes, kPlaneThreads, f.plane_smem, st, a);
        s->launches += 1;
    }
    return e;
}

}  // namespace mdg
