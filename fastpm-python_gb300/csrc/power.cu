// Integer-shell power spectrum of a complex half mesh (fastpm/utils.py:77-164).
// Shell d = floor(sqrt(n^2)) (utils.py find_root: its refinement loop re-tests
// every mode, so every mode ends in floor(sqrt(n^2))); weight 1 on the l = 0 and l = n/2 planes, 2 elsewhere
// (utils.py:147-149); modes of shells past n/2 - 1 count nowhere and are not read.
//
// The sums of k and of the weights depend on n alone: they are tabulated once per
// device (fpm_device_init) and each call adds them.
//
// One warp takes the rows (+-i, +-j) of a pair (i, j), 0 <= i, j <= n/2: the
// same n^2 in up to four rows of the mesh, lanes along l.  Shells do not
// decrease along the lanes, so the lanes of a shell are summed by a segmented
// warp reduction and the first lane adds the sum to the warp's own bins in
// shared memory (one lane per bin: no atomics); the CTA's bins meet at the end.
//
// FP64 bounds it (a warp-wide FP64 instruction holds an SM for 16 cycles on
// GB300).  Three square roots, the shell search and three float64 shared
// atomics per mode took 43 of them; now the squares of an auto spectrum's four
// modes add up in float32 with their errors (PwSum) and take about five FP64
// additions in all: 512^3 4961 -> 233 us (402 us with FP64 multiply-adds
// per mode; its 0.55 GB take 41 us of HBM).  The sums' error against float64 is
// what it was (1e-16 to 4e-14 of a shell).
#include "ff.cuh"
#include <math.h>
#include "trace.h"

namespace {
constexpr int PW_WARPS = 4;
// sums of sqrt(n^2) and of the weights per shell, of every supported size
constexpr int PW_SIZES[] = {16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512, 1024};
constexpr int PW_BINS = 1388;   // sum of n / 2
__device__ double g_geom[2][PW_BINS];

int geom_offset(int n) {
    int o = 0;
    for (int m : PW_SIZES) {
        if (m == n) return o;
        o += m / 2;
    }
    return -1;
}

// one (i, j >= 0) row per warp, its sign copies by weight
__global__ void __launch_bounds__(128) geom_kernel(int n, double* ksum, double* wsum) {
    extern __shared__ double gs[];
    const int nb = n / 2, h = nb + 1;
    for (int b = threadIdx.x; b < 2 * nb; b += blockDim.x) gs[b] = 0.0;
    __syncthreads();
    for (int r = blockIdx.x * 4 + (threadIdx.x >> 5); r < h * h; r += gridDim.x * 4) {
        const int i = r / h, j = r - i * h, t2 = i * i + j * j;
        const double m = (double)((i == 0 || i == nb ? 1 : 2) * (j == 0 || j == nb ? 1 : 2));
        for (int l = threadIdx.x & 31; l < nb && t2 + l * l < nb * nb; l += 32) {
            const double k = sqrt((double)(t2 + l * l));
            const int d = (int)__fsqrt_rn((float)(t2 + l * l));
            const double w = l == 0 ? m : 2.0 * m;
            atomicAdd(&gs[d], k * w);
            atomicAdd(&gs[nb + d], w);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        atomicAdd(&ksum[b], gs[b]);
        atomicAdd(&wsum[b], gs[nb + b]);
    }
}

// float32 -> float64 without the FP64 pipe for normal numbers
__device__ __forceinline__ double pw_widen(float x) {
    const unsigned b = __float_as_uint(x), e = b & 0x7f800000u;
    if (e == 0u || e == 0x7f800000u) return (double)x;   // zero, subnormal, inf, NaN
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}

// values whose squares float-float products hold exactly
__device__ __forceinline__ bool pw_in_range(float x) {
    const float a = fabsf(x);
    return a == 0.f || (a >= 0x1p-50f && a < 0x1p50f);
}
// a sum of squares as three float32 (about 70 bits): exact products and
// error-free sums, so one rounding to float64 is left at the end
struct PwSum {
    float h = 0.f, l = 0.f, e = 0.f;
    __device__ __forceinline__ void add_square(float x) {
        const ff p = ff_two_prod(x, x);
        const ff a = ff_two_sum(h, p.h), b = ff_two_sum(l, p.l), c = ff_two_sum(b.h, a.l);
        h = a.h;
        l = c.h;
        e = __fadd_rn(e, __fadd_rn(b.l, c.l));
    }
};

// |a conj(b)|
__device__ __forceinline__ double pw_cross(float2 a, float2 b) {
    const double re = (double)a.x * b.x + (double)a.y * b.y;
    const double im = (double)a.y * b.x - (double)a.x * b.y;
    return sqrt(re * re + im * im);
}

template <bool CROSS>
__global__ void __launch_bounds__(32 * PW_WARPS)
power_kernel(const float2* __restrict__ f1, const float2* __restrict__ f2, int n, int zp, double kf,
             const double* __restrict__ geom_k, const double* __restrict__ geom_w, double* ksum, double* psum,
             double* wsum) {
    extern __shared__ double sh[];
    const int nb = n / 2, h = nb + 1;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double* bins = sh + wid * nb;   // this warp's own
    for (int b = threadIdx.x; b < PW_WARPS * nb; b += blockDim.x) sh[b] = 0.0;
    if (blockIdx.x == 0)
        for (int b = threadIdx.x; b < nb; b += blockDim.x) {
            atomicAdd(&ksum[b], geom_k[b] * kf);
            atomicAdd(&wsum[b], geom_w[b]);
        }
    __syncthreads();
    const unsigned full = 0xffffffffu;
    const int nwarp = gridDim.x * PW_WARPS;
    for (int r = blockIdx.x * PW_WARPS + wid; r < h * h; r += nwarp) {
        const int i = r / h, j = r - i * h;
        const int t2 = i * i + j * j;
        if (t2 >= nb * nb) continue;
        // the distinct rows of (+-i, +-j) (i, j < n/2 here)
        const bool mi = i != 0, mj = j != 0;
        const long long ri = (long long)i * n, rm = (long long)(n - i) * n;
        const float2* row[4] = {f1 + (ri + j) * zp, f1 + (ri + (n - j)) * zp, f1 + (rm + j) * zp,
                                f1 + (rm + (n - j)) * zp};
        const long long other = f2 - f1;
        for (int l0 = 0; l0 * l0 + t2 < nb * nb; l0 += 32) {   // warp-uniform
            const int l = l0 + lane;
            const int kk = t2 + l * l;
            const bool in = kk < nb * nb;
            // floor(sqrt(kk)): kk < 2^24 is exact and its float32 root cannot round up to the next integer
            const int d = in ? (int)__fsqrt_rn((float)kk) : -1;
            double p = 0.0;
            if (in) {
                float2 a[4], b[4];
                bool fast = !CROSS;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const bool on = (q < 2 || mi) && ((q & 1) == 0 || mj);
                    a[q] = on ? __ldg(row[q] + l) : make_float2(0.f, 0.f);
                    b[q] = CROSS && on ? __ldg(row[q] + other + l) : a[q];
                    fast = fast && pw_in_range(a[q].x) && pw_in_range(a[q].y);
                }
                if (fast) {
                    PwSum t;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {   // |a conj(a)| = x^2 + y^2
                        t.add_square(a[q].x);
                        t.add_square(a[q].y);
                    }
                    p = pw_widen(t.h) + (pw_widen(t.l) + pw_widen(t.e));
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) p += pw_cross(a[q], b[q]);
                }
                if (l != 0) p *= 2.0;
            }
            // segmented reduction: the first lane of a shell collects its lanes
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int od = __shfl_down_sync(full, d, o);
                const bool same = lane + o < 32 && od == d && d >= 0;
                // no shell reaches past the lanes already summed: done (warp-uniform)
                if (!__any_sync(full, same)) break;
                const double op = __shfl_down_sync(full, p, o);
                if (same) p += op;
            }
            const int pd = __shfl_up_sync(full, d, 1);
            if (in && (lane == 0 || pd != d)) bins[d] += p;
            __syncwarp();
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        double p = 0.0;
#pragma unroll
        for (int w = 0; w < PW_WARPS; ++w) p += sh[w * nb + b];
        if (p != 0.0) atomicAdd(&psum[b], p);
    }
}
}  // namespace

// fill this device's geometry tables (part of the one-time device set-up)
int fpm_internal_power_init() {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_geom) != cudaSuccess) return FPM_ERR_CUDA;
    double* g = (double*)p;
    if (cudaMemsetAsync(g, 0, sizeof(double) * 2 * PW_BINS, cudaStreamLegacy) != cudaSuccess) return FPM_ERR_CUDA;
    for (int n : PW_SIZES) {
        const int o = geom_offset(n), rows = (n / 2 + 1) * (n / 2 + 1);
        geom_kernel<<<(rows + 31) / 32, 128, n * (int)sizeof(double), cudaStreamLegacy>>>(n, g + o, g + PW_BINS + o);
    }
    if (cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) return FPM_ERR_CUDA;
    return fpm_launch_status();
}

extern "C" int fpm_power_accumulate(const void* f1, const void* f2, int n, double boxsize,
                                    double* ksum, double* psum, double* wsum, void* stream) {
    if (!f1 || !ksum || !psum || !wsum || boxsize <= 0) return FPM_ERR_ARG;
    if (!fpm_fft_supported(n)) return FPM_ERR_SHAPE;
    int rc = fpm_device_init();
    if (rc) return rc;
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_geom) != cudaSuccess) return FPM_ERR_CUDA;
    const double *gk = (const double*)p + geom_offset(n), *gw = gk + PW_BINS;
    const int zp = fpm_complex_row(n), nb = n / 2;
    const int smem = nb * PW_WARPS * (int)sizeof(double);   // 16 KB at n = 1024
    // enough warps to fill the SMs, at least 8 rows a warp (its bins are zeroed and merged once)
    const long long rows = (long long)(nb + 1) * (nb + 1);
    long long grid = (rows + 8 * PW_WARPS - 1) / (8 * PW_WARPS);
    if (grid > 152 * 8) grid = 152 * 8;
    const double kf = 2.0 * M_PI / boxsize;
    cudaStream_t st = (cudaStream_t)stream;
    FPM_TRACE("power", st);
    if (f2 && f2 != f1)
        power_kernel<true><<<(unsigned)grid, 32 * PW_WARPS, smem, st>>>((const float2*)f1, (const float2*)f2, n, zp,
                                                                       kf, gk, gw, ksum, psum, wsum);
    else
        power_kernel<false><<<(unsigned)grid, 32 * PW_WARPS, smem, st>>>((const float2*)f1, (const float2*)f1, n, zp,
                                                                        kf, gk, gw, ksum, psum, wsum);
    return fpm_launch_status();
}
