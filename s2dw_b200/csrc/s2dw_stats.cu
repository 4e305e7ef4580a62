// Moments of the wavelet coefficients per scale (s2dw_stat_moments,
// src/mod/s2dw_stat_mod.f90:81-275) for batches of maps resident on the GPU.
//
// Two passes over each (map, scale) block of the packed wavelet layout:
//   pass 1: sum of the (masked) coefficients and of the mask -> mean, nj;
//   pass 2: sums of s, s^2, ..., s^6 with s = w - mean over the samples whose
//           mask is 1 (all samples without a mask);
// then the reference's normalisations (n-1 variance, standardised skewness,
// excess kurtosis, fifth and excess sixth moments; zero variance -> zeros).
// Every reduction runs in a fixed order (per-thread sums, shuffle and
// shared-memory trees, then the blocks' partials in a warp's tree), so
// results are bit-reproducible.
//
// Bound by HBM: two reads of the coefficients (and mask).  Each thread has two or
// four 16-byte loads in flight, whatever boundary the arrays start on, and the
// partials are summed by a warp at the start of the pass that needs them.  Against
// one 8-byte load in flight, 64 blocks per scale and single threads summing the
// partials, B200 at B=512, N=4 (us): 4 maps with a mask 251 -> 138 (mask on another
// 16-byte boundary 239 -> 144), without 167 -> 115; 16 maps 784 -> 464 and 459 -> 400.
#include <cuda_runtime.h>

#include "s2dw_internal.h"

namespace s2dw {
namespace {

constexpr int STAT_T = 256;
constexpr double TOL_ZERO = 1e-12;

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of v over the block, in thread 0.
template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K])
{
    __shared__ double sh[K][STAT_T / 32];
    const int t = threadIdx.x;
#pragma unroll
    for (int k = 0; k < K; k++) {
        v[k] = warp_sum(v[k]);
        if ((t & 31) == 0) sh[k][t >> 5] = v[k];
    }
    __syncthreads();
    if (t == 0)
#pragma unroll
        for (int k = 0; k < K; k++) {
            v[k] = sh[k][0];
            for (int w = 1; w < STAT_T / 32; w++) v[k] += sh[k][w];
        }
}

// Sum over the P blocks' partials of pass 1's value k of row y, by one warp.
template <int P>
__device__ __forceinline__ double partial_sum(const StatArgs &a, int y, int k)
{
    double s = 0.0;
#pragma unroll
    for (int x = threadIdx.x & 31; x < P; x += 32) s += a.part[((size_t)y * P + x) * 2 + k];
    return warp_sum(s);
}

// Grid (map, share, scale): the blocks of one share of a scale run together
// over the maps, which read the same part of the mask (map-major, every map read
// the mask from HBM: 4 maps at B=512, N=4 180 us instead of 153; without a mask
// 137 and 117).  Row y = map (J+1) + scale of the partials, and the coefficient
// block.
struct StatBlock {
    const double *w, *mk;
    long long n;
    int y, x;
};
template <int MASK>
__device__ __forceinline__ StatBlock stat_block(const StatArgs &a)
{
    const int k = blockIdx.x, j = blockIdx.z;
    StatBlock b;
    b.x = blockIdx.y;
    b.y = k * (a.J + 1) + j;
    b.w = a.wav + (size_t)k * a.wtot + a.off[j];
    b.mk = MASK ? a.mask + a.off[j] : nullptr;
    b.n = a.off[j + 1] - a.off[j];
    return b;
}

// Calls f(w, mask) for the block's share of the (map, scale) block's values, U
// pairs per thread at a time, from the coefficients' first 16-byte boundary on: a
// block holds an even number of values, and one that starts off a boundary has a
// single first and last value.  The mask is read in pairs where its boundaries
// are the same (MASK_PAIRS).
enum StatMask { MASK_NONE, MASK_PAIRS, MASK_SINGLE };
template <int MASK, int U, int P, typename F>
__device__ __forceinline__ void stat_values(const StatBlock &b, F &&f)
{
    constexpr long long step = (long long)P * STAT_T;
    const long long t = (long long)b.x * STAT_T + threadIdx.x;
    const int odd = ((uintptr_t)b.w >> 3) & 1;
    if (odd && t < 2) {
        const long long i = t ? b.n - 1 : 0;
        f(b.w[i], MASK ? b.mk[i] : 1.0);
    }
    const double2 *w = reinterpret_cast<const double2 *>(b.w + odd);
    const double *m = b.mk + odd;
    const long long n = b.n / 2 - odd;
    for (long long i0 = t; i0 < n; i0 += U * step) {
        double2 x[U], y[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long long i = i0 + u * step;
            if (i < n) {
                x[u] = w[i];
                y[u] = MASK == MASK_NONE    ? make_double2(1.0, 1.0)
                       : MASK == MASK_PAIRS ? reinterpret_cast<const double2 *>(m)[i]
                                            : make_double2(m[2 * i], m[2 * i + 1]);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * step < n) {
                f(x[u].x, y[u].x);
                f(x[u].y, y[u].y);
            }
    }
}

template <int MASK, int U, int P>
__global__ void __launch_bounds__(STAT_T) stat_pass1(const __grid_constant__ StatArgs a)
{
    const StatBlock b = stat_block<MASK>(a);
    double v[2] = {0.0, 0.0};
    stat_values<MASK, U, P>(b, [&](double w, double m) {
        if (!MASK || fabs(m - 1.0) < TOL_ZERO) v[0] += w * m;
        v[1] += m;
    });
    block_sum<2>(v);
    if (threadIdx.x == 0) {
        double *p = a.part + ((size_t)b.y * P + b.x) * 2;
        p[0] = v[0];
        p[1] = v[1];
    }
}

// mean and nj of row y, by one warp
template <int P>
__device__ __forceinline__ double2 stat_mean(const StatArgs &a, int y)
{
    const int j = y % (a.J + 1);
    const double s = partial_sum<P>(a, y, 0), c = partial_sum<P>(a, y, 1);
    const double nj = a.mask ? rint(c) : (double)(a.off[j + 1] - a.off[j]);
    return make_double2(s / nj, nj);
}

template <int MASK, int U, int P>
__global__ void __launch_bounds__(STAT_T) stat_pass2(const __grid_constant__ StatArgs a)
{
    __shared__ double smu;
    const StatBlock b = stat_block<MASK>(a);
    if (threadIdx.x < 32) {
        const double2 m = stat_mean<P>(a, b.y);
        if (threadIdx.x == 0) {
            smu = m.x;
            if (b.x == 0) {
                a.mean_nj[2 * b.y] = m.x;
                a.mean_nj[2 * b.y + 1] = m.y;
            }
        }
    }
    __syncthreads();
    const double mu = smu;
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    stat_values<MASK, U, P>(b, [&](double w, double m) {
        if (MASK && !(fabs(m - 1.0) < TOL_ZERO)) return;
        const double s = w * m - mu;
        double p = s * s;
        v[0] += s;
        v[1] += p;
        p *= s;
        v[2] += p;
        p *= s;
        v[3] += p;
        p *= s;
        v[4] += p;
        p *= s;
        v[5] += p;
    });
    block_sum<6>(v);
    if (threadIdx.x == 0) {
        double *p = a.part2 + ((size_t)b.y * P + b.x) * 6;
#pragma unroll
        for (int k = 0; k < 6; k++) p[k] = v[k];
    }
}

// moments per (map, scale), a warp each: out[y*6 + {mean, var, skew, kur,
// five, six}], flags[y] = 1 zero variance, 2 fewer than two samples
template <int P>
__global__ void __launch_bounds__(128) stat_final(const __grid_constant__ StatArgs a)
{
    const int y = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (y >= a.nmaps * (a.J + 1)) return;
    double s[6];
#pragma unroll
    for (int k = 0; k < 6; k++) {
        double t = 0.0;
#pragma unroll
        for (int x = threadIdx.x & 31; x < P; x += 32) t += a.part2[((size_t)y * P + x) * 6 + k];
        s[k] = warp_sum(t);
    }
    if (threadIdx.x & 31) return;
    const double mu = a.mean_nj[2 * y], nj = a.mean_nj[2 * y + 1];
    double *o = a.out + (size_t)y * 6;
    o[0] = mu;
    if (nj < 2.0) {
        a.flags[y] = 2;
        for (int k = 1; k < 6; k++) o[k] = 0.0;
        return;
    }
    const double v = (s[1] - s[0] * s[0] / nj) / (nj - 1.0);
    const double sd = sqrt(v);
    o[1] = v;
    if (v < TOL_ZERO) {
        a.flags[y] = 1;
        o[2] = o[3] = o[4] = o[5] = 0.0;
    } else {
        a.flags[y] = 0;
        o[2] = s[2] / (nj * sd * sd * sd);
        o[3] = s[3] / (nj * v * v) - 3.0;
        o[4] = s[4] / (nj * sd * sd * sd * sd * sd);
        o[5] = s[5] / (nj * v * v * v) - 15.0;
    }
}

}  // namespace

template <int MASK, int U, int P>
static void launch_passes(const StatArgs &a, cudaStream_t s)
{
    const dim3 grid(a.nmaps, P, a.J + 1);
    stat_pass1<MASK, U, P><<<grid, STAT_T, 0, s>>>(a);
    stat_pass2<MASK, U, P><<<grid, STAT_T, 0, s>>>(a);
    stat_final<P><<<(a.nmaps * (a.J + 1) + 3) / 4, 128, 0, s>>>(a);
}

int launch_stat_moments(const StatArgs &a, cudaStream_t s)
{
    if (a.nmaps <= 0) return S2DWC_OK;
    // (maps and scales have an even number of values: one boundary for all)
    if (a.mask && (((uintptr_t)a.wav ^ (uintptr_t)a.mask) & 15) == 0) launch_passes<MASK_PAIRS, 4, 96>(a, s);
    else if (a.mask) launch_passes<MASK_SINGLE, 4, 96>(a, s);
    else if (a.P == 96) launch_passes<MASK_NONE, 4, 96>(a, s);
    else launch_passes<MASK_NONE, 2, 48>(a, s);
    S2DW_CUDA_TRY(cudaGetLastError());
    return S2DWC_OK;
}

}  // namespace s2dw
