// Beta stages of transforms of up to 2048 points (see RowFft): the analysis
// beta sums (s2dw_core_mod.f90:708-743) and the synthesis gamma DFT, weights,
// beta sums and +-m' fold (:1132-1198), all scales of a group in one launch.
//
// Bound by shared memory and launch width, not HBM: a 1024-point row of 16
// values per thread makes two exchanges.  The general engine this replaced
// ran CTAs of 512 threads (4 ... 64 CTAs per launch at bl <= 256) with run-time
// radices and twiddles from a two-level table.  Both stages of a pair at
// B = 256, N = 5: a launch per scale and engine -> one launch each, 226 -> 206 us
// per pair with the alpha stages'; the scales bl <= 512 of B = 1024, N = 4 take 34
// (analysis) and 44 us (synthesis), 151 and 228 before.
#include <cuda_runtime.h>

#include "s2dw_fft.cuh"
#include "s2dw_internal.h"

namespace s2dw {
namespace {

template <int MODE, int LG>
__device__ __forceinline__ void ana_beta(const StageArgs &a, const StageEnt &e, int cta, double2 *smem)
{
    using F = RowFft<LG>;
    constexpr int M = F::M, V = F::V, TPR = F::TPR;
    const int t = threadIdx.x % TPR, r = threadIdx.x / TPR, bl = e.bl, N = a.N;
    const int row = cta * F::ROWS + r, per = e.rows_map;
    const bool valid = row < e.rows;
    const int k = valid ? row / per : 0, gm = valid ? row - k * per : 0, m = gm % bl;
    const double2 *X = static_cast<const double2 *>(e.in) + k * e.in_map + (size_t)gm * bl;
    double2 *Y = static_cast<double2 *>(e.out) + k * e.out_map + (size_t)gm * (2 * bl);
    const bool sn = (m + N - 1) & 1;
    double2 *buf = smem + r * F::PITCH;
    double2 v[V];
    if (MODE == FFT_ANA_BETA) {
        // DCT-III input (see s2dw_fft.cuh), M = 2 bl: X(k) e_k at k < bl and
        // X(k) conj(e_k) at M - k, which its reader takes from shared memory,
        // so that every X and e is loaded once, all loads of a thread together
        constexpr int BL = M / 2;
        double2 xe[V / 2], w[V / 2];
#pragma unroll
        for (int i = 0; i < V / 2; i++) w[i] = __ldg(e.pre + t + i * TPR);
        pdl_wait();
#pragma unroll
        for (int i = 0; i < V / 2; i++) xe[i] = X[t + i * TPR];
        double2 x0 = make_double2(0.0, 0.0);
        if (sn) x0 = X[0];
#pragma unroll
        for (int i = 0; i < V / 2; i++) {
            const int k = t + i * TPR;
            const double2 y = cmul(xe[i], w[i]), z = cmul(xe[i], cconj(w[i]));
            v[i] = sn ? make_double2(y.y, -y.x) : y;  // -i y
            if (k > 0) buf[F::pad(M - k)] = sn ? make_double2(-z.y, z.x) : z;  // i z
            else {
                if (sn) v[i] = make_double2(0.0, 0.0);
                buf[F::pad(BL)] = make_double2(0.0, 0.0);
            }
        }
        F::sync();
#pragma unroll
        for (int i = V / 2; i < V; i++) v[i] = buf[F::pad(t + i * TPR)];
        F::sync();
        F::template run<+1>(v, buf, t, a.tw);
        // even and odd b from the two halves: through shared memory, so that
        // the stores are contiguous
#pragma unroll
        for (int i = 0; i < V; i++) {
            int b;
            const double2 y = ana_beta_out(v[i], t + i * TPR, bl, sn, x0, &b);
            buf[F::pad(b)] = y;
        }
        F::sync();
        if (!valid) return;
#pragma unroll
        for (int i = 0; i < V; i++) Y[t + i * TPR] = buf[F::pad(t + i * TPR)];
    } else {  // k <-> m' = k - (bl - 1)
        const int K = 2 * bl - 1;
        pdl_wait();
#pragma unroll
        for (int i = 0; i < V; i++) {
            const int kk = t + i * TPR, mpv = kk - (bl - 1);
            double2 x = make_double2(0.0, 0.0);
            if (kk < K) {
                x = X[mpv < 0 ? -mpv : mpv];
                if (sn && mpv < 0) x = make_double2(-x.x, -x.y);
                x = cmul(x, __ldg(e.pre + kk));
            }
            v[i] = x;
        }
        F::template run<-1>(v, buf, t, a.tw);
#pragma unroll
        for (int i = 0; i < V; i++) v[i] = cmul(v[i], __ldg(e.Hf + t + i * TPR));
        F::template run<+1>(v, buf, t, a.tw);
        if (!valid) return;
#pragma unroll
        for (int i = 0; i < V; i++) {
            const int b = t + i * TPR;
            if (b < 2 * bl) Y[b] = cmul(v[i], __ldg(e.post + b));
        }
    }
}

template <int MODE, int LG>
__device__ __forceinline__ void syn_beta(const StageArgs &a, const StageEnt &e, int cta, double2 *smem)
{
    using F = RowFft<LG>;
    constexpr int M = F::M, V = F::V, TPR = F::TPR;
    const int t = threadIdx.x % TPR, r = threadIdx.x / TPR, bl = e.bl, N = a.N, NP = a.NP;
    const int row = cta * F::ROWS + r, per = e.rows_map;
    const bool valid = row < e.rows;
    // q fastest: rows that read the same V share a CTA
    const int k = valid ? row / per : 0, mq = valid ? row - k * per : 0, m = mq / NP, q = mq - m * NP, n = a.nq[q];
    const double2 *X = static_cast<const double2 *>(e.in) + k * e.in_map + (size_t)m * (2 * bl);
    double2 *Y = static_cast<double2 *>(e.out) + k * e.out_map + ((size_t)q * bl + m) * e.out_stride;
    const double2 *ph = a.ph + N - 1 - n;  // exp(-i pi n g / N), g rows of 2N-1
    const bool odd = (m + n) & 1;
    double2 *buf = smem + r * F::PITCH;
    double2 v[V];
#pragma unroll
    for (int i = 0; i < V; i++) v[i] = make_double2(0.0, 0.0);
    pdl_wait();
    // gamma DFT, one sample at a time: its loads are in flight together
    for (int g = 0; g < N; g++, X += (size_t)bl * (2 * bl)) {
        const double2 w = __ldg(ph + g * (2 * N - 1));
#pragma unroll
        for (int i = 0; i < V; i++) {
            const int b = t + i * TPR;
            if (MODE == FFT_SYN_BETA || b < 2 * bl) v[i] = cadd(v[i], cmul(X[b], w));
        }
    }
    if (MODE == FFT_SYN_BETA) {
        // value of b at its place in the DCT-II reordering
#pragma unroll
        for (int i = 0; i < V; i++) {
            const int b = t + i * TPR;
            double2 u = cscale(v[i], __ldg(e.wq + b));
            if (odd && (b & 1)) u = make_double2(-u.x, -u.y);
            buf[F::pad((b & 1) ? (4 * bl - 1 - b) >> 1 : b >> 1)] = u;
        }
        F::sync();
#pragma unroll
        for (int i = 0; i < V; i++) v[i] = buf[F::pad(t + i * TPR)];
        F::sync();
        F::template run<-1>(v, buf, t, a.tw);
    } else {
#pragma unroll
        for (int i = 0; i < V; i++) {
            const int b = t + i * TPR;
            v[i] = b < 2 * bl ? cmul(cscale(v[i], __ldg(e.wq + b)), __ldg(e.pre + b)) : make_double2(0.0, 0.0);
        }
        F::template run<-1>(v, buf, t, a.tw);
#pragma unroll
        for (int i = 0; i < V; i++) v[i] = cmul(v[i], __ldg(e.Hf + t + i * TPR));
        F::template run<+1>(v, buf, t, a.tw);
    }
#pragma unroll
    for (int i = 0; i < V; i++) buf[F::pad(t + i * TPR)] = v[i];
    F::sync();
    if (!valid) return;
    for (int mp = t; mp < bl; mp += TPR) {
        double2 y;
        if (MODE == FFT_SYN_BETA) {
            y = syn_beta_out(buf[F::pad(mp)], buf[F::pad((M - mp) & (M - 1))], mp, odd, e.pre);
        } else {
            const int t0 = bl - 1 + mp, t1 = bl - 1 - mp;
            y = cmul(buf[F::pad(t0)], __ldg(e.post + t0));
            double2 z = cmul(buf[F::pad(t1)], __ldg(e.post + t1));
            if (mp > 0) y = odd ? csub(y, z) : cadd(y, z);
        }
        Y[mp] = y;
    }
}

template <int MODE, int LG>
__device__ __forceinline__ void beta_row(const StageArgs &a, const StageEnt &e, int cta, double2 *smem)
{
    if constexpr (MODE == FFT_ANA_BETA || MODE == CZT_ANA_BETA) ana_beta<MODE, LG>(a, e, cta, smem);
    else syn_beta<MODE, LG>(a, e, cta, smem);
}

template <int MODE>
__device__ __forceinline__ void beta_size(const StageArgs &a, const StageEnt &e, int cta, double2 *smem)
{
    switch (e.lg) {
    case 4: beta_row<MODE, 4>(a, e, cta, smem); break;
    case 5: beta_row<MODE, 5>(a, e, cta, smem); break;
    case 6: beta_row<MODE, 6>(a, e, cta, smem); break;
    case 7: beta_row<MODE, 7>(a, e, cta, smem); break;
    case 8: beta_row<MODE, 8>(a, e, cta, smem); break;
    case 9: beta_row<MODE, 9>(a, e, cta, smem); break;
    case 10: beta_row<MODE, 10>(a, e, cta, smem); break;
    case 11: beta_row<MODE, 11>(a, e, cta, smem); break;
    }
}

template <int FFT, int CZT>
__global__ void __launch_bounds__(ST_THREADS, 4) beta_kernel(const __grid_constant__ StageArgs a)
{
    extern __shared__ __align__(16) double2 smem[];
    pdl_start();
    int cta;
    const StageEnt &e = stage_entry(a, cta);
    if (e.kind == FFT) beta_size<FFT>(a, e, cta, smem);
    else beta_size<CZT>(a, e, cta, smem);
}

// shared values of a CTA: 128/TPR rows of PITCH, the largest over the sizes
constexpr size_t BETA_SMEM = sizeof(double2) * (2048 + 2048 / 4 + 32);

}  // namespace

int launch_stage_beta(Stage st, const StageArgs &a, bool dep, cudaStream_t s)
{
    if (a.ncta <= 0) return S2DWC_OK;
    auto *k = st == STAGE_ANA_BETA ? beta_kernel<FFT_ANA_BETA, CZT_ANA_BETA> : beta_kernel<FFT_SYN_BETA, CZT_SYN_BETA>;
    S2DW_CUDA_TRY(launch_dep(k, a.ncta, ST_THREADS, BETA_SMEM, s, dep, a));
    return S2DWC_OK;
}

}  // namespace s2dw
