// Device kernels of libs2dw_cuda (sm_100a, FP64).
//
//  * fprep_kernel  : the analysis input scaled and transposed for the
//                    contraction (s2dw_contract.cu)
//  * fft_large / fft_pf : FFTs of 2048 to 8192 points of the large scales'
//                    beta and (Bluestein) alpha stages (:708-768, :1104-1198)
//  * pfa*          : prime-factor alpha stages of the power-of-two band limits
//  * alpha_kernel  : alpha stages of a group of scales of up to 512
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <mutex>
#include <vector>
#include <cstdio>
#include <type_traits>

#include "s2dw_fft.cuh"
#include "s2dw_internal.h"

namespace s2dw {

// Per-scale factor tables of the split form (built once per set of kernel
// tables).
__global__ void gprep_kernel(GprepArgs a)
{
    const int nl = a.bl - a.blo - 1;
    const long long total = (long long)nl * a.NP * a.stride;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % a.stride);
        const long long r = i / a.stride;
        const int q = (int)(r % a.NP), l = a.blo + 1 + (int)(r / a.NP);
        double v = 0.0;
        if (x <= l && x < a.bl)
            v = a.T[(size_t)l * a.Bp + x] * a.H[hpack(l, a.NP, q, x)] * a.kappa[(size_t)l * a.NP + q];
        a.out[i] = v;
    }
}

// F[l*Bp + m] = i^{-m} Om[l*Bp+m] flm[l + B m]: transpose of the column-major flm
// through a 32x32 shared tile.
__global__ void fprep_kernel(double2 *F, double2 *scoeff, const double2 *flm, const double *Om, int B, int Bp, int bs)
{
    __shared__ double2 tile[32][33];
    pdl_start();
    const int l0 = blockIdx.x * 32, mb = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    for (int k = ty; k < 32; k += 8) {
        const int l = l0 + tx, m = mb + k;
        tile[k][tx] = (l < B && m < B) ? flm[(size_t)l + (size_t)B * m] : make_double2(0.0, 0.0);
        if (l < bs && m < bs) scoeff[l + (size_t)bs * m] = tile[k][tx];
    }
    __syncthreads();
    for (int k = ty; k < 32; k += 8) {
        const int l = l0 + k, m = mb + tx;
        if (l < B && m < Bp) {
            double2 v = make_double2(0.0, 0.0);
            if (m <= l && m < B) {
                v = cscale(tile[tx][k], Om[(size_t)l * Bp + m]);
                if (m & 1) v = make_double2(v.y, -v.x);  // i^{-m}
                if (m & 2) v = make_double2(-v.x, -v.y);
            }
            F[(size_t)l * Bp + m] = v;
        }
    }
}

// ===========================================================================
// Chirp-z transform engine: power-of-two FFTs in shared memory
// ===========================================================================

__host__ __device__ __forceinline__ int padix(int i) { return i + (i >> 4); }

// W_M^x (forward) from the two-level tables.
__device__ __forceinline__ double2 twid(const double2 *twh, const double2 *twl, int x)
{
    return cmul(twh[x >> 6], twl[x & 63]);
}

// ===========================================================================
// Large transforms (M = 4096, 8192): one transform per CTA, compile-time size
//
// Radix-16 Stockham passes with 16 values per thread (THREADS = M/16), the
// shape with the fewest shared-memory exchanges.  The twiddles of a pass are
// the powers w^s (s = 1..15) of one root w = W_M^step: w from the two-level
// table, w^2..w^15 by products (w^8 and w^4 squarings, then products), which
// keeps shared-memory traffic to the data exchanges.  The row (g, m) or
// (g, b pair) comes from the 2-D grid, so no integer division is needed.
// ===========================================================================
template <int LGM, int LNS, int SIGN>
__device__ __forceinline__ void pass16(double2 (&v)[16], int t, const double2 *twh, const double2 *twl)
{
    if (LNS > 0) {
        const int k = t & ((1 << LNS) - 1);
        twiddle_powers16<SIGN>(v, twid(twh, twl, k << (LGM - LNS - 4)));
    }
    Dft<16, SIGN>::run(v);
}

// Radix-2 pass for LGM = 13 (the remainder of 13 = 4+4+4+1), 8 butterflies per thread.
template <int LGM, int LNS, int SIGN>
__device__ __forceinline__ void pass2x8(double2 (&v)[16], int t, const double2 *twh, const double2 *twl)
{
#pragma unroll
    for (int u = 0; u < 8; u++) {
        if (LNS > 0) {
            const int j = (t * 8 + u) & ((1 << (LGM - 1)) - 1), k = j & ((1 << LNS) - 1);
            double2 w = twid(twh, twl, k << (LGM - LNS - 1));
            if (SIGN > 0) w = cconj(w);
            v[2 * u + 1] = cmul(v[2 * u + 1], w);
        }
        const double2 a = v[2 * u], b = v[2 * u + 1];
        v[2 * u] = cadd(a, b);
        v[2 * u + 1] = csub(a, b);
    }
}

// Radix-8 pass for LGM = 11 (the remainder of 11 = 4+4+3), 2 butterflies per thread.
template <int LGM, int LNS, int SIGN>
__device__ __forceinline__ void pass8x2(double2 (&v)[16], int t, const double2 *twh, const double2 *twl)
{
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if (LNS > 0) {
            const int j = (t * 2 + u) & ((1 << (LGM - 3)) - 1), k = j & ((1 << LNS) - 1);
            double2 w = twid(twh, twl, k << (LGM - LNS - 3));
            if (SIGN > 0) w = cconj(w);
            const double2 w2 = cmul(w, w), w3 = cmul(w2, w), w4 = cmul(w2, w2);
            v[8 * u + 1] = cmul(v[8 * u + 1], w);
            v[8 * u + 2] = cmul(v[8 * u + 2], w2);
            v[8 * u + 3] = cmul(v[8 * u + 3], w3);
            v[8 * u + 4] = cmul(v[8 * u + 4], w4);
            v[8 * u + 5] = cmul(v[8 * u + 5], cmul(w4, w));
            v[8 * u + 6] = cmul(v[8 * u + 6], cmul(w4, w2));
            v[8 * u + 7] = cmul(v[8 * u + 7], cmul(w4, w3));
        }
        Dft<8, SIGN>::run(&v[8 * u]);
    }
}

// Radix of the first pass of the forward (SIGN < 0) or inverse (SIGN > 0)
// transform of size 2^LGM, and of its last pass.
template <int LGM, int SIGN>
__host__ __device__ constexpr int first_radix()
{
    return SIGN < 0 ? 16 : (LGM == 13 ? 2 : LGM == 11 ? 8 : 16);
}
template <int LGM, int SIGN>
__host__ __device__ constexpr int last_radix()
{
    return SIGN > 0 ? 16 : (LGM == 13 ? 2 : LGM == 11 ? 8 : 16);
}

// Shared-memory exchange after a pass of radix R at LNS into the input
// positions of the next pass of radix RN (values per thread: 16).
template <int LGM, int R, int LNS, int RN>
__device__ __forceinline__ void exchange(double2 (&v)[16], double2 *buf, int t)
{
    constexpr int NB = 16 / R, LR = (R == 16 ? 4 : R == 8 ? 3 : 1), NBN = 16 / RN,
                  LRN = (RN == 16 ? 4 : RN == 8 ? 3 : 1);
#pragma unroll
    for (int u = 0; u < NB; u++) {
        const int j = t * NB + u;
        const int idx = ((j >> LNS) << (LNS + LR)) + (j & ((1 << LNS) - 1));
#pragma unroll
        for (int s = 0; s < R; s++) buf[padix(idx + (s << LNS))] = v[u * R + s];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < NBN; u++) {
        const int j = t * NBN + u;
#pragma unroll
        for (int s = 0; s < RN; s++) v[u * RN + s] = buf[padix(j + (s << (LGM - LRN)))];
    }
    __syncthreads();
}

// Forward (SIGN=-1, radices 16,16,16[,2]) or inverse (SIGN=+1, [2,]16,16,16)
// FFT of the values in registers; input positions of the first pass, output
// positions of the last pass.
template <int LGM, int SIGN>
__device__ __forceinline__ void fft_large(double2 (&v)[16], double2 *buf, int t, const double2 *twh,
                                          const double2 *twl)
{
    if (LGM == 11 && SIGN < 0) {  // forward: 16,16,8
        pass16<11, 0, SIGN>(v, t, twh, twl);
        exchange<11, 16, 0, 16>(v, buf, t);
        pass16<11, 4, SIGN>(v, t, twh, twl);
        exchange<11, 16, 4, 8>(v, buf, t);
        pass8x2<11, 8, SIGN>(v, t, twh, twl);
    } else if (LGM == 11) {  // inverse: 8,16,16
        pass8x2<11, 0, SIGN>(v, t, twh, twl);
        exchange<11, 8, 0, 16>(v, buf, t);
        pass16<11, 3, SIGN>(v, t, twh, twl);
        exchange<11, 16, 3, 16>(v, buf, t);
        pass16<11, 7, SIGN>(v, t, twh, twl);
    } else if (LGM == 12) {
        pass16<12, 0, SIGN>(v, t, twh, twl);
        exchange<12, 16, 0, 16>(v, buf, t);
        pass16<12, 4, SIGN>(v, t, twh, twl);
        exchange<12, 16, 4, 16>(v, buf, t);
        pass16<12, 8, SIGN>(v, t, twh, twl);
    } else if (SIGN < 0) {  // LGM == 13 forward: 16,16,16,2
        pass16<13, 0, SIGN>(v, t, twh, twl);
        exchange<13, 16, 0, 16>(v, buf, t);
        pass16<13, 4, SIGN>(v, t, twh, twl);
        exchange<13, 16, 4, 16>(v, buf, t);
        pass16<13, 8, SIGN>(v, t, twh, twl);
        exchange<13, 16, 8, 2>(v, buf, t);
        pass2x8<13, 12, SIGN>(v, t, twh, twl);
    } else {  // LGM == 13 inverse: 2,16,16,16
        pass2x8<13, 0, SIGN>(v, t, twh, twl);
        exchange<13, 2, 0, 16>(v, buf, t);
        pass16<13, 1, SIGN>(v, t, twh, twl);
        exchange<13, 16, 1, 16>(v, buf, t);
        pass16<13, 5, SIGN>(v, t, twh, twl);
        exchange<13, 16, 5, 16>(v, buf, t);
        pass16<13, 9, SIGN>(v, t, twh, twl);
    }
}

// Position in [0, M) of value i held by thread t at the input of a pass of
// radix R (R = 16: i = s; R = 2: i = 2u + s).
template <int LGM, int R>
__device__ __forceinline__ int lpos(int t, int i)
{
    if (R == 16) return t + (i << (LGM - 4));
    if (R == 8) return ((t * 2 + (i >> 3)) & ((1 << (LGM - 3)) - 1)) + ((i & 7) << (LGM - 3));
    const int u = i >> 1, s = i & 1;
    return ((t * 8 + u) & ((1 << (LGM - 1)) - 1)) + (s << (LGM - 1));
}

template <int MODE, int LGM>
__global__ void __launch_bounds__((1 << LGM) / 16, (LGM == 11 ? 4 : LGM == 12 ? 2 : 1)) fft_large_kernel(CztArgs a)
{
    constexpr int M = 1 << LGM, THREADS = M / 16;
    constexpr bool CHIRP = (MODE != FFT_ANA_BETA && MODE != FFT_SYN_BETA);
    constexpr bool SYNB = (MODE == CZT_SYN_BETA || MODE == FFT_SYN_BETA);
    // first-pass radix of the transform run first, last-pass radix of the last
    constexpr int R0 = MODE == FFT_ANA_BETA ? first_radix<LGM, +1>() : first_radix<LGM, -1>();
    constexpr int RL = MODE == FFT_SYN_BETA ? last_radix<LGM, -1>() : last_radix<LGM, +1>();
    extern __shared__ double2 smem[];
    double2 *buf = smem;
    double2 *twh = smem + padix(M) + 1;
    double2 *twl = twh + M / 64;
    double2 *ph = twl + 64;
    const int t = threadIdx.x;
    const int bl = a.bl, n = 2 * bl - 1, N = a.N, Bout = a.czt.spec.Bout;
    // row = (g or q, m or b pair); the synthesis beta modes put q on the fast
    // grid axis so that the CTAs of one m, which read the same N rows of V,
    // run together and the repeated reads hit L2
    const int g = SYNB ? blockIdx.x : blockIdx.y, rr = SYNB ? blockIdx.y : blockIdx.x;
    const double2 zero = make_double2(0.0, 0.0);

    for (int i = t; i < M / 64; i += THREADS) twh[i] = a.tw.hi[i];
    for (int i = t; i < 64; i += THREADS) twl[i] = a.tw.lo[i];
    if (SYNB && t < N) {
        double sn, cs;
        sincospi(-(double)(a.nq[g] * t) / (double)N, &sn, &cs);
        ph[t] = make_double2(cs, sn);
    }
    __syncthreads();

    double2 v[16];
    if (MODE == FFT_SYN_BETA) {
        // gamma DFT of the row with coalesced loads (b contiguous across the
        // threads), then the DCT-II reordering through shared memory: the
        // value of b goes to FFT index b/2 (b even) or (4bl-1-b)/2 (b odd)
        const bool sn = (rr + a.nq[g]) & 1;
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = zero;
        // Two rows of V at a time, the second through this transform's shared
        // memory, each thread its own values: both are in flight together (B=2048
        // N=8: 1.36 -> 1.21 ms per synthesis; in the stage kernels' smaller CTAs it
        // was slower)
        for (int gg = 0; gg < N; gg += 2) {
            const double2 *row = a.in_c + ((size_t)gg * bl + rr) * (2 * bl);
            const bool two = gg + 1 < N;
            if (two)
#pragma unroll
                for (int i = 0; i < 16; i++)
                    cp16_own(buf + t + i * THREADS, row + (size_t)bl * (2 * bl) + t + i * THREADS);
            const double2 w = ph[gg];
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = cadd(v[i], cmul(row[t + i * THREADS], w));
            if (two) {
                cp_own_wait();
                const double2 w1 = ph[gg + 1];
#pragma unroll
                for (int i = 0; i < 16; i++) v[i] = cadd(v[i], cmul(buf[t + i * THREADS], w1));
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int b = t + i * THREADS;
            double2 u = cscale(v[i], a.wq[b]);
            if (sn && (b & 1)) u = make_double2(-u.x, -u.y);
            buf[padix((b & 1) ? (4 * bl - 1 - b) >> 1 : b >> 1)] = u;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = buf[padix(lpos<LGM, R0>(t, i))];
        __syncthreads();  // the exchanges of the FFT reuse buf
    }
#pragma unroll
    for (int i = 0; i < 16 && MODE != FFT_SYN_BETA; i++) {
        const int k = lpos<LGM, R0>(t, i);
        double2 x = zero;
        if (MODE == CZT_ANA_ALPHA) {  // (g, b pair rr); Hermitian completion in m
            if (k < n) {
                const bool lo = k < bl;
                const double2 *p = a.in_c + ((size_t)g * bl + (lo ? k : n - k)) * (2 * bl) + 2 * rr;
                double2 x1, x2;
                ld_pair(p, x1, x2);
                if (!lo) { x1 = cconj(x1); x2 = cconj(x2); }
                if (k == 0) { x1.y = 0.0; x2.y = 0.0; }
                x = cmul(make_double2(x1.x - x2.y, x1.y + x2.x), a.czt.pre[k]);
            }
        } else if (MODE == CZT_SYN_ALPHA) {  // (g, b pair rr)
            if (k < n) {
                const double *p = a.in_r + (size_t)k + (size_t)n * (2 * rr + (size_t)2 * bl * g);
                x = cmul(make_double2(p[0], p[n]), a.czt.pre[k]);
            }
        } else if (MODE == CZT_ANA_BETA) {  // (g, m = rr)
            if (k < a.czt.spec.K) {
                const int mpv = k - (bl - 1), ab = mpv < 0 ? -mpv : mpv;
                x = a.in_c[((size_t)g * bl + rr) * bl + ab];
                if (((rr + N - 1) & 1) && mpv < 0) x = make_double2(-x.x, -x.y);
                x = cmul(x, a.czt.pre[k]);
            }
        } else if (MODE == FFT_ANA_BETA) {  // (g, m = rr), DCT-III input
            x = ana_beta_in(a.in_c + ((size_t)g * bl + rr) * bl, k, bl, (rr + N - 1) & 1, a.czt.pre);
        } else {  // CZT_SYN_BETA, (q = g, m = rr), k = b
            if (k < 2 * bl) {
                double2 u = zero;
                for (int gg = 0; gg < N; gg++)
                    u = cadd(u, cmul(a.in_c[((size_t)gg * bl + rr) * (2 * bl) + k], ph[gg]));
                x = cmul(cscale(u, a.wq[k]), a.czt.pre[k]);
            }
        }
        v[i] = x;
    }

    if (MODE == FFT_ANA_BETA) {
        fft_large<LGM, +1>(v, buf, t, twh, twl);
    } else if (MODE == FFT_SYN_BETA) {
        fft_large<LGM, -1>(v, buf, t, twh, twl);
    } else {
        fft_large<LGM, -1>(v, buf, t, twh, twl);
        constexpr int RF = last_radix<LGM, -1>();
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = cmul(v[i], hf_at<MODE>(a.czt.Hf, lpos<LGM, RF>(t, i), M));
        fft_large<LGM, +1>(v, buf, t, twh, twl);
    }

    if (MODE == CZT_ANA_BETA || MODE == FFT_ANA_BETA || MODE == CZT_ANA_ALPHA) {
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int b = lpos<LGM, RL>(t, i);
            if (b >= Bout) continue;
            if (MODE == FFT_ANA_BETA) {
                const bool sn = (rr + N - 1) & 1;
                const double2 *X = a.in_c + ((size_t)g * bl + rr) * bl;
                int bo;
                const double2 y = ana_beta_out(v[i], b, bl, sn, sn ? X[0] : zero, &bo);
                a.out_c[((size_t)g * bl + rr) * (2 * bl) + bo] = y;
                continue;
            }
            const double2 y = CHIRP ? cmul(v[i], a.czt.post[b]) : v[i];
            if (MODE == CZT_ANA_ALPHA) {
                double *p = a.out_r + (size_t)b + (size_t)n * (2 * rr + (size_t)2 * bl * g);
                p[0] = y.x;
                p[n] = y.y;
            } else {
                a.out_c[((size_t)g * bl + rr) * (2 * bl) + b] = y;
            }
        }
        return;
    }
    // pair stores through shared memory
#pragma unroll
    for (int i = 0; i < 16; i++) buf[padix(lpos<LGM, RL>(t, i))] = v[i];
    __syncthreads();
    if (MODE == CZT_SYN_ALPHA) {
        for (int m = t; m < bl; m += THREADS) {
            const int mc = (m == 0) ? 0 : n - m;
            const double2 Z = cmul(buf[padix(m)], a.czt.post[m]);
            const double2 Zc = cconj(cmul(buf[padix(mc)], a.czt.post[mc]));
            const double2 sm = cadd(Z, Zc), d = csub(Z, Zc);
            const double hh = 0.5 * a.scale;
            st_pair(a.out_c + ((size_t)g * bl + m) * (2 * bl) + 2 * rr, make_double2(sm.x * hh, sm.y * hh),
                    make_double2(d.y * hh, -d.x * hh));
        }
        return;
    }
    for (int mpv = t; mpv < bl; mpv += THREADS) {
        double2 y;
        if (MODE == CZT_SYN_BETA) {
            const int t0 = bl - 1 + mpv, t1 = bl - 1 - mpv;
            y = cmul(buf[padix(t0)], a.czt.post[t0]);
            double2 z = cmul(buf[padix(t1)], a.czt.post[t1]);
            if (mpv > 0) {
                if ((rr + a.nq[g]) & 1) z = make_double2(-z.x, -z.y);
                y = cadd(y, z);
            }
        } else {
            y = syn_beta_out(buf[padix(mpv)], buf[padix((M - mpv) & (M - 1))], mpv, (rr + a.nq[g]) & 1, a.czt.pre);
        }
        a.out_c[((size_t)g * bl + rr) * a.out_stride + mpv] = y;
    }
}

// ===========================================================================
// Stages with the input prefetched (M = 4096, 8192): synthesis alpha and
// analysis beta
//
// A persistent form of fft_large_kernel for the two modes whose input row is
// contiguous in HBM: each CTA loops over rows and copies the next row's input
// into shared memory with cp.async while the current row's transforms run,
// so the input's DRAM latency is hidden behind the FFT arithmetic instead of
// stalling every warp of the CTA at the start of each row.  The twiddle
// tables are loaded once per CTA.  Staged input per row:
//   CZT_SYN_ALPHA (row = (g, b pair)): the two real rows of the b pair,
//     2n contiguous doubles at a multiple of 2n doubles from in_r;
//   FFT_ANA_BETA (row = (g, m)): Tg(g, m, 0..bl-1), bl complex values.
// ===========================================================================
__device__ __forceinline__ void pf_cp16(void *smem, const void *gmem)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void pf_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void pf_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// 16-byte chunks of one row's staged input.
template <int MODE>
__host__ __device__ constexpr int pf_chunks(int bl)
{
    return MODE == CZT_SYN_ALPHA ? 2 * bl - 1 : bl;
}

// Issues the copies of row r's input into stg.
template <int MODE, int THREADS>
__device__ __forceinline__ void pf_prefetch(const CztArgs &a, int r, double2 *stg, int t)
{
    const int bl = a.bl, n = 2 * bl - 1, g = r / bl, rr = r - g * bl;
    const double2 *base;
    if (MODE == CZT_SYN_ALPHA)
        base = reinterpret_cast<const double2 *>(a.in_r + (size_t)n * (2 * rr + (size_t)2 * bl * g));
    else
        base = a.in_c + ((size_t)g * bl + rr) * bl;
    for (int i = t; i < pf_chunks<MODE>(bl); i += THREADS) pf_cp16(stg + i, base + i);
}

template <int MODE, int LGM>
__global__ void __launch_bounds__((1 << LGM) / 16, (LGM == 11 ? 4 : LGM == 12 ? 2 : 1)) fft_pf_kernel(CztArgs a)
{
    static_assert(MODE == CZT_SYN_ALPHA || MODE == FFT_ANA_BETA, "contiguous-input stages only");
    constexpr int M = 1 << LGM, THREADS = M / 16;
    // first-pass radix of the transform run first (as fft_large_kernel)
    constexpr int R0 = MODE == FFT_ANA_BETA ? first_radix<LGM, +1>() : first_radix<LGM, -1>();
    extern __shared__ double2 smem[];
    double2 *buf = smem;
    double2 *twh = smem + padix(M) + 1;
    double2 *twl = twh + M / 64;
    double2 *stg = twl + 64;
    const int t = threadIdx.x;
    const int bl = a.bl, n = 2 * bl - 1, rows = a.rows, N = a.N, Bout = a.czt.spec.Bout;
    const double2 zero = make_double2(0.0, 0.0);

    for (int i = t; i < M / 64; i += THREADS) twh[i] = a.tw.hi[i];
    for (int i = t; i < 64; i += THREADS) twl[i] = a.tw.lo[i];
    if ((int)blockIdx.x < rows) pf_prefetch<MODE, THREADS>(a, blockIdx.x, stg, t);
    pf_commit();

    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const int g = r / bl, rr = r - g * bl;
        pf_wait_all();
        __syncthreads();  // row r staged; the previous row's reads of buf done
        double2 v[16];
        bool sn = false;     // FFT_ANA_BETA: sin row
        double2 x0 = zero;   // FFT_ANA_BETA: the row's X(0)
        if (MODE == CZT_SYN_ALPHA) {
            const double *sd = reinterpret_cast<const double *>(stg);
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int k = lpos<LGM, R0>(t, i);
                v[i] = (k < n) ? cmul(make_double2(sd[k], sd[n + k]), a.czt.pre[k]) : zero;
            }
        } else {  // DCT-III input, as fft_large_kernel's FFT_ANA_BETA load
            sn = (rr + N - 1) & 1;
            x0 = stg[0];
            // ana_beta_in with M = 2 bl and the half of each k known from i: no
            // conditions between the twiddle loads, which are in flight together
            double2 w[16];
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int k = lpos<LGM, R0>(t, i);
                const bool up = R0 == 8 ? (i & 7) >= 4 : i >= 8;
                w[i] = __ldg(a.czt.pre + (up ? (M - k) & (M / 2 - 1) : k));
            }
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int k = lpos<LGM, R0>(t, i);
                const bool up = R0 == 8 ? (i & 7) >= 4 : i >= 8;
                const double2 x = stg[up ? (M - k) & (M / 2 - 1) : k];
                const double2 y = cmul(x, up ? cconj(w[i]) : w[i]);
                v[i] = !sn ? y : up ? make_double2(-y.y, y.x) : make_double2(y.y, -y.x);
                if (up ? k == M / 2 : (sn && k == 0)) v[i] = zero;
            }
        }
        __syncthreads();  // staging free: copy the next row while this one runs
        if (r + (int)gridDim.x < rows) pf_prefetch<MODE, THREADS>(a, r + gridDim.x, stg, t);
        pf_commit();

        if (MODE == CZT_SYN_ALPHA) {
            fft_large<LGM, -1>(v, buf, t, twh, twl);
            constexpr int RF = last_radix<LGM, -1>();
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = cmul(v[i], hf_at<MODE>(a.czt.Hf, lpos<LGM, RF>(t, i), M));
            fft_large<LGM, +1>(v, buf, t, twh, twl);
            // pair split through shared memory, as fft_large_kernel
#pragma unroll
            for (int i = 0; i < 16; i++) buf[padix(lpos<LGM, 16>(t, i))] = v[i];
            __syncthreads();
            for (int m = t; m < bl; m += THREADS) {
                const int mc = (m == 0) ? 0 : n - m;
                const double2 Z = cmul(buf[padix(m)], a.czt.post[m]);
                const double2 Zc = cconj(cmul(buf[padix(mc)], a.czt.post[mc]));
                const double2 sm = cadd(Z, Zc), d = csub(Z, Zc);
                const double hh = 0.5 * a.scale;
                st_pair(a.out_c + ((size_t)g * bl + m) * (2 * bl) + 2 * rr, make_double2(sm.x * hh, sm.y * hh),
                        make_double2(d.y * hh, -d.x * hh));
            }
        } else {
            fft_large<LGM, +1>(v, buf, t, twh, twl);
#pragma unroll
            for (int i = 0; i < 16; i++) {
                int b;
                const double2 y = ana_beta_out(v[i], lpos<LGM, 16>(t, i), bl, sn, x0, &b);
                a.out_c[((size_t)g * bl + rr) * (2 * bl) + b] = y;
            }
        }
    }
    pf_wait_all();
}

// ===========================================================================
// Prime-factor alpha stages at bl = 2048: n = 2bl-1 = 4095 = 5 * 7 * 9 * 13
//
// For the smooth odd length of the full-band scales at B = 2048 the alpha
// transforms (the c2r of s2dw_core_mod.f90:746-768 and the r2c of :1104-1130,
// two real rows packed into one complex transform as in the Bluestein
// engines) run as a Good-Thomas prime-factor DFT: the 4095 values of a row go
// into shared memory in the 4-D layout L = d1 + 5 d2 + 35 d3 + 315 d4 with
// input digits d_i = (n u_i) mod R_i, u_i = (4095/R_i)^-1 mod R_i = 4, 2, 2, 9;
// plain DFTs of length R_i = 5, 7, 9, 13 run along each dimension in place (no
// twiddles between them); output k sits at digits k mod R_i.  Each small DFT
// uses the symmetric pairs x_k +- x_{R-k}: (R-1)^2 real-by-complex products
// instead of R^2.  About 40 FP64 operations per point against ~240 for the
// 8192-point Bluestein convolution of the general engine.
// ===========================================================================
// Load phase of the prime-factor alpha kernels: the row pair (g, rr) of one
// transform of odd length N into shared memory, value m at X[pos(m)], with
// all of a thread's global loads in flight before the first shared store.
// Analysis: only the rows m < bl = (N+1)/2 are read; the Hermitian completion
// m >= bl is their conjugate (z(N - m) from the same two values).  Synthesis:
// the two real rows, z = w(:, b1) + i w(:, b2).
template <int MODE, int NT, int N, typename Pos>
__device__ __forceinline__ void pfa_load(const CztArgs &a, double2 *X, Pos pos)
{
    constexpr int BL = (N + 1) / 2;
    const int t = threadIdx.x, g = blockIdx.y, rr = blockIdx.x;
    if (MODE == CZT_ANA_ALPHA) {
        constexpr int PB = (BL + NT - 1) / NT;
        double2 x1[PB], x2[PB];
#pragma unroll
        for (int i = 0; i < PB; i++) {
            const int m = t + i * NT;
            if (m < BL) ld_pair(a.in_c + ((size_t)g * BL + m) * (2 * BL) + 2 * rr, x1[i], x2[i]);
        }
#pragma unroll
        for (int i = 0; i < PB; i++) {
            const int m = t + i * NT;
            if (m < BL) {
                if (m == 0) { x1[i].y = 0.0; x2[i].y = 0.0; }
                X[pos(m)] = make_double2(x1[i].x - x2[i].y, x1[i].y + x2[i].x);
                if (m > 0) X[pos(N - m)] = make_double2(x1[i].x + x2[i].y, x2[i].x - x1[i].y);
            }
        }
    } else {
        constexpr int PB = (N + NT - 1) / NT;
        const double *p = a.in_r + (size_t)N * (2 * rr + (size_t)2 * BL * g);
        double z0[PB], z1[PB];
#pragma unroll
        for (int i = 0; i < PB; i++) {
            const int m = t + i * NT;
            if (m < N) {
                z0[i] = p[m];
                z1[i] = p[N + m];
            }
        }
#pragma unroll
        for (int i = 0; i < PB; i++) {
            const int m = t + i * NT;
            if (m < N) X[pos(m)] = make_double2(z0[i], z1[i]);
        }
    }
}

constexpr int PFA_N = 4095, PFA_THREADS = 256;

// DFTs of length R along the dimension of stride S of the 4-D layout.
template <int R, int S, int SIGN>
__device__ __forceinline__ void pfa_stage(double2 *sm, int t)
{
    for (int d = t; d < PFA_N / R; d += PFA_THREADS) {
        const int base = (d % S) + (d / S) * (S * R);
        double2 x[R];
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = sm[base + r * S];
        pfa_dft<R, SIGN>(x);
#pragma unroll
        for (int r = 0; r < R; r++) sm[base + r * S] = x[r];
    }
}

__device__ __forceinline__ int pfa_in_pos(int n)
{
    return (n * 4) % 5 + 5 * ((n * 2) % 7) + 35 * ((n * 2) % 9) + 315 * ((n * 9) % 13);
}
__device__ __forceinline__ int pfa_out_pos(int k) { return k % 5 + 5 * (k % 7) + 35 * (k % 9) + 315 * (k % 13); }

// One CTA per (g, b pair): the two real rows of the pair, as fft_large_kernel.
template <int MODE>
__global__ void __launch_bounds__(PFA_THREADS, 3) pfa_alpha_kernel(CztArgs a)
{
    static_assert(MODE == CZT_ANA_ALPHA || MODE == CZT_SYN_ALPHA, "alpha stages only");
    constexpr int SIGN = MODE == CZT_ANA_ALPHA ? +1 : -1;
    extern __shared__ double2 smem[];
    const int t = threadIdx.x;
    const int bl = a.bl, n = PFA_N;  // n = 2 bl - 1
    const int g = blockIdx.y, rr = blockIdx.x;
    pfa_load<MODE, PFA_THREADS, PFA_N>(a, smem, [](int m) { return pfa_in_pos(m); });
    __syncthreads();
    pfa_stage<5, 1, SIGN>(smem, t);
    __syncthreads();
    pfa_stage<7, 5, SIGN>(smem, t);
    __syncthreads();
    pfa_stage<9, 35, SIGN>(smem, t);
    __syncthreads();
    pfa_stage<13, 315, SIGN>(smem, t);
    __syncthreads();
    if (MODE == CZT_ANA_ALPHA) {
        for (int k = t; k < n; k += PFA_THREADS) {
            const double2 y = smem[pfa_out_pos(k)];
            double *p = a.out_r + (size_t)k + (size_t)n * (2 * rr + (size_t)2 * bl * g);
            p[0] = y.x;
            p[n] = y.y;
        }
    } else {  // even / odd split of the two real rows' spectra, m < bl
        const double hh = 0.5 * a.scale;
        for (int m = t; m < bl; m += PFA_THREADS) {
            const double2 Z = smem[pfa_out_pos(m)];
            const double2 Zc = cconj(smem[pfa_out_pos(m == 0 ? 0 : n - m)]);
            const double2 sm = cadd(Z, Zc), d = csub(Z, Zc);
            st_pair(a.out_c + ((size_t)g * bl + m) * (2 * bl) + 2 * rr, make_double2(sm.x * hh, sm.y * hh),
                    make_double2(d.y * hh, -d.x * hh));
        }
    }
}

// ---------------------------------------------------------------------------
// Prime-factor alpha stages at bl = 1024: n = 2047 = 23 * 89
//
// Good-Thomas over 23 x 89 as above (layout L = d1 + 23 d2, input digits
// (n 15) mod 23 and (n 31) mod 89, output digits k mod 23, k mod 89).  The
// length-89 DFTs run by Rader's algorithm: with the primitive root g = 3,
// y_{g^r} = x_0 + sum_q x_{g^-q} w_{r-q}, w_j = exp(SIGN 2 pi i g^j / 89), a cyclic
// convolution of length 88 done as a forward DFT of 88 = 8 x 11 (Good-Thomas
// again: radix-8 in registers, then length 11), a product with the DFT of w
// (g_rader_w, built once per device by rader_init_kernel), and the inverse
// DFT; y_0 = x_0 + the convolution input's sum.  About 60 FP64 operations per
// point against ~240 for the 4096-point Bluestein convolution.
// ---------------------------------------------------------------------------
constexpr int PFB_N = 2047, PFB_THREADS = 128;
constexpr int PFB_P = 25;              // pitch of d2 in the shared row
constexpr int PFB_XS = PFB_P * 89;     // shared row size
constexpr int PFB_SP = 103;            // pitch of a Rader column (positions i + 9 j, i < 8, j < 11)

// per position L = i + 8 j of the 88-layout (input digits (q 3) mod 8,
// (q 7) mod 11): the length-89 index g^-q whose value goes there, and g^q,
// where the convolution's output at L goes
__constant__ int c_rader_src[88] = {
    1, 77, 55, 52, 88, 12, 34, 37, 32, 61, 69, 62, 57, 28, 20, 27, 45, 83, 72, 26, 44, 6, 17, 63, 16, 75, 79, 31,
    73, 14, 10, 58, 67, 86, 36, 13, 22, 3, 53, 76, 8, 82, 84, 60, 81, 7, 5, 29, 78, 43, 18, 51, 11, 46, 71, 38, 4,
    41, 42, 30, 85, 48, 47, 59, 39, 66, 9, 70, 50, 23, 80, 19, 2, 65, 21, 15, 87, 24, 68, 74, 64, 33, 49, 35, 25,
    56, 40, 54};
__constant__ int c_rader_dst[88] = {
    1, 37, 34, 12, 88, 52, 55, 77, 64, 54, 40, 56, 25, 35, 49, 33, 2, 74, 68, 24, 87, 15, 21, 65, 39, 19, 80, 23,
    50, 70, 9, 66, 4, 59, 47, 48, 85, 30, 42, 41, 78, 38, 71, 46, 11, 51, 18, 43, 8, 29, 5, 7, 81, 60, 84, 82, 67,
    76, 53, 3, 22, 13, 36, 86, 16, 58, 10, 14, 73, 31, 79, 75, 45, 63, 17, 6, 44, 26, 72, 83, 32, 27, 20, 28, 57,
    62, 69, 61};
// [0]: SIGN -1, [1]: SIGN +1; entry L_out(k) = k mod 8 + 8 (k mod 11) holds
// (1/88) sum_j w_j exp(-2 pi i j k / 88)
__device__ double2 g_rader_w[2][88];

__global__ void rader_init_kernel()
{
    const int sgn = blockIdx.x ? 1 : -1, k = threadIdx.x;
    if (k >= 88) return;
    double re = 0.0, im = 0.0;
    int gj = 1;  // 3^j mod 89
    for (int j = 0; j < 88; j++) {
        double s1, c1, s2, c2;
        sincospi(2.0 * sgn * gj / 89.0, &s1, &c1);
        sincospi(-2.0 * ((j * k) % 88) / 88.0, &s2, &c2);
        re += c1 * c2 - s1 * s2;
        im += c1 * s2 + s1 * c2;
        gj = (gj * 3) % 89;
    }
    g_rader_w[blockIdx.x][k % 8 + 8 * (k % 11)] = make_double2(re / 88.0, im / 88.0);
}

template <int MODE>
__global__ void __launch_bounds__(PFB_THREADS, 3) pfa2047_alpha_kernel(CztArgs a)
{
    static_assert(MODE == CZT_ANA_ALPHA || MODE == CZT_SYN_ALPHA, "alpha stages only");
    constexpr int SIGN = MODE == CZT_ANA_ALPHA ? +1 : -1, NT = PFB_THREADS;
    extern __shared__ double2 smem[];
    // the row in layout d1 + 25 d2 (pitch 25: conflict-free shared-memory
    // access for the length-23 DFTs, two-way for the output gather); the 23
    // Rader convolutions in layout i + 9 j (pitch 103 per column: with the
    // work items (c1, j) taken c1-fastest, the gathers from the row, the
    // column stores and their reads back are conflict-free but for the
    // items where j changes)
    double2 *X = smem;
    double2 *Sc = smem + PFB_XS;
    double2 *X0 = Sc + 23 * PFB_SP;
    const int t = threadIdx.x;
    const int bl = a.bl, n = PFB_N;  // n = 2 bl - 1
    const int g = blockIdx.y, rr = blockIdx.x;
    pfa_load<MODE, NT, PFB_N>(a, X, [](int m) { return (m * 15) % 23 + PFB_P * ((m * 31) % 89); });
    __syncthreads();
    // length-23 DFTs along d1
    for (int d2 = t; d2 < 89; d2 += NT) {
        double2 x[23];
#pragma unroll
        for (int r = 0; r < 23; r++) x[r] = X[PFB_P * d2 + r];
        pfa_dft_out<23, SIGN>(x, X, PFB_P * d2, 1);
    }
    __syncthreads();
    // length-89 DFTs along d2 (column c1) by Rader: forward length-8 DFTs of
    // the permuted inputs
    for (int u = t; u < 23 * 11; u += NT) {
        const int c1 = u % 23, j = u / 23;
        double2 v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = X[c1 + PFB_P * c_rader_src[i + 8 * j]];
        Dft<8, -1>::run(v);
#pragma unroll
        for (int i = 0; i < 8; i++) Sc[c1 * PFB_SP + i + 9 * j] = v[i];
        if (j == 0) X0[c1] = X[c1];
    }
    __syncthreads();
    // forward length-11 DFTs, product with the DFT of w, inverse length-11
    for (int u = t; u < 23 * 8; u += NT) {
        const int c1 = u / 8, i = u % 8;
        double2 v[11];
#pragma unroll
        for (int jj = 0; jj < 11; jj++) v[jj] = Sc[c1 * PFB_SP + i + 9 * jj];
        pfa_dft<11, -1>(v);
        if (i == 0) X[c1] = cadd(X0[c1], v[0]);  // y_0 = x_0 + sum of the other inputs
#pragma unroll
        for (int kk = 0; kk < 11; kk++) v[kk] = cmul(v[kk], g_rader_w[SIGN > 0 ? 1 : 0][i + 8 * kk]);
        pfa_dft<11, +1>(v);
#pragma unroll
        for (int jj = 0; jj < 11; jj++) Sc[c1 * PFB_SP + i + 9 * jj] = v[jj];
    }
    __syncthreads();
    // inverse length-8 DFTs; y_{g^q} = x_0 + convolution
    for (int u = t; u < 23 * 11; u += NT) {
        const int c1 = u % 23, j = u / 23;
        double2 v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = Sc[c1 * PFB_SP + i + 9 * j];
        Dft<8, +1>::run(v);
        const double2 x0 = X0[c1];
#pragma unroll
        for (int i = 0; i < 8; i++) X[c1 + PFB_P * c_rader_dst[i + 8 * j]] = cadd(x0, v[i]);
    }
    __syncthreads();
    if (MODE == CZT_ANA_ALPHA) {
        for (int k = t; k < n; k += NT) {
            const double2 y = X[k % 23 + PFB_P * (k % 89)];
            double *p = a.out_r + (size_t)k + (size_t)n * (2 * rr + (size_t)2 * bl * g);
            p[0] = y.x;
            p[n] = y.y;
        }
    } else {
        const double hh = 0.5 * a.scale;
        for (int m = t; m < bl; m += NT) {
            const int mc = m == 0 ? 0 : n - m;
            const double2 Z = X[m % 23 + PFB_P * (m % 89)];
            const double2 Zc = cconj(X[mc % 23 + PFB_P * (mc % 89)]);
            const double2 sm = cadd(Z, Zc), d = csub(Z, Zc);
            st_pair(a.out_c + ((size_t)g * bl + m) * (2 * bl) + 2 * rr, make_double2(sm.x * hh, sm.y * hh),
                    make_double2(d.y * hh, -d.x * hh));
        }
    }
}

// ---------------------------------------------------------------------------
// Row pairs of an alpha stage into and out of shared memory: RP pairs (g, rr)
// of the transform of odd length N = 2 bl - 1, value m of pair r at at(r, m).
// Consecutive threads take consecutive pairs of one m where the rows are
// strided (32 bytes per pair: RP pairs are one contiguous piece), consecutive
// values where they are contiguous.
// ---------------------------------------------------------------------------
template <int MODE, int N, int RP, int NT = ST_THREADS, typename At>
__device__ __forceinline__ void alpha_rows_in(const StageEnt &e, int cta, At at)
{
    constexpr int BL = (N + 1) / 2;
    const int t = threadIdx.x, row0 = cta * RP, per = e.rows_map;
    if (MODE == CZT_ANA_ALPHA) {  // rows m < bl; the Hermitian half from the same values
        constexpr int IT = (RP * BL + NT - 1) / NT, U = IT < 6 ? IT : 6;  // loads in flight
        for (int i0 = t; i0 < RP * BL; i0 += U * NT) {
            double2 x1[U], x2[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 + u * NT, r = i % RP, m = i / RP, row = row0 + r;
                if (m >= BL || row >= e.rows) continue;
                const int k = row / per, gr = row - k * per, g = gr / BL, rr = gr - g * BL;
                ld_pair(static_cast<const double2 *>(e.in) + k * e.in_map + ((size_t)g * BL + m) * (2 * BL) + 2 * rr,
                        x1[u], x2[u]);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 + u * NT, r = i % RP, m = i / RP;
                if (m >= BL || row0 + r >= e.rows) continue;
                if (m == 0) { x1[u].y = 0.0; x2[u].y = 0.0; }
                at(r, m) = make_double2(x1[u].x - x2[u].y, x1[u].y + x2[u].x);
                if (m > 0) at(r, N - m) = make_double2(x1[u].x + x2[u].y, x2[u].x - x1[u].y);
            }
        }
    } else {  // the two real rows of a pair, z = w(:, b1) + i w(:, b2)
        constexpr int IT = (RP * N + NT - 1) / NT, U = IT < 8 ? IT : 8;
        for (int i0 = t; i0 < RP * N; i0 += U * NT) {
            double z0[U], z1[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 + u * NT, r = i / N, m = i - r * N, row = row0 + r;
                if (i >= RP * N || row >= e.rows) continue;
                const int k = row / per, gr = row - k * per;
                const double *p = static_cast<const double *>(e.in) + k * e.in_map + (size_t)(2 * N) * gr + m;
                z0[u] = __ldg(p);
                z1[u] = __ldg(p + N);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 + u * NT, r = i / N, m = i - r * N;
                if (i < RP * N && row0 + r < e.rows) at(r, m) = make_double2(z0[u], z1[u]);
            }
        }
    }
}

template <int MODE, int N, int RP, int NT = ST_THREADS, typename At>
__device__ __forceinline__ void alpha_rows_out(const StageEnt &e, int cta, At at)
{
    constexpr int BL = (N + 1) / 2;
    const int t = threadIdx.x, row0 = cta * RP, per = e.rows_map;
    if (MODE == CZT_ANA_ALPHA) {
        for (int i = t; i < RP * N; i += NT) {
            const int r = i / N, m = i - r * N, row = row0 + r;
            if (row >= e.rows) continue;
            const int k = row / per, gr = row - k * per;
            const double2 y = at(r, m);
            double *p = static_cast<double *>(e.out) + k * e.out_map + (size_t)(2 * N) * gr + m;
            p[0] = y.x;
            p[N] = y.y;
        }
    } else {
        const double hh = 0.5 * e.scale;
        for (int i = t; i < RP * BL; i += NT) {
            const int r = i % RP, m = i / RP, row = row0 + r;
            if (row >= e.rows) continue;
            const int k = row / per, gr = row - k * per, g = gr / BL, rr = gr - g * BL;
            const double2 Z = at(r, m), Zc = cconj(at(r, m == 0 ? 0 : N - m));
            const double2 sm = cadd(Z, Zc), d = csub(Z, Zc);
            st_pair(static_cast<double2 *>(e.out) + k * e.out_map + ((size_t)g * BL + m) * (2 * BL) + 2 * rr,
                    make_double2(sm.x * hh, sm.y * hh), make_double2(d.y * hh, -d.x * hh));
        }
    }
}

// ---------------------------------------------------------------------------
// Prime-factor alpha stages of the small scales: n = 2bl - 1 = R1 R2 R3 with
// small pairwise coprime factors (bl = 2: 3; 4: 7; 8: 3 * 5; 32: 7 * 9;
// 128: 3 * 5 * 17; bl = 16 and 64, whose n is prime, are Bluestein transforms), Good-Thomas with direct symmetric-pair DFTs (factors of 1
// are skipped), RP row pairs per CTA.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int pfs_inv(int a, int r)
{
    int x = 1;
    while (r > 1 && (a * x) % r != 1) x++;
    return x;
}
// row pairs per CTA: about a thousand values
__host__ __device__ constexpr int pfs_rows(int n) { return n >= 255 ? 4 : n >= 63 ? 8 : n >= 15 ? 16 : 32; }

template <int N, int R, int S, int RP, int SIGN, int NT = ST_THREADS>
__device__ __forceinline__ void pfs_stage(double2 *sm, int t)
{
    for (int i = t; i < RP * (N / R); i += NT) {
        const int d = i % (N / R), base = (i / (N / R)) * N + (d % S) + (d / S) * (S * R);
        double2 x[R];
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = sm[base + r * S];
        pfa_dft<R, SIGN>(x);
#pragma unroll
        for (int r = 0; r < R; r++) sm[base + r * S] = x[r];
    }
}

template <int R1, int R2, int R3, int MODE>
__device__ __forceinline__ void pfs_rows_run(const StageEnt &e, int cta, double2 *smem)
{
    constexpr int SIGN = MODE == CZT_ANA_ALPHA ? +1 : -1;
    constexpr int N = R1 * R2 * R3, RP = pfs_rows(N);
    constexpr int U1 = pfs_inv((N / R1) % R1, R1), U2 = pfs_inv((N / R2) % R2, R2), U3 = pfs_inv((N / R3) % R3, R3);
    const int t = threadIdx.x;
    alpha_rows_in<MODE, N, RP>(e, cta, [&](int r, int m) -> double2 & {
        return smem[r * N + (m * U1) % R1 + R1 * ((m * U2) % R2) + R1 * R2 * ((m * U3) % R3)];
    });
    __syncthreads();
    if constexpr (R1 > 1) {
        pfs_stage<N, R1, 1, RP, SIGN>(smem, t);
        __syncthreads();
    }
    if constexpr (R2 > 1) {
        pfs_stage<N, R2, R1, RP, SIGN>(smem, t);
        __syncthreads();
    }
    if constexpr (R3 > 1) {
        pfs_stage<N, R3, R1 * R2, RP, SIGN>(smem, t);
        __syncthreads();
    }
    alpha_rows_out<MODE, N, RP>(e, cta, [&](int r, int k) -> double2 {
        return smem[r * N + k % R1 + R1 * (k % R2) + R1 * R2 * (k % R3)];
    });
}

// ---------------------------------------------------------------------------
// Prime-factor alpha stages at bl = 256: n = 511 = 7 * 73
//
// As at bl = 1024 with 23 x 89 replaced by 7 x 73: row layout d1 + 9 d2 (input
// digits (5n) mod 7, (21n) mod 73), length-7 DFTs along d1, and the length-73
// DFTs by Rader's algorithm with the primitive root 5: a cyclic convolution of
// length 72 = 8 x 9 (radix 8 in registers, then length 9; layout L = i + 8 j
// with input digits q mod 8, (8q) mod 9), the product with the DFT of
// w_j = exp(SIGN 2 pi i 5^j / 73) (g_rader73_w, built with the length-89 table
// by pfa_prepare), and the inverse.
// ---------------------------------------------------------------------------
constexpr int PFD_N = 511;
constexpr int PFD_P = 9;               // pitch of d2 in the shared row
constexpr int PFD_XS = PFD_P * 73;
constexpr int PFD_SP = 83;             // pitch of a Rader column (positions i + 9 j, i < 8, j < 9)

__constant__ int c_rader73_src[72] = {
    1, 22, 46, 63, 72, 51, 27, 10, 37, 11, 23, 68, 36, 62, 50, 5, 55, 42, 48, 34, 18, 31, 25, 39, 64, 21, 24, 17,
    9, 52, 49, 56, 32, 47, 12, 45, 41, 26, 61, 28, 16, 60, 6, 59, 57, 13, 67, 14, 8, 30, 3, 66, 65, 43, 70, 7, 4,
    15, 38, 33, 69, 58, 35, 40, 2, 44, 19, 53, 71, 29, 54, 20};
__constant__ int c_rader73_dst[72] = {
    1, 10, 27, 51, 72, 63, 46, 22, 2, 20, 54, 29, 71, 53, 19, 44, 4, 40, 35, 58, 69, 33, 38, 15, 8, 7, 70, 43, 65,
    66, 3, 30, 16, 14, 67, 13, 57, 59, 6, 60, 32, 28, 61, 26, 41, 45, 12, 47, 64, 56, 49, 52, 9, 17, 24, 21, 55,
    39, 25, 31, 18, 34, 48, 42, 37, 5, 50, 62, 36, 68, 23, 11};
// [0]: SIGN -1, [1]: SIGN +1; entry k mod 8 + 8 (k mod 9) holds
// (1/72) sum_j w_j exp(-2 pi i j k / 72)
__device__ double2 g_rader73_w[2][72];

__global__ void rader73_init_kernel()
{
    const int sgn = blockIdx.x ? 1 : -1, k = threadIdx.x;
    if (k >= 72) return;
    double re = 0.0, im = 0.0;
    int gj = 1;  // 5^j mod 73
    for (int j = 0; j < 72; j++) {
        double s1, c1, s2, c2;
        sincospi(2.0 * sgn * gj / 73.0, &s1, &c1);
        sincospi(-2.0 * ((j * k) % 72) / 72.0, &s2, &c2);
        re += c1 * c2 - s1 * s2;
        im += c1 * s2 + s1 * c2;
        gj = (gj * 5) % 73;
    }
    g_rader73_w[blockIdx.x][k % 8 + 8 * (k % 9)] = make_double2(re / 72.0, im / 72.0);
}

// Two row pairs per CTA: 126 or 112 threads of 128 work in the convolution's
// phases, and five CTAs hold ten rows on an SM (one row pair per CTA: 63 or 56
// threads, six rows).
constexpr int PFD_RP = 2;
constexpr int PFD_ROW = PFD_XS + 7 * PFD_SP + 7;  // shared values of a row

template <int MODE>
__device__ __forceinline__ void pfa511_rows(const StageEnt &e, int cta, double2 *smem)
{
    constexpr int SIGN = MODE == CZT_ANA_ALPHA ? +1 : -1;
    constexpr int NT = ST_THREADS, RP = PFD_RP;
    const int t = threadIdx.x;
    alpha_rows_in<MODE, PFD_N, RP>(e, cta, [&](int r, int m) -> double2 & {
        return smem[r * PFD_ROW + (m * 5) % 7 + PFD_P * ((m * 21) % 73)];
    });
    __syncthreads();
    // length-7 DFTs along d1
    for (int i = t; i < RP * 73; i += NT) {
        double2 *X = smem + (i / 73) * PFD_ROW + PFD_P * (i % 73);
        double2 x[7];
#pragma unroll
        for (int r = 0; r < 7; r++) x[r] = X[r];
        pfa_dft_out<7, SIGN>(x, X, 0, 1);
    }
    __syncthreads();
    // length-73 DFTs along d2 (column c1) by Rader: forward length-8 DFTs
    for (int i = t; i < RP * 7 * 9; i += NT) {
        double2 *X = smem + (i / 63) * PFD_ROW, *Sc = X + PFD_XS, *X0 = Sc + 7 * PFD_SP;
        const int u = i % 63, c1 = u % 7, j = u / 7;
        double2 v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = X[c1 + PFD_P * c_rader73_src[k + 8 * j]];
        Dft<8, -1>::run(v);
#pragma unroll
        for (int k = 0; k < 8; k++) Sc[c1 * PFD_SP + k + 9 * j] = v[k];
        if (j == 0) X0[c1] = X[c1];
    }
    __syncthreads();
    // forward length-9 DFTs, product with the DFT of w, inverse length-9
    for (int k = t; k < RP * 7 * 8; k += NT) {
        double2 *X = smem + (k / 56) * PFD_ROW, *Sc = X + PFD_XS, *X0 = Sc + 7 * PFD_SP;
        const int u = k % 56, c1 = u / 8, i = u % 8;
        double2 v[9];
#pragma unroll
        for (int jj = 0; jj < 9; jj++) v[jj] = Sc[c1 * PFD_SP + i + 9 * jj];
        pfa_dft<9, -1>(v);
        if (i == 0) X[c1] = cadd(X0[c1], v[0]);  // y_0 = x_0 + sum of the other inputs
#pragma unroll
        for (int kk = 0; kk < 9; kk++) v[kk] = cmul(v[kk], g_rader73_w[SIGN > 0 ? 1 : 0][i + 8 * kk]);
        pfa_dft<9, +1>(v);
#pragma unroll
        for (int jj = 0; jj < 9; jj++) Sc[c1 * PFD_SP + i + 9 * jj] = v[jj];
    }
    __syncthreads();
    // inverse length-8 DFTs; y_{g^q} = x_0 + convolution
    for (int i = t; i < RP * 7 * 9; i += NT) {
        double2 *X = smem + (i / 63) * PFD_ROW, *Sc = X + PFD_XS, *X0 = Sc + 7 * PFD_SP;
        const int u = i % 63, c1 = u % 7, j = u / 7;
        double2 v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = Sc[c1 * PFD_SP + k + 9 * j];
        Dft<8, +1>::run(v);
        const double2 x0 = X0[c1];
#pragma unroll
        for (int k = 0; k < 8; k++) X[c1 + PFD_P * c_rader73_dst[k + 8 * j]] = cadd(x0, v[k]);
    }
    __syncthreads();
    alpha_rows_out<MODE, PFD_N, RP>(e, cta, [&](int r, int k) -> double2 {
        return smem[r * PFD_ROW + k % 7 + PFD_P * (k % 73)];
    });
}

// ---------------------------------------------------------------------------
// Prime-factor alpha stages at bl = 512: n = 1023 = 3 * 11 * 31
//
// Good-Thomas as at bl = 2048 (layout L = d1 + 3 d2 + 33 d3, input digits
// (n u_i) mod R_i with u_i = (1023/R_i)^-1 mod R_i = 2, 9, 16, output k at
// digits k mod R_i), DFTs of length 3 and 11 in place, then the length-31 DFTs
// written straight to their output positions (pfa_dft_out keeps their
// registers to about 31 complex values).  About 45 FP64 operations per point
// against ~220 for the 2048-point Bluestein convolution.
// ---------------------------------------------------------------------------
constexpr int PFC_N = 1023;

__device__ __forceinline__ int pfc_in_pos(int n) { return (n * 2) % 3 + 3 * ((n * 9) % 11) + 33 * ((n * 16) % 31); }
__device__ __forceinline__ int pfc_out_pos(int k) { return k % 3 + 3 * (k % 11) + 33 * (k % 31); }

// A row pair per CTA of 96 threads: 93 length-11 DFTs are one pass, and so are
// the 33 length-31 DFTs with a column's real and imaginary parts in two lanes
// (66 lanes; one thread per column took 168 registers and left 95 of 128 threads
// waiting).
// The launch follows the other scales' alpha launch of its stage (where they share
// a group).  Run beside it, forked to a second stream, it took the same time: B =
// 512, N = 4 analysis 196 and 194 us, synthesis 222 and 222, B = 1024 810 and 813, 862
// and 861.
constexpr int PFC_THREADS = 96;

template <int MODE>
__global__ void __launch_bounds__(PFC_THREADS, 6) pfa1023_kernel(const __grid_constant__ StageArgs a)
{
    constexpr int SIGN = MODE == CZT_ANA_ALPHA ? +1 : -1, NT = PFC_THREADS;
    extern __shared__ __align__(16) double2 smem[];
    int cta;
    const StageEnt &e = stage_entry(a, cta);
    pdl_wait();
    pdl_start();
    const int t = threadIdx.x;
    alpha_rows_in<MODE, PFC_N, 1, NT>(e, cta, [&](int, int m) -> double2 & { return smem[pfc_in_pos(m)]; });
    __syncthreads();
    pfs_stage<PFC_N, 3, 1, 1, SIGN, NT>(smem, t);
    __syncthreads();
    pfs_stage<PFC_N, 11, 3, 1, SIGN, NT>(smem, t);
    __syncthreads();
    // length-31 DFTs along d3 (stride 33), in registers, back to the same positions
    {
        double *sd = reinterpret_cast<double *>(smem) + (t & 1);
        const bool live = t < 66;
        const int d = live ? t >> 1 : 0;
        double x[31];
#pragma unroll
        for (int r = 0; r < 31; r++) x[r] = sd[2 * (d + 33 * r)];
        pfa_dft_part<31, SIGN>(x, sd, d, 33, live);
    }
    __syncthreads();
    alpha_rows_out<MODE, PFC_N, 1, NT>(e, cta, [&](int, int k) -> double2 { return smem[pfc_out_pos(k)]; });
}

// ---------------------------------------------------------------------------
// Bluestein alpha stages of up to 2048 points (bl <= 512): one row pair per
// RowFft row
// ---------------------------------------------------------------------------
template <int MODE, int LG, int VMAX>
__device__ __forceinline__ void czt_alpha(const StageArgs &a, const StageEnt &e, int cta, double2 *smem)
{
    using F = RowFft<LG, VMAX>;
    constexpr int M = F::M, V = F::V, TPR = F::TPR;
    const int t = threadIdx.x % TPR, r = threadIdx.x / TPR, bl = e.bl, n = 2 * bl - 1;
    const int row = cta * F::ROWS + r, per = e.rows_map;
    const bool valid = row < e.rows;
    const int k = valid ? row / per : 0, gr = valid ? row - k * per : 0, g = gr / bl, rr = gr - g * bl;
    double2 *buf = smem + r * F::PITCH;
    double2 v[V];
    if (MODE == CZT_ANA_ALPHA) {  // Hermitian completion in m
        const double2 *p = static_cast<const double2 *>(e.in) + k * e.in_map + (size_t)g * bl * (2 * bl) + 2 * rr;
#pragma unroll
        for (int i = 0; i < V; i++) {
            const int m = t + i * TPR;
            v[i] = make_double2(0.0, 0.0);
            if (m >= n) continue;
            const bool lo = m < bl;
            double2 x1, x2;
            ld_pair(p + (size_t)(lo ? m : n - m) * (2 * bl), x1, x2);
            if (!lo) { x1 = cconj(x1); x2 = cconj(x2); }
            if (m == 0) { x1.y = 0.0; x2.y = 0.0; }
            v[i] = cmul(make_double2(x1.x - x2.y, x1.y + x2.x), __ldg(e.pre + m));
        }
    } else {
        const double *p = static_cast<const double *>(e.in) + k * e.in_map + (size_t)(2 * n) * gr;
#pragma unroll
        for (int i = 0; i < V; i++) {
            const int m = t + i * TPR;
            v[i] = m < n ? cmul(make_double2(__ldg(p + m), __ldg(p + n + m)), __ldg(e.pre + m)) : make_double2(0.0, 0.0);
        }
    }
    F::template run<-1>(v, buf, t, a.tw);
#pragma unroll
    for (int i = 0; i < V; i++) v[i] = cmul(v[i], hf_at<MODE>(e.Hf, t + i * TPR, M));
    F::template run<+1>(v, buf, t, a.tw);
    if (MODE == CZT_ANA_ALPHA) {
        if (!valid) return;
        double *p = static_cast<double *>(e.out) + k * e.out_map + (size_t)(2 * n) * gr;
#pragma unroll
        for (int i = 0; i < V; i++) {
            const int b = t + i * TPR;
            if (b >= n) continue;
            const double2 y = cmul(v[i], __ldg(e.post + b));
            p[b] = y.x;
            p[n + b] = y.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < V; i++) buf[F::pad(t + i * TPR)] = v[i];
        F::sync();
        if (!valid) return;
        const double hh = 0.5 * e.scale;
        double2 *p = static_cast<double2 *>(e.out) + k * e.out_map + (size_t)g * bl * (2 * bl) + 2 * rr;
        for (int m = t; m < bl; m += TPR) {
            const int mc = m == 0 ? 0 : n - m;
            const double2 Z = cmul(buf[F::pad(m)], __ldg(e.post + m));
            const double2 Zc = cconj(cmul(buf[F::pad(mc)], __ldg(e.post + mc)));
            const double2 sm = cadd(Z, Zc), d = csub(Z, Zc);
            st_pair(p + (size_t)m * (2 * bl), make_double2(sm.x * hh, sm.y * hh), make_double2(d.y * hh, -d.x * hh));
        }
    }
}

// Alpha stages of the scales of a group, one launch (bl <= 512).  Two kernels:
// without the 1024- and 2048-point transforms 80 registers are enough and six
// CTAs fit on an SM.  With the length-1023 rows in their own kernel the B = 512,
// N = 4 stage went from 109 to 83 us per analysis.
template <int MODE, bool BIG>
__global__ void __launch_bounds__(ST_THREADS, BIG ? 4 : 6) alpha_kernel(const __grid_constant__ StageArgs a)
{
    extern __shared__ __align__(16) double2 smem[];
    int cta;
    const StageEnt &e = stage_entry(a, cta);
    pdl_wait();
    pdl_start();
    if (e.kind == STAGE_PFA) {
        switch (e.bl) {
        case 2: pfs_rows_run<3, 1, 1, MODE>(e, cta, smem); break;
        case 4: pfs_rows_run<7, 1, 1, MODE>(e, cta, smem); break;
        case 8: pfs_rows_run<3, 5, 1, MODE>(e, cta, smem); break;
        case 32: pfs_rows_run<7, 9, 1, MODE>(e, cta, smem); break;
        case 128: pfs_rows_run<3, 5, 17, MODE>(e, cta, smem); break;
        case 256: pfa511_rows<MODE>(e, cta, smem); break;
        }
        return;
    }
    switch (e.lg) {
    case 4: czt_alpha<MODE, 4, 8>(a, e, cta, smem); break;
    case 5: czt_alpha<MODE, 5, 8>(a, e, cta, smem); break;
    case 6: czt_alpha<MODE, 6, 8>(a, e, cta, smem); break;
    case 7: czt_alpha<MODE, 7, 8>(a, e, cta, smem); break;
    case 8: czt_alpha<MODE, 8, 8>(a, e, cta, smem); break;
    case 9: czt_alpha<MODE, 9, 8>(a, e, cta, smem); break;
    case 10:
        if constexpr (BIG) czt_alpha<MODE, 10, 16>(a, e, cta, smem);
        break;
    case 11:
        if constexpr (BIG) czt_alpha<MODE, 11, 16>(a, e, cta, smem);
        break;
    }
}

// scoeff(0:bs-1,0:bs-1) = flm(0:bs-1,0:bs-1), s2dw_core_mod.f90:773
__global__ void scoeff_copy_kernel(double2 *sc, const double2 *flm, int B, int bs)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (i < bs * bs) sc[(size_t)k * bs * bs + i] = flm[(size_t)k * B * B + (i % bs) + (size_t)B * (i / bs)];
}

__global__ void combine_kernel(const __grid_constant__ CombineArgs a)
{
    const int B = a.B, k = blockIdx.y;
    const double2 *parts = a.parts + k * a.pstride, *scoeff = a.scoeff + (size_t)k * a.bs * a.bs;
    double2 *flm = a.flm + (size_t)k * B * B;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)B * B;
         i += (long long)gridDim.x * blockDim.x) {
        const int l = (int)(i % B), m = (int)(i / B);
        double2 f = make_double2(0.0, 0.0);
        if (m <= l) {
            for (int j = 0; j <= a.J; j++)
                if (l > a.blo[j] && l < a.bl[j]) f = cadd(f, parts[a.off[j] + (size_t)(l - a.blo[j] - 1) * a.bl[j] + m]);
        }
        if (l < a.bs && m < a.bs) f = cadd(f, cscale(scoeff[l + (size_t)a.bs * m], a.Phi2[l]));
        flm[i] = f;
    }
}

// ===========================================================================
// Launchers
// ===========================================================================
int launch_gprep(const GprepArgs &a, cudaStream_t s)
{
    const long long total = (long long)(a.bl - a.blo - 1) * a.NP * a.stride;
    if (total <= 0) return S2DWC_OK;
    long long blocks = (total + 255) / 256;
    if (blocks > 148 * 32) blocks = 148 * 32;
    gprep_kernel<<<(int)blocks, 256, 0, s>>>(a);
    S2DW_CUDA_TRY(cudaGetLastError());
    return S2DWC_OK;
}

int launch_fprep(double2 *F, double2 *scoeff, const double2 *flm, const double *Om, int B, int Bp, int bs,
                 cudaStream_t s)
{
    dim3 grid((B + 31) / 32, (Bp + 31) / 32), block(32, 8);
    fprep_kernel<<<grid, block, 0, s>>>(F, scoeff, flm, Om, B, Bp, bs);
    S2DW_CUDA_TRY(cudaGetLastError());
    return S2DWC_OK;
}

template <int MODE, int LGM>
static int launch_large_t(const CztArgs &a, cudaStream_t s)
{
    constexpr int M = 1 << LGM;
    const size_t smem = sizeof(double2) * ((size_t)padix(M) + 1 + M / 64 + 64 + S2DW_NMAX);  // + phases ph[g], g < N
    static bool attr[64] = {false};
    int dev = 0;
    S2DW_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 64 && !attr[dev]) {
        S2DW_CUDA_TRY(cudaFuncSetAttribute(fft_large_kernel<MODE, LGM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
        attr[dev] = true;
    }
    // rows are (g or q) x (m or b pair); every mode has bl rows per g
    const int ng = a.rows / a.bl;
    constexpr bool synb = (MODE == CZT_SYN_BETA || MODE == FFT_SYN_BETA);
    const dim3 grid = synb ? dim3(ng, a.bl) : dim3(a.bl, ng);
    fft_large_kernel<MODE, LGM><<<grid, M / 16, smem, s>>>(a);
    S2DW_CUDA_TRY(cudaGetLastError());
    return S2DWC_OK;
}

template <int LGM>
static int launch_large(const CztArgs &a, cudaStream_t s)
{
    switch (a.mode) {
    case FFT_ANA_BETA: return launch_large_t<FFT_ANA_BETA, LGM>(a, s);
    case FFT_SYN_BETA: return launch_large_t<FFT_SYN_BETA, LGM>(a, s);
    default: break;
    }
    if constexpr (LGM > 11) {  // chirp-z transforms of 2048 points: the stage kernels
        switch (a.mode) {
        case CZT_ANA_BETA: return launch_large_t<CZT_ANA_BETA, LGM>(a, s);
        case CZT_ANA_ALPHA: return launch_large_t<CZT_ANA_ALPHA, LGM>(a, s);
        case CZT_SYN_ALPHA: return launch_large_t<CZT_SYN_ALPHA, LGM>(a, s);
        case CZT_SYN_BETA: return launch_large_t<CZT_SYN_BETA, LGM>(a, s);
        default: break;
        }
    }
    return set_error(S2DWC_ERROR_ARG_INVALID, "transform mode %d of %d points", a.mode, 1 << LGM);
}

template <int MODE>
static int launch_pfa(const CztArgs &a, cudaStream_t s)
{
    const size_t smem = sizeof(double2) * PFA_N;
    static bool attr[64] = {false};
    int dev = 0;
    S2DW_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 64 && !attr[dev]) {
        S2DW_CUDA_TRY(cudaFuncSetAttribute(pfa_alpha_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
        attr[dev] = true;
    }
    const dim3 grid(a.bl, a.rows / a.bl);  // (b pair, g)
    pfa_alpha_kernel<MODE><<<grid, PFA_THREADS, smem, s>>>(a);
    S2DW_CUDA_TRY(cudaGetLastError());
    return S2DWC_OK;
}

template <int MODE>
static int launch_pfa2047(const CztArgs &a, cudaStream_t s)
{
    const size_t smem = sizeof(double2) * (PFB_XS + 23 * PFB_SP + 23);
    static bool attr[64] = {false};
    int dev = 0;
    S2DW_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 64 && !attr[dev]) {
        S2DW_CUDA_TRY(cudaFuncSetAttribute(pfa2047_alpha_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
        attr[dev] = true;
    }
    const dim3 grid(a.bl, a.rows / a.bl);  // (b pair, g)
    pfa2047_alpha_kernel<MODE><<<grid, PFB_THREADS, smem, s>>>(a);
    S2DW_CUDA_TRY(cudaGetLastError());
    return S2DWC_OK;
}

static bool g_rader_ready[64] = {false};
static __device__ double2 g_tw[ST_TW];

int pfa_prepare()
{
    int dev = 0;
    S2DW_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_error(S2DWC_ERROR_ARG_INVALID, "device index %d", dev);
    static std::mutex mu;
    std::lock_guard<std::mutex> g(mu);
    if (g_rader_ready[dev]) return S2DWC_OK;
    static const std::vector<double2> tw = [] {
        std::vector<double2> v(ST_TW);
        for (int k = 0; k < ST_TW; k++) {
            const long double x = -2.0L * 3.141592653589793238462643383279502884L * (long double)k / (long double)ST_TW;
            v[k] = make_double2((double)cosl(x), (double)sinl(x));
        }
        return v;
    }();
    S2DW_CUDA_TRY(cudaMemcpyToSymbol(g_tw, tw.data(), sizeof(double2) * ST_TW));
    rader_init_kernel<<<2, 96>>>();
    S2DW_CUDA_TRY(cudaGetLastError());
    rader73_init_kernel<<<2, 96>>>();
    S2DW_CUDA_TRY(cudaGetLastError());
    S2DW_CUDA_TRY(cudaStreamSynchronize(0));
    g_rader_ready[dev] = true;
    return S2DWC_OK;
}

int stage_twiddles(const double2 **tw)
{
    void *p = nullptr;
    S2DW_CUDA_TRY(cudaGetSymbolAddress(&p, g_tw));
    *tw = static_cast<const double2 *>(p);
    return S2DWC_OK;
}

static bool g_alpha_prefetch = true;  // contiguous-input stages: persistent kernel with prefetched input

// Persistent launch of the prefetching stages: as many CTAs as fit on the
// device at once, each looping over rows.
template <int MODE, int LGM>
static int launch_pf(const CztArgs &a, cudaStream_t s)
{
    constexpr int M = 1 << LGM, THREADS = M / 16;
    const int chunks = pf_chunks<MODE>(a.bl);
    if (chunks > M) return set_error(S2DWC_ERROR_SIZE_INVALID, "prefetch stage: bl=%d does not fit M=%d", a.bl, M);
    const size_t smem = sizeof(double2) * ((size_t)padix(M) + 1 + M / 64 + 64 + (size_t)chunks);
    static int resident[64] = {0};
    static size_t smem_set[64] = {0};
    int dev = 0;
    S2DW_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 64) return set_error(S2DWC_ERROR_ARG_INVALID, "device index %d", dev);
    if (smem_set[dev] < smem) {
        S2DW_CUDA_TRY(cudaFuncSetAttribute(fft_pf_kernel<MODE, LGM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
        int per_sm = 0, sms = 0;
        S2DW_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fft_pf_kernel<MODE, LGM>, THREADS, smem));
        S2DW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        resident[dev] = std::max(1, per_sm) * sms;
        smem_set[dev] = smem;
    }
    const int grid = std::min(a.rows, resident[dev]);
    if (grid <= 0) return S2DWC_OK;
    fft_pf_kernel<MODE, LGM><<<grid, THREADS, smem, s>>>(a);
    S2DW_CUDA_TRY(cudaGetLastError());
    return S2DWC_OK;
}

void set_alpha_prefetch(bool on) { g_alpha_prefetch = on; }

int launch_czt(const CztArgs &a, cudaStream_t s)
{
    if (a.rows % a.bl) return set_error(S2DWC_ERROR_ARG_INVALID, "transform of %d rows at bl=%d", a.rows, a.bl);
    if (a.pfa && a.bl == 2048)
        return a.mode == CZT_ANA_ALPHA ? launch_pfa<CZT_ANA_ALPHA>(a, s) : launch_pfa<CZT_SYN_ALPHA>(a, s);
    if (a.pfa && a.bl == 1024) {
        int dev = 0;
        S2DW_CUDA_TRY(cudaGetDevice(&dev));
        if (dev < 0 || dev >= 64 || !g_rader_ready[dev])
            return set_error(S2DWC_ERROR_NOT_INIT, "the length-2047 alpha tables are not built on device %d", dev);
        return a.mode == CZT_ANA_ALPHA ? launch_pfa2047<CZT_ANA_ALPHA>(a, s)
                                       : launch_pfa2047<CZT_SYN_ALPHA>(a, s);
    }
    // Stages whose input row is contiguous: persistent kernel with the next
    // row prefetched (synthesis alpha 4% faster than one row per CTA at
    // bl = 1024).  The analysis alpha stage stays one row per CTA: its
    // row-strided input gathered by cp.async gave no gain over 256-bit loads
    // (the chirp-table loads from L2, not the input, dominate its remaining
    // memory stalls).
    const int M = a.czt.M;
    if (g_alpha_prefetch && a.mode == CZT_SYN_ALPHA && ((uintptr_t)a.in_r & 15) == 0) {
        if (M == 4096) return launch_pf<CZT_SYN_ALPHA, 12>(a, s);
        if (M == 8192) return launch_pf<CZT_SYN_ALPHA, 13>(a, s);
    }
    if (g_alpha_prefetch && a.mode == FFT_ANA_BETA && ((uintptr_t)a.in_c & 15) == 0) {
        if (M == 2048) return launch_pf<FFT_ANA_BETA, 11>(a, s);
        if (M == 4096) return launch_pf<FFT_ANA_BETA, 12>(a, s);
    }
    if (M == 2048) return launch_large<11>(a, s);
    if (M == 4096) return launch_large<12>(a, s);
    if (M == 8192) return launch_large<13>(a, s);
    return set_error(S2DWC_ERROR_SIZE_INVALID, "transform size %d unsupported", M);
}

bool pfa_size(int mode, int bl)
{
    return (mode == CZT_ANA_ALPHA || mode == CZT_SYN_ALPHA) && bl >= 2 && bl <= 2048 && (bl & (bl - 1)) == 0 && bl != 64 &&
           bl != 16;
}

bool stage_plan(int mode, int bl, int M, bool pfa, int rows, StageEnt *e, int *ncta)
{
    const bool alpha = mode == CZT_ANA_ALPHA || mode == CZT_SYN_ALPHA;
    int per = 0;  // rows per CTA
    if (pfa && pfa_size(mode, bl)) {
        if (bl > 512) return false;
        e->kind = STAGE_PFA;
        e->lg = 0;
        per = bl == 512 ? 1 : bl == 256 ? PFD_RP : pfs_rows(2 * bl - 1);
    } else {
        // the 2048-point beta transforms of bl = 1024 keep their own kernels
        if (M < 16 || M > 2048 || (M & (M - 1)) || bl > 512) return false;
        int lg = 4;
        while ((1 << lg) < M) lg++;
        e->kind = (short)mode;
        e->lg = (short)lg;
        per = ST_THREADS * row_fft_v(lg, alpha && lg < 10 ? 8 : 16) / M;
    }
    *ncta = (rows + per - 1) / per;
    return true;
}

bool stage_alone(const StageEnt &e) { return e.kind == STAGE_PFA && e.bl == 512; }

int launch_stage(Stage st, const StageArgs &a, bool dep, cudaStream_t s)
{
    if (st == STAGE_ANA_BETA || st == STAGE_SYN_BETA) return launch_stage_beta(st, a, dep, s);
    if (a.ncta <= 0) return S2DWC_OK;
    if (stage_alone(a.e[0])) {
        auto *k = st == STAGE_ANA_ALPHA ? pfa1023_kernel<CZT_ANA_ALPHA> : pfa1023_kernel<CZT_SYN_ALPHA>;
        S2DW_CUDA_TRY(launch_dep(k, a.ncta, PFC_THREADS, sizeof(double2) * PFC_N, s, dep, a));
        return S2DWC_OK;
    }
    size_t smem = 0;  // of the group's largest row set
    bool big = false;
    for (int i = 0; i < a.n; i++) {
        const StageEnt &e = a.e[i];
        size_t n;
        if (e.kind != STAGE_PFA) {
            n = ST_THREADS * row_fft_v(e.lg, e.lg < 10 ? 8 : 16) * 5 / 4 + 32;
        } else if (e.bl == 256) {
            int dev = 0;
            S2DW_CUDA_TRY(cudaGetDevice(&dev));
            if (dev < 0 || dev >= 64 || !g_rader_ready[dev])
                return set_error(S2DWC_ERROR_NOT_INIT, "the length-511 alpha tables are not built on device %d", dev);
            n = PFD_RP * PFD_ROW;
        } else {
            n = (size_t)pfs_rows(2 * e.bl - 1) * (2 * e.bl - 1);
        }
        smem = std::max(smem, n * sizeof(double2));
        big = big || e.lg >= 10;
    }
    auto *k = st == STAGE_ANA_ALPHA ? (big ? alpha_kernel<CZT_ANA_ALPHA, true> : alpha_kernel<CZT_ANA_ALPHA, false>)
                                    : (big ? alpha_kernel<CZT_SYN_ALPHA, true> : alpha_kernel<CZT_SYN_ALPHA, false>);
    S2DW_CUDA_TRY(launch_dep(k, a.ncta, ST_THREADS, smem, s, dep, a));
    return S2DWC_OK;
}

int launch_combine(const CombineArgs &a, cudaStream_t s)
{
    long long n = (long long)a.B * a.B, blocks = (n + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    combine_kernel<<<dim3((int)blocks, a.maps), 256, 0, s>>>(a);
    S2DW_CUDA_TRY(cudaGetLastError());
    return S2DWC_OK;
}

int launch_scoeff_copy(double2 *scoeff, const double2 *flm, int B, int bs, int maps, cudaStream_t s)
{
    const int n = bs * bs;
    if (n <= 0 || maps <= 0) return S2DWC_OK;
    scoeff_copy_kernel<<<dim3((n + 255) / 256, maps), 256, 0, s>>>(scoeff, flm, B, bs);
    S2DW_CUDA_TRY(cudaGetLastError());
    return S2DWC_OK;
}

}  // namespace s2dw
