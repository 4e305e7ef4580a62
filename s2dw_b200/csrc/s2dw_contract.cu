// The contractions over l (analysis) and m' (synthesis) with d^l_{m'm}(pi/2)
// generated in registers, all scales of a transform in one walk.
//
// A degree l lies in the range of at most two scales (bl_lo < l < bl_hi; the
// ranges of scales j and j + 2 are disjoint), whose indices differ by one.  So
// one walk of the recurrence serves every scale: two accumulator sets, the
// slots j & 1, hold the two scales of the current l, and the recurrence, the
// products with f(l, m) and the table reads that do not depend on the scale
// are shared.  Per (l, m', m) that is 4 + 4 NP FP64 instructions for both
// scales instead of 2 (4 + 2 NP) in a walk per scale.
//
// Both kernels are bound by the FP64 pipe (64 lanes per SM and clock) as long
// as the shared-memory reads stay below it.  A warp's 32 lanes are 16 values
// of the table index by 2 values of the broadcast index: an 8-byte read of 16
// distinct doubles is one shared-memory cycle where 32 distinct ones are two
// (measured: 1.00 and 2.00 cycles per warp read on B200; a 16-byte read that
// all lanes of a half-warp share costs two in either layout).
//
// Against a launch per scale (us per pair, B200): B = 1024, N = 4 analysis 787
// -> 430 (26.7 TFLOP/s algorithmic, FP64 pipe 60 %), synthesis 869 -> 465
// (12.3 TFLOP/s, 58 %); B = 2048, N = 8 7110 -> 5990 and 7720 -> 5600.  What is
// left: two CTAs of 250 registers per SM (eight warps) cover the dependent FP64
// chain only in part, and an FP64 instruction with three distinct operands
// issues every 0.565 cycles per SM instead of 0.5.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <type_traits>
#include <vector>

#include "s2dw_fft.cuh"
#include "s2dw_internal.h"

namespace s2dw {
namespace {

// z * i^k
__device__ __forceinline__ double2 cipow(double2 z, int k)
{
    switch (k & 3) {
    case 0: return z;
    case 1: return make_double2(-z.y, z.x);
    case 2: return make_double2(-z.x, -z.y);
    default: return make_double2(z.y, -z.x);
    }
}
__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ int warp_max_i(int v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ void cp16(void *smem, const void *gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

constexpr int WARPS = 4;
constexpr int THREADS = WARPS * 32;

// ===========================================================================
// Analysis: walk over l, fused with the gamma DFT
//
// CTA tile: 16 m' (half a warp's lanes) by MT = 8 S values of m (S per half
// warp, 4 warps).  A thread walks l for its S pairs (m', m) up to the largest
// band limit; per step it reads a(l, m') and G(l, slot, q, m') by lane and
// a(l, m), F(l, m) by broadcast, staged 16 values of l at a time in three
// buffers (one barrier per chunk).  Where a scale ends (l = bl_j) its
// accumulators go through the gamma DFT to T_j and its slot restarts at zero
// for scale j - 2.  With S = 4, NP = 2 a step costs 24 FP64-pipe cycles per
// warp and SM against 17 of shared memory.
//
// S: as many pairs per thread as the accumulators allow in registers (16 NP
// each), fewer where the tiles would not fill the GPU
// (lwalk_pairs).  NS = 1: one scale only (a.only), one slot, tiles in plain order.
// ===========================================================================
constexpr int LW_CH = 16;
constexpr int LW_ST = 3;  // staging buffers

template <int NP, int S, int NS>
struct LwalkSmem {
    static constexpr int MT = 2 * WARPS * S;
    static constexpr int F_OFF = 0;                         // double2 [CH][MT]
    static constexpr int AP_OFF = F_OFF + 2 * LW_CH * MT;   // [CH][16]
    static constexpr int G_OFF = AP_OFF + LW_CH * 16;       // [CH][NS*NP][16]
    static constexpr int AM_OFF = G_OFF + LW_CH * NS * NP * 16;  // [CH][MT]
    static constexpr int BUF = AM_OFF + LW_CH * MT;
    static constexpr size_t BYTES = (size_t)LW_ST * BUF * sizeof(double);
};

template <int NP, int S, int NS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) lwalk_kernel(const __grid_constant__ LwalkArgs a)
{
    using L = LwalkSmem<NP, S, NS>;
    constexpr int MT = L::MT, NR = NS * NP;
    extern __shared__ __align__(16) double lsm[];
    pdl_start();

    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, lp = lane & 15;
    const int B = a.B, Bp = a.Bp, N = a.N;
    int2 tile;
    int jlast = 0, jfirst = a.J;  // the scales of this CTA: jlast <= j <= jfirst
    if (NS == 1) {
        jlast = jfirst = a.only;
        const int tm = (a.bl[jlast] + MT - 1) / MT;
        tile = make_int2((int)blockIdx.x / tm, (int)blockIdx.x % tm);
    } else {
        tile = a.tiles[blockIdx.x];
        if (S == 1) {  // see lwalk_split
            if (tile.x >> 16) jlast = a.jsplit;
            else if (tile.y >> 16) jfirst = a.jsplit - 1;
            tile.x &= 0xffff;
            tile.y &= 0xffff;
        }
    }
    const int bend = a.bl[jlast];  // the largest band limit of the walk
    const int p0 = tile.x * 16, m0 = tile.y * MT;
    const int mp = p0 + lp, mi = (w * 2 + (lane >> 4)) * S, mb = m0 + mi;

    // the scale that ends next: the last one that holds pairs of this tile
    int jd = jlast;
    if (NS == 2)
        while (jd < jfirst && a.bl[jd + 1] > max(p0, m0)) jd++;

    const int lstart = max(p0, m0) & ~(LW_CH - 1);
    const int rampEnd = min(max(p0 + 15, m0 + MT - 1), bend - 1);
    const int nchunks = (bend - lstart + LW_CH - 1) / LW_CH;

    // Staging in a fixed pattern of 16-byte pieces per thread.  Rows of l past
    // the last one repeat it; columns are not bounded: a row's values past m = B - 1
    // are zeros up to Bp and, with tiles of more than 32 m, the next row's or the
    // slack behind the last.  Both are read but belong to pairs that stay at zero
    // and are not stored, or to steps that do not run.
    auto lrow = [&](int l) { return (size_t)min(l, B - 1) * Bp; };
    auto stage_tables = [&](int c) {
        const int lc = lstart + c * LW_CH;
        double *b = lsm + (c % LW_ST) * L::BUF;
        {
            const int li = tid >> 3, pc = 2 * (tid & 7);
            cp16(b + L::AP_OFF + li * 16 + pc, a.Acoef + lrow(lc + li) + p0 + pc);
            // G rows (l, slot, q), packed: gpack_len(l) doubles each, the
            // rows of the 16 l of a chunk consecutive
            const int len = gpack_len(lc);
            const double *g = a.G + gpack_row(lc, 2 * NP) + p0 + pc;
            if (NS == 2) {
                g += li * len;
#pragma unroll
                for (int i = 0; i < NR; i++) {
                    cp16(b + L::G_OFF + (li + 16 * i) * 16 + pc, g);
                    g += 16 * len;
                }
            } else {
#pragma unroll
                for (int i = 0; i < NR; i++) {
                    const int r = li + 16 * i, src = (r / NP) * 2 * NP + (a.only & 1) * NP + r % NP;
                    cp16(b + L::G_OFF + r * 16 + pc, g + src * len);
                }
            }
        }
        constexpr int AP = MT / 2;  // pieces of a row a(l, m)
#pragma unroll
        for (int i = 0; i < (LW_CH * AP + THREADS - 1) / THREADS; i++) {
            const int f = tid + THREADS * i, li = f / AP, pc = 2 * (f % AP);
            if (LW_CH * AP % THREADS == 0 || f < LW_CH * AP)
                cp16(b + L::AM_OFF + li * MT + pc, a.Acoef + lrow(lc + li) + m0 + pc);
        }
    };
    auto stage_f = [&](int c) {
        const int lc = lstart + c * LW_CH;
        double *b = lsm + (c % LW_ST) * L::BUF;
#pragma unroll
        for (int i = 0; i < LW_CH * MT / THREADS; i++) {
            const int f = tid + THREADS * i, li = f / MT, pc = f % MT;
            cp16(b + L::F_OFF + 2 * (li * MT + pc), a.F + lrow(lc + li) + m0 + pc);
        }
    };
    // the first chunks' tables are on their way while the start values are
    // read (and the kernel that writes F ends)
#pragma unroll
    for (int c = 0; c < LW_ST - 1; c++)
        if (c < nchunks) stage_tables(c);

    // ---- start values of the pairs (m', m = mb + s), all in the domain scaled by 2^Kw
    double st[S];
    int maxe = INT_MIN;
#pragma unroll
    for (int s = 0; s < S; s++)
        if (mp < bend && mb + s < bend) maxe = max(maxe, (int)a.Ste[(size_t)max(mp, mb + s) * B + min(mp, mb + s)]);
    maxe = warp_max_i(maxe);
    int Kw = (maxe != INT_MIN && maxe < S2DW_SCALE_EXP) ? -maxe : 0;
#pragma unroll
    for (int s = 0; s < S; s++) {
        const int m = mb + s;
        st[s] = 0.0;
        if (mp < bend && m < bend) {
            const size_t o = (size_t)max(mp, m) * B + min(mp, m);
            const double v = ldexp(a.Stm[o], (int)a.Ste[o] + Kw);
            st[s] = (mp >= m && ((mp - m) & 1)) ? -v : v;
        }
    }
    pdl_wait();
#pragma unroll
    for (int c = 0; c < LW_ST - 1; c++) {
        if (c < nchunks) stage_f(c);
        cp_commit();
    }
    double x[2][S];
    double2 acc[NS][2][S][NP];
#pragma unroll
    for (int s = 0; s < S; s++) {
        x[0][s] = x[1][s] = 0.0;
#pragma unroll
        for (int q = 0; q < NP; q++)
#pragma unroll
            for (int k = 0; k < NS; k++) acc[k][0][s][q] = acc[k][1][s][q] = make_double2(0.0, 0.0);
    }

    // one recurrence step at chunk row li (l parity PAR); act[k]: slot k accumulates
    auto step = [&](const double *b, const int li, auto par_tag, const bool inj, const int l, const bool act0,
                    const bool act1) {
        constexpr int PAR = decltype(par_tag)::value;
        const double ap = b[L::AP_OFF + li * 16 + lp];
        double g[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) g[r] = b[L::G_OFF + (li * NR + r) * 16 + lp];
        const double2 *Fr = reinterpret_cast<const double2 *>(b + L::F_OFF) + li * MT + mi;
        const double *Amr = b + L::AM_OFF + li * MT + mi;
        double xr[S], xi[S], p[S];
#pragma unroll
        for (int s = 0; s < S; s++) {
            if (inj && l == max(mp, mb + s)) x[PAR][s] = st[s];
            const double2 F = Fr[s];
            xr[s] = x[PAR][s] * F.x;
            xi[s] = x[PAR][s] * F.y;
            p[s] = Amr[s] * ap;
        }
#pragma unroll
        for (int s = 0; s < S; s++) x[PAR ^ 1][s] = fma(-p[s], x[PAR][s], -x[PAR ^ 1][s]);
#pragma unroll
        for (int k = 0; k < NS; k++) {
            if (k == 0 ? !act0 : !act1) continue;
#pragma unroll
            for (int q = 0; q < NP; q++)
#pragma unroll
                for (int s = 0; s < S; s++) {
                    acc[k][PAR][s][q].x = fma(xr[s], g[k * NP + q], acc[k][PAR][s][q].x);
                    acc[k][PAR][s][q].y = fma(xi[s], g[k * NP + q], acc[k][PAR][s][q].y);
                }
        }
    };
    using P0 = std::integral_constant<int, 0>;
    using P1 = std::integral_constant<int, 1>;

    // Scale j ends: T(m, m', +-n) from the even- and odd-l sums of its slot,
    // then the gamma DFT, and the slot restarts at zero.
    // T(+n) = i^{n-m} conj(eta) (E+O), T(-n) = i^{-n-m} (-1)^{m'+n} eta (E-O),
    // T(0) = i^{-m} (E+O); eta = 1 (N odd) or i (N even); F carries the i^{-m}.
    // One copy of the code, for slot 0, between exchanges of the slots: small
    // transforms meet most of this kernel's code once, cold.
    auto flush = [&](const int j) {
        const bool odd = NS == 2 && (j & 1);
        auto exchange = [&]() {
#pragma unroll
            for (int s = 0; s < S; s++)
#pragma unroll
                for (int q = 0; q < NP; q++)
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        const double2 u = acc[0][p][s][q], v = acc[NS - 1][p][s][q];
                        acc[0][p][s][q] = odd ? v : u;
                        acc[NS - 1][p][s][q] = odd ? u : v;
                    }
        };
        if (NS == 2) exchange();
        const int bl = a.bl[j];
        const double sc = ldexp(1.0, -Kw);
        const int ev = (N % 2 == 0) ? 1 : 0, ai = a.acc_imag ? 1 : 0;
#pragma unroll
        for (int s = 0; s < S; s++) {
            const int m = mb + s;
            if (mp < bl && m < bl) {
                // gamma DFT of the pair (n, -n): sum cos(n g) + i dif sin(n g)
                double2 Ts[NP], Td[NP];
#pragma unroll
                for (int q = 0; q < NP; q++) {
                    const int n = a.nq[q];
                    const double2 E = cscale(acc[0][0][s][q], sc), O = cscale(acc[0][1][s][q], sc);
                    // acc_imag: the b part of S enters the +n terms times -i (i^-1)
                    // and the -n terms times +i
                    if (n == 0) {
                        Ts[q] = cipow(cadd(E, O), -ai);
                        Td[q] = make_double2(0.0, 0.0);
                    } else {
                        const double2 tp = cipow(cadd(E, O), n - ev - ai);
                        double2 tm = cipow(csub(E, O), -n + ev + ai);
                        if ((mp + n) & 1) tm = make_double2(-tm.x, -tm.y);
                        Ts[q] = cadd(tp, tm);
                        Td[q] = make_double2(tm.y - tp.y, tp.x - tm.x);  // i (tp - tm)
                    }
                }
                double2 *dst = a.Tg + a.off[j] + (size_t)m * bl + mp;
                const double2 *ph = a.ph + N - 1;
                for (int gg = 0; gg < N; gg++, dst += (size_t)bl * bl, ph += 2 * N - 1) {
                    double2 y = make_double2(0.0, 0.0);
#pragma unroll
                    for (int q = 0; q < NP; q++) {
                        const double2 w = __ldg(ph + a.nq[q]);
                        y.x = fma(Ts[q].x, w.x, fma(Td[q].x, w.y, y.x));
                        y.y = fma(Ts[q].y, w.x, fma(Td[q].y, w.y, y.y));
                    }
                    *dst = a.acc_imag ? cadd(*dst, y) : y;
                }
            }
#pragma unroll
            for (int q = 0; q < NP; q++) acc[0][0][s][q] = acc[0][1][s][q] = make_double2(0.0, 0.0);
        }
        if (NS == 2) exchange();
    };

    // in the scaled domain: keep the values in range (warp-uniform)
    auto rescale = [&]() {
        double mx = 0.0;
#pragma unroll
        for (int s = 0; s < S; s++) mx = fmax(mx, fmax(fabs(x[0][s]), fabs(x[1][s])));
        mx = warp_max(mx);
        if (mx > ldexp(1.0, S2DW_RENORM_EXP)) {
            const int R = min(S2DW_RENORM_EXP, Kw);
            const double f = ldexp(1.0, -R);
#pragma unroll
            for (int s = 0; s < S; s++) {
                x[0][s] *= f;
                x[1][s] *= f;
#pragma unroll
                for (int k = 0; k < NS; k++)
#pragma unroll
                    for (int q = 0; q < NP; q++) {
                        acc[k][0][s][q] = cscale(acc[k][0][s][q], f);
                        acc[k][1][s][q] = cscale(acc[k][1][s][q], f);
                    }
            }
            Kw -= R;
        }
    };
    auto full_chunk = [&](const double *b, int first) {
        // more unrolling hoists loads past the register cap
        constexpr int UNR = S == 1 || NP > 4 ? 2 : NP <= 2 ? 4 : 8;
#pragma unroll UNR
        for (int i = first; i < LW_CH; i += 2) {
            step(b, i, P0{}, false, 0, true, true);
            step(b, i + 1, P1{}, false, 0, true, true);
        }
    };

    // the next end, and the l up to which a slot has no scale in range yet
    int nextb, b0, b1, btop;
    auto next_scale = [&]() {
        nextb = INT_MAX;
        b0 = b1 = btop = INT_MAX;
        if (jd < jlast) return;
        nextb = a.bl[jd];
        const int bD = a.blo[jd], bM = NS == 2 && jd > jlast ? a.blo[jd - 1] : INT_MAX;
        const bool odd = NS == 2 && (jd & 1);
        b0 = odd ? bM : bD;
        b1 = odd ? bD : bM;
        btop = NS == 1 ? b0 : max(b0, b1);
    };
    next_scale();
    for (int c = 0; c <= nchunks; c++) {
        const int lc = lstart + c * LW_CH;
        const int nl = c < nchunks ? min(LW_CH, bend - lc) : 0;
        const double *b = lsm + (c % LW_ST) * L::BUF;
        if (c < nchunks) {
            cp_wait<LW_ST - 2>();
            __syncthreads();  // chunk c in shared memory, buffer of chunk c - 1 free
            if (c + LW_ST - 1 < nchunks) {
                stage_tables(c + LW_ST - 1);
                stage_f(c + LW_ST - 1);
            }
            cp_commit();
        }
        for (int li = 0;;) {
            // the scales that end here (the walk's last ones at l = bend)
            while (lc + li >= nextb) {
                flush(jd);
                jd--;
                next_scale();
            }
            if (li >= nl) break;
            // run to the next scale's end
            int le = min(nl, nextb - lc);
            const int lo = lc + li;
            if (li == 0 && le == LW_CH && lc > rampEnd && lc > btop) {
                // both slots accumulate at every step, no start value enters
                if (NP <= 2 && S > 1 && Kw == 0) {
                    full_chunk(b, 0);
                    li = le;
                    continue;
                }
                full_chunk(b, 0);
            } else if (S == 1 && li == 0 && le == LW_CH && lc > rampEnd && lc == btop) {
                // one slot's scale starts after the first row
                step(b, 0, P0{}, false, 0, lc > b0, lc > b1);
                step(b, 1, P1{}, false, 0, true, true);
                full_chunk(b, 2);
            } else if (S > 1 && li == 0 && le == LW_CH && lc > rampEnd && lc + LW_CH - 1 <= min(b0, b1)) {
                // below every scale's range: the recurrence alone
#pragma unroll 1
                for (int i = 0; i < LW_CH; i += 2) {
                    step(b, i, P0{}, false, 0, false, false);
                    step(b, i + 1, P1{}, false, 0, false, false);
                }
            } else if (S > 1 && lo > btop) {
                // start values enter, or a part of a chunk
                int l = lo;
                if ((l & 1) && l < lc + le) {
                    step(b, l - lc, P1{}, true, l, true, true);
                    l++;
                }
#pragma unroll 1
                for (; l + 1 < lc + le; l += 2) {
                    step(b, l - lc, P0{}, true, l, true, true);
                    step(b, l + 1 - lc, P1{}, true, l + 1, true, true);
                }
                if (l < lc + le) step(b, l - lc, P0{}, true, l, true, true);
            } else {
                // any l (for S > 1: a slot without a scale in range, only up to
                // where both are)
                if (S > 1 && btop < lc + le) le = btop + 1 - lc;
#pragma unroll 1
                for (int l = lo & ~1; l < lc + le; l += 2) {
                    if (l >= lo) step(b, l - lc, P0{}, true, l, l > b0, l > b1);
                    if (l + 1 < lc + le) step(b, l + 1 - lc, P1{}, true, l + 1, l + 1 > b0, l + 1 > b1);
                }
            }
            if (Kw > 0) rescale();
            li = le;
        }
    }
}

// ===========================================================================
// Synthesis: walk over m' and harmonic accumulation, both scales of an l
//
// CTA tile: TL = 16 P values of l by MT = 8 S values of m; a thread walks m'
// from the largest l of the tile down to 0 for its P S pairs (l, m), l = l0 +
// lane % 16 + 16 i.  Per step it reads b(l, m') and G(l, slot, q, m') of its l
// by lane and V_j(m, m', q) of the two scales by broadcast, staged 4 to 16
// values of m' at a time.  The sum over the scales is in the accumulator, so flm is
// written directly (with the scaling part), without partial rows per scale.
// P = 2, S = 4, NP = 2: 48 FP64-pipe cycles per step against 42 of shared
// memory.  Tiles lie in one interval of l with the same two scales (MwalkArgs).
// ===========================================================================
template <int NP, int P, int S>
struct MwalkSmem {
    static constexpr int TL = 16 * P, MT = 2 * WARPS * S, R = 2 * NP + 1;
    // m' per chunk: a barrier and the staging per chunk against shared memory.
    // Measured on B200 (us): 2 x 4, N = 4: 4 510, 8 461; N = 8: 4 788, 8 932;
    // 1 x 1 at B = 256, N = 2: 4 31, 8 23, 16 21, N = 5: 4 43, 8 38; 2 x 2 at B = 512, N = 8: 4 171, 8
    // 163
    static constexpr int MW_CH = P * S == 8   ? (NP <= 2 ? 8 : 4)
                                 : P * S == 4 ? 8
                                 : NP <= 2    ? 16
                                 : NP <= 4    ? 8
                                              : 4;
    static constexpr int ST = NP > 4 ? 2 : 3;                // staging buffers
    static constexpr int T_OFF = 0;                             // [CH][R][TL]
    static constexpr int V_OFF = T_OFF + MW_CH * R * TL;        // double2 [2][NP][MT][CH]
    static constexpr int BUF = V_OFF + 2 * 2 * NP * MT * MW_CH;
    static constexpr size_t BYTES = (size_t)ST * BUF * sizeof(double);
};

// flm outside the contraction's tiles: the scaling part, or zero
__device__ __forceinline__ void mwalk_fill(const MwalkArgs &a, int part, int nparts)
{
    const int B = a.B;
    for (long long i = (long long)part * THREADS + threadIdx.x; i < (long long)B * B; i += (long long)nparts * THREADS) {
        const int l = (int)(i % B), m = (int)(i / B);
        bool in = false;
        if (m <= l)
            for (int v = 0; v < a.niv; v++) in = in || (l >= a.iv_lo[v] && l < a.iv_hi[v]);
        if (in) continue;
        double2 f = make_double2(0.0, 0.0);
        if (l < a.bs && m < a.bs) f = cadd(f, cscale(a.scoeff[l + (size_t)a.bs * m], a.Phi2[l]));
        a.flm[i] = f;
    }
}

template <int NP, int P, int S, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) mwalk_kernel(const __grid_constant__ MwalkArgs a)
{
    using L = MwalkSmem<NP, P, S>;
    constexpr int TL = L::TL, MT = L::MT, R = L::R, NST = L::ST, MW_CH = L::MW_CH;
    extern __shared__ __align__(16) double msm[];
    pdl_start();
    if ((int)blockIdx.x >= a.ntiles) {
        pdl_wait();
        mwalk_fill(a, (int)blockIdx.x - a.ntiles, (int)gridDim.x - a.ntiles);
        return;
    }
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, lp = lane & 15;
    const int2 tile = a.tiles[blockIdx.x];
    const int l0 = tile.x & 0xffff, iv = tile.x >> 16, m0 = tile.y;
    const int B = a.B, vlo = a.iv_lo[iv], vhi = a.iv_hi[iv];
    const int jA = a.iv_j[iv], jB = a.iv_two[iv] ? jA + 1 : -1;
    const int MH = min(l0 + TL - 1, vhi - 1);
    const int mi = (w * 2 + (lane >> 4)) * S, mb = m0 + mi;

    // V rows that no copy fills: m past a scale's band limit, a missing scale
    const int blA = a.bl[jA], blB = jB >= 0 ? a.bl[jB] : 0;
    if (m0 + MT > min(blA, blB))
        for (int i = tid; i < NST * 2 * NP * MT * MW_CH; i += THREADS) {
            const int bufi = i / (2 * NP * MT * MW_CH), r = i % (2 * NP * MT * MW_CH);
            const int row = r / MW_CH, u = row % MT;
            if (m0 + u >= (row / MT >= NP ? blB : blA))
                reinterpret_cast<double2 *>(msm + bufi * L::BUF + L::V_OFF)[r] = make_double2(0.0, 0.0);
        }
    const int gA = (jA & 1) * NP, gB = NP - gA;  // G rows of the two scales: slot j & 1
    const int VsA = a.Vs[jA], VsB = jB >= 0 ? a.Vs[jB] : 0;
    const double2 *VA = a.V2f + a.offV[jA], *VB = jB >= 0 ? a.V2f + a.offV[jB] : a.V2f;
    // l = blo of scale jA lies in the interval but not in the scale's range
    const int actA = a.blo[jA];
    const bool edge = l0 <= actA;

    auto stage_tables = [&](int c, int buf) {
        double *b = msm + buf * L::BUF;
        const int c0 = c * MW_CH, len = gtpack_len(c0, a.Lp);
        const double *src = a.GT + gtpack_row(c0, R, a.Lp) + (l0 - gtpack_start(c0));
        constexpr int TP = TL / 2, NT = MW_CH * R * TP;
#pragma unroll
        for (int i = 0; i < (NT + THREADS - 1) / THREADS; i++) {
            const int f = tid + THREADS * i, row = f / TP, pc = 2 * (f % TP);
            if (NT % THREADS == 0 || f < NT) cp16(b + L::T_OFF + row * TL + pc, src + (size_t)row * len + pc);
        }
    };
    auto stage_v = [&](int c, int buf) {
        double *b = msm + buf * L::BUF;
        const int c0 = c * MW_CH;
        constexpr int NV = 2 * NP * MT * MW_CH;
#pragma unroll
        for (int i = 0; i < (NV + THREADS - 1) / THREADS; i++) {
            const int f = tid + THREADS * i, k = f % MW_CH, r = f / MW_CH, u = r % MT, sq = r / MT;
            const bool isB = sq >= NP;
            const int q = isB ? sq - NP : sq, bl = isB ? blB : blA;
            // (chunks of 16 m' pass the end of a V row, padded to 8)
            if ((NV % THREADS == 0 || f < NV) && m0 + u < bl && (MW_CH <= 8 || c0 + k < (isB ? VsB : VsA)))
                cp16(b + L::V_OFF + 2 * f,
                     (isB ? VB : VA) + ((size_t)q * bl + m0 + u) * (isB ? VsB : VsA) + c0 + k);
        }
    };

    const int ctop = MH / MW_CH;
#pragma unroll
    for (int i = 0; i < NST - 1; i++)
        if (ctop - i >= 0) stage_tables(ctop - i, i);

    double st[P][S], mq[S];
    int maxe = INT_MIN;
#pragma unroll
    for (int i = 0; i < P; i++)
#pragma unroll
        for (int s = 0; s < S; s++) {
            const int l = l0 + lp + 16 * i, m = mb + s;
            if (l >= vlo && l < vhi && m <= l) maxe = max(maxe, (int)a.Ee[(size_t)l * B + m]);
        }
#pragma unroll
    for (int s = 0; s < S; s++) mq[s] = (double)(mb + s);
    maxe = warp_max_i(maxe);
    int Kw = (maxe != INT_MIN && maxe < S2DW_SCALE_EXP) ? -maxe : 0;
    double e[P][S], ep[P][S];
    double2 acc[P][S];
#pragma unroll
    for (int i = 0; i < P; i++)
#pragma unroll
        for (int s = 0; s < S; s++) {
            const int l = l0 + lp + 16 * i, m = mb + s;
            st[i][s] = 0.0;
            if (l >= vlo && l < vhi && m <= l) {
                const double v = ldexp(a.Em[(size_t)l * B + m], (int)a.Ee[(size_t)l * B + m] + Kw);
                st[i][s] = ((l - m) & 1) ? -v : v;
            }
            e[i][s] = ep[i][s] = 0.0;
            acc[i][s] = make_double2(0.0, 0.0);
        }

    pdl_wait();
#pragma unroll
    for (int i = 0; i < NST - 1; i++) {
        if (ctop - i >= 0) stage_v(ctop - i, i);
        cp_commit();
    }
    for (int c = ctop, it = 0; c >= 0; c--, it++) {
        cp_wait<NST - 2>();
        __syncthreads();  // chunk c in shared memory, the previous chunk's buffer free
        if (c - (NST - 1) >= 0) {
            stage_tables(c - (NST - 1), (it + NST - 1) % NST);
            stage_v(c - (NST - 1), (it + NST - 1) % NST);
        }
        cp_commit();
        const double *b = msm + (it % NST) * L::BUF;
        const double *T = b + L::T_OFF + lp;
        const double2 *Vb = reinterpret_cast<const double2 *>(b + L::V_OFF) + mi * MW_CH;
        const int c0 = c * MW_CH;
        // one m' step at chunk row k; inj: start values enter here; excl: scale
        // jA left out where l = bl_lo of jA
        auto mstep = [&](const int k, const bool inj, const bool excl) {
            const int mpv = c0 + k;
            double2 z[P][S];
#pragma unroll
            for (int i = 0; i < P; i++)
#pragma unroll
                for (int s = 0; s < S; s++) z[i][s] = make_double2(0.0, 0.0);
#pragma unroll
            for (int r = 0; r < 2 * NP; r++) {
                const int gr = r < NP ? gA + r : gB + r - NP;
                double g[P];
#pragma unroll
                for (int i = 0; i < P; i++) g[i] = T[(k * R + gr) * TL + 16 * i];
#pragma unroll
                for (int s = 0; s < S; s++) {
                    const double2 v = Vb[(r * MT + s) * MW_CH + k];
#pragma unroll
                    for (int i = 0; i < P; i++) {
                        if (excl && i == 0 && r < NP && l0 + lp <= actA) continue;
                        z[i][s].x = fma(g[i], v.x, z[i][s].x);
                        z[i][s].y = fma(g[i], v.y, z[i][s].y);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < P; i++) {
                const double bk = T[(k * R + 2 * NP) * TL + 16 * i];
#pragma unroll
                for (int s = 0; s < S; s++) {
                    if (inj && mpv == l0 + lp + 16 * i) e[i][s] = st[i][s];
                    acc[i][s].x = fma(e[i][s], z[i][s].x, acc[i][s].x);
                    acc[i][s].y = fma(e[i][s], z[i][s].y, acc[i][s].y);
                    const double en = fma(mq[s] * bk, e[i][s], -ep[i][s]);
                    ep[i][s] = e[i][s];
                    e[i][s] = en;
                }
            }
        };
        if (c0 + MW_CH <= l0) {
            // below the tile's l: every step runs, no start value enters
            if (!edge) {
#pragma unroll
                for (int k = MW_CH - 1; k >= 0; k--) mstep(k, false, false);
            } else {
#pragma unroll
                for (int k = MW_CH - 1; k >= 0; k--) mstep(k, false, true);
            }
        } else {
#pragma unroll
            for (int k = MW_CH - 1; k >= 0; k--)
                if (c0 + k <= MH) mstep(k, true, true);
        }
        if (Kw > 0) {
            double mx = 0.0;
#pragma unroll
            for (int i = 0; i < P; i++)
#pragma unroll
                for (int s = 0; s < S; s++) mx = fmax(mx, fmax(fabs(e[i][s]), fabs(ep[i][s])));
            mx = warp_max(mx);
            if (mx > ldexp(1.0, S2DW_RENORM_EXP)) {
                const int Rr = min(S2DW_RENORM_EXP, Kw);
                const double f = ldexp(1.0, -Rr);
#pragma unroll
                for (int i = 0; i < P; i++)
#pragma unroll
                    for (int s = 0; s < S; s++) {
                        e[i][s] *= f;
                        ep[i][s] *= f;
                        acc[i][s] = cscale(acc[i][s], f);
                    }
                Kw -= Rr;
            }
        }
    }
    const double sc = ldexp(1.0, -Kw);
#pragma unroll
    for (int i = 0; i < P; i++)
#pragma unroll
        for (int s = 0; s < S; s++) {
            const int l = l0 + lp + 16 * i, m = mb + s;
            if (l < vlo || l >= vhi || m > l) continue;
            double2 *dst = a.flm + l + (size_t)B * m;
            // flm(l, m) += i^m * acc (the eta and i^{-n} phases are folded into G)
            double2 f = cipow(cscale(acc[i][s], sc), a.acc_imag ? m + 1 : m);
            if (a.acc_imag) f = cadd(*dst, f);
            else if (l < a.bs && m < a.bs) f = cadd(f, cscale(a.scoeff[l + (size_t)a.bs * m], a.Phi2[l]));
            *dst = f;
        }
}

// ===========================================================================
// Tables
// ===========================================================================
// One thread per entry of the padded tables: the analysis table G(l, slot, q,
// m') = Om(l, m') d^l_{m'n_q} K_j(l) s(l, n_q) and the synthesis table
// GT(m', r, l), r = slot NP + q: Gam(l, m') d^l_{m'n_q} c_j(l, n_q), r = 2 NP:
// b(l, m'); j the scale with j & 1 = slot whose range holds l.  Zero where
// there is none, or m' > l.
__global__ void gpack_kernel(GpackArgs a)
{
    const int kb = (a.B + 15) / 16, NP = a.NP;
    const long long total = gpack_row(16 * kb, 2 * NP);  // whole chunks of 16 l
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        // row block k holds 32 l of 2 NP rows of 32 (k + 1) values
        int k = (int)((sqrt(1.0 + (double)i / (256.0 * NP)) - 1.0) * 0.5);
        while (gpack_row(32 * (k + 1), 2 * NP) <= i) k++;
        while (gpack_row(32 * k, 2 * NP) > i) k--;
        const int len = 32 * (k + 1);
        const long long r = i - gpack_row(32 * k, 2 * NP);
        const int x = (int)(r % len), row = (int)(r / len);
        const int l = 32 * k + row / (2 * NP), sq = row % (2 * NP), slot = sq / NP, q = sq % NP;
        double v = 0.0;
        if (l < a.B && x <= l) {
            int j = slot;
            while (j <= a.J && !(a.blo[j] < l && l < a.bl[j])) j += 2;
            if (j <= a.J)
                v = a.T[(size_t)l * a.Bp + x] * a.H[hpack(l, NP, q, x)] *
                    a.kappa[((size_t)j * a.B + l) * NP + q];
        }
        a.out[i] = v;
    }
}

__global__ void gtpack_kernel(GpackArgs a)
{
    const int R = 2 * a.NP + 1, NP = a.NP, mp = blockIdx.y;
    const int len = gtpack_len(mp, a.Lp), s = gtpack_start(mp);
    double *out = a.out + gtpack_row(mp, R, a.Lp);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < R * len; i += gridDim.x * blockDim.x) {
        const int r = i / len, l = s + i % len;
        double v = 0.0;
        if (l < a.B && mp <= l) {
            if (r == 2 * NP) {
                v = a.Bcoef[(size_t)l * a.Bp + mp];
            } else {
                const int q = r % NP;
                int j = r / NP;
                while (j <= a.J && !(a.blo[j] < l && l < a.bl[j])) j += 2;
                if (j <= a.J)
                    v = a.T[(size_t)l * a.Bp + mp] * a.H[hpack(l, NP, q, mp)] *
                        a.kappa[((size_t)j * a.B + l) * NP + q];
            }
        }
        out[i] = v;
    }
}

// Largest S of the analysis kernel: 16 NP S registers of accumulators, at most 128.
constexpr int lwalk_smax(int NP) { return NP == 1 ? 8 : NP == 2 ? 4 : NP <= 4 ? 2 : 1; }

template <int NP, int S, int NS, int MINB>
int launch_lwalk_t(const LwalkArgs &a, bool dep, cudaStream_t s)
{
    using L = LwalkSmem<NP, S, NS>;
    static bool attr[64] = {false};
    int dev = 0;
    S2DW_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 64 || !attr[dev]) {
        S2DW_CUDA_TRY(cudaFuncSetAttribute(lwalk_kernel<NP, S, NS, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)L::BYTES));
        if (dev < 64) attr[dev] = true;
    }
    const int bl = a.bl[std::max(0, a.only)];
    const int grid = NS == 1 ? ((bl + 15) / 16) * ((bl + L::MT - 1) / L::MT) : a.ntiles;
    if (grid <= 0) return S2DWC_OK;
    S2DW_CUDA_TRY(launch_dep(lwalk_kernel<NP, S, NS, MINB>, grid, THREADS, L::BYTES, s, dep, a));
    return S2DWC_OK;
}

template <int NP, int P, int S, int MINB>
int launch_mwalk_t(const MwalkArgs &a, bool dep, cudaStream_t s)
{
    using L = MwalkSmem<NP, P, S>;
    static bool attr[64] = {false};
    int dev = 0;
    S2DW_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 64 || !attr[dev]) {
        S2DW_CUDA_TRY(cudaFuncSetAttribute(mwalk_kernel<NP, P, S, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)L::BYTES));
        if (dev < 64) attr[dev] = true;
    }
    const int fill = a.acc_imag ? 0 : std::min(148, (a.B * a.B + 8 * THREADS - 1) / (8 * THREADS));
    if (a.ntiles + fill <= 0) return S2DWC_OK;
    S2DW_CUDA_TRY(launch_dep(mwalk_kernel<NP, P, S, MINB>, a.ntiles + fill, THREADS, L::BYTES, s, dep, a));
    return S2DWC_OK;
}

}  // namespace

// Pairs per thread of the analysis kernel: the register limit, halved while
// the tiles would give fewer than four CTAs per SM (the launch is then bound
// by the longest walk, which fewer pairs per thread shorten); with few n, whose
// steps are short, four pairs need more CTAs than that.  Kernel on B200 (us, S = 1,
// 2, 4, 8): N = 2 (NP = 1) B = 384 41, 45, 64, 89; 448 56, 53, 74, 103; 560 92, 72, 95,
// 127; 640 129, 91, 107, 141; 700 165, 117, 119, 152; 768 207, 145, 144, 164; 900 326,
// 226, 221, 223; 1024 461, 320, 308, 302.  N = 4 (NP = 2) 384 52, 60, 76; 448 72, 70, 87;
// 560 123, 95, 105; 600 150, 114, 113; 640 174, 131, 127; 768 285, 211, 199.  N = 8 (NP =
// 4) 384 82, 89; 448 121, 99; 560 216, 170.
int lwalk_pairs(int B, int NP)
{
    int S = lwalk_smax(NP);
    const long long tp = (B + 15) / 16;
    auto ctas = [&](int s) { return s == 4 && NP == 1 ? 940 : s == 4 && NP == 2 ? 700 : 592; };
    while (S > 1 && tp * ((B + 8 * S - 1) / (8 * S)) < ctas(S)) S /= 2;
    return S;
}

// Whether the analysis walks once per scale (`only`, two pairs per thread) instead
// of once for all: with NP = 7 and 8 the merged walk's accumulators leave one pair
// per thread, whose table reads then weigh as much as its arithmetic.  Measured on
// B200 (ms per analysis, one walk and one per scale): N = 14, B = 512 0.726,
// 0.720; 640 2.54, 2.36; 1024 3.42, 2.89; 2048 19.0, 16.0; N = 16, B = 384 0.81,
// 0.87; 640 2.90, 2.69; 1024 3.97, 3.28; 2048 22.5, 17.9.  (N = 12: 1024 2.73, 2.56,
// but 512 0.56, 0.63.)  Up to B = 512 the scales share their stages' launches.
bool lwalk_per_scale(int B, int NP) { return NP >= 7 && B > 512; }

// Where the launch is bound by its longest walk (S = 1), the tiles that hold
// pairs of the small scales (bl <= B/4) are two CTAs: one walks the small
// scales' l and ends them (their many short ranges are cold code and flushes),
// the other leaves them out.  B=256 N=4: 60,000 cycles in the longest CTA, half
// of them before l = 64.
int lwalk_split(const std::vector<int> &bl, int S)
{
    int j = 0;
    while (j < (int)bl.size() && bl[j] > (bl[0] + 3) / 4) j++;
    return S == 1 && j >= 2 && j < (int)bl.size() ? j : 0;
}

void build_lwalk_tiles(const std::vector<int> &bl, int S, int jsplit, std::vector<int2> &t)
{
    // work of tile (pt, mt): the walk from max(p0, m0) up; longest first.
    // Bit 16 of y: without the small scales; of x: these alone
    t.clear();
    const int B = bl[0], MT = 2 * WARPS * S, tp = (B + 15) / 16, tm = (B + MT - 1) / MT;
    const int small = jsplit ? bl[jsplit] : 0;
    for (int pt = 0; pt < tp; pt++)
        for (int mt = 0; mt < tm; mt++) {
            const bool both = std::max(pt * 16, mt * MT) < small;
            t.push_back(make_int2(pt, mt | (both ? 1 << 16 : 0)));
            if (both) t.push_back(make_int2(pt | 1 << 16, mt));
        }
    auto length = [&](int2 a) {
        return (a.x >> 16 ? small : B) - std::max((a.x & 0xffff) * 16, (a.y & 0xffff) * MT);
    };
    std::stable_sort(t.begin(), t.end(), [&](int2 a, int2 b) { return length(a) > length(b); });
}

// P and S of the synthesis kernel by band limit: the smallest tile while there
// are fewer tiles than CTA slots (the longest walk bounds the launch), larger
// ones as the shared reads per pair begin to.  Measured on B200 (us per
// synthesis of N = 4, 1 x 1, 2 x 2, 2 x 4): B = 384 61, 70, 86; 416 74, 77, 91;
// 448 89, 83, 98; 512 121, 97, 113; 640 214, 162, 193; 768 356, 233, 272;
// 896 556, 353, 324; 1024 824, 513, 465.  N = 2: 448 51, 58, 68; 480 60, 65,
// 70; 512 72, 69, 76; 768 210, 157, 186; 896 326, 225, 218.  N = 8: 448 158,
// 136, 162; 512 218, 160, 183; 896 1029, 602, 558.  (One l and two m per
// thread lay between: N = 4 at 384 69, 512 100, 768 304.)
int2 mwalk_shape(int B, int NP)
{
    if (B >= 832) return make_int2(2, 4);
    if (B >= (NP == 1 ? 496 : 432)) return make_int2(2, 2);
    return make_int2(1, 1);
}

int build_mwalk_intervals(const std::vector<int> &bl, const std::vector<int> &blo, int B, std::vector<MwalkInterval> &iv)
{
    // maximal runs of l with the same scales
    iv.clear();
    const int J = (int)bl.size() - 1;
    for (int l = 1; l < B; l++) {
        int j = -1, n = 0;
        for (int k = J; k >= 0; k--)
            if (blo[k] < l && l < bl[k]) {
                if (n > 0 && j != k + 1) n = 2;  // not adjacent: refused below
                j = k;
                n++;
            }
        if (n > 2) return set_error(S2DWC_ERROR_SIZE_INVALID, "more than two scales at l=%d", l);
        if (n == 0) continue;
        if (!iv.empty() && iv.back().hi == l && iv.back().j == j && iv.back().two == (n == 2)) iv.back().hi = l + 1;
        else iv.push_back({l, l + 1, j, n == 2});
    }
    // the single l = bl_lo of scale j between the ranges of j + 2 and j joins
    // the interval above it (scales j, j + 1), whose kernel leaves scale j out
    // at that l
    std::vector<MwalkInterval> out;
    for (const auto &v : iv) {
        if (!out.empty() && !out.back().two && out.back().hi - out.back().lo == 1 && v.two && out.back().hi == v.lo &&
            out.back().j == v.j + 1 && out.back().lo == blo[v.j]) {
            out.back() = {out.back().lo, v.hi, v.j, true};
            continue;
        }
        out.push_back(v);
    }
    iv.swap(out);
    return S2DWC_OK;
}

void build_mwalk_tiles(const std::vector<MwalkInterval> &iv, int2 shape, std::vector<int2> &t)
{
    t.clear();
    const int TL = 16 * shape.x, MT = 2 * WARPS * shape.y;
    for (size_t v = 0; v < iv.size(); v++)
        for (int l0 = iv[v].lo & ~1; l0 < iv[v].hi; l0 += TL) {  // even: 16-byte pieces
            const int MH = std::min(l0 + TL - 1, iv[v].hi - 1);
            for (int m0 = 0; m0 <= MH; m0 += MT) t.push_back(make_int2(l0 | (int)(v << 16), m0));
        }
    std::stable_sort(t.begin(), t.end(), [](int2 a, int2 b) { return (a.x & 0xffff) > (b.x & 0xffff); });
}

int launch_lwalk(const LwalkArgs &a, bool dep, cudaStream_t s)
{
    if (a.only >= 0) {
        switch (a.NP) {
        case 1: return launch_lwalk_t<1, 2, 1, 1>(a, dep, s);
        case 2: return launch_lwalk_t<2, 2, 1, 1>(a, dep, s);
        case 3: return launch_lwalk_t<3, 2, 1, 1>(a, dep, s);
        case 4: return launch_lwalk_t<4, 2, 1, 1>(a, dep, s);
        case 5: return launch_lwalk_t<5, 2, 1, 1>(a, dep, s);
        case 6: return launch_lwalk_t<6, 2, 1, 1>(a, dep, s);
        case 7: return launch_lwalk_t<7, 2, 1, 1>(a, dep, s);
        case 8: return launch_lwalk_t<8, 2, 1, 1>(a, dep, s);
        }
    } else {
        switch (a.NP * 16 + a.S) {
        case 16 + 8: return launch_lwalk_t<1, 8, 2, 2>(a, dep, s);
        case 16 + 4: return launch_lwalk_t<1, 4, 2, 3>(a, dep, s);
        case 16 + 2: return launch_lwalk_t<1, 2, 2, 4>(a, dep, s);
        case 16 + 1: return launch_lwalk_t<1, 1, 2, 5>(a, dep, s);
        case 32 + 4: return launch_lwalk_t<2, 4, 2, 2>(a, dep, s);
        case 32 + 2: return launch_lwalk_t<2, 2, 2, 3>(a, dep, s);
        case 32 + 1: return launch_lwalk_t<2, 1, 2, 4>(a, dep, s);
        case 48 + 2: return launch_lwalk_t<3, 2, 2, 2>(a, dep, s);
        case 48 + 1: return launch_lwalk_t<3, 1, 2, 3>(a, dep, s);
        case 64 + 2: return launch_lwalk_t<4, 2, 2, 2>(a, dep, s);
        case 64 + 1: return launch_lwalk_t<4, 1, 2, 3>(a, dep, s);
        case 80 + 1: return launch_lwalk_t<5, 1, 2, 1>(a, dep, s);
        case 96 + 1: return launch_lwalk_t<6, 1, 2, 1>(a, dep, s);
        case 112 + 1: return launch_lwalk_t<7, 1, 2, 1>(a, dep, s);
        case 128 + 1: return launch_lwalk_t<8, 1, 2, 1>(a, dep, s);
        }
    }
    return set_error(S2DWC_ERROR_SIZE_INVALID, "lwalk: unsupported N=%d (N<=%d)", a.N, S2DW_NMAX);
}

template <int NP>
static int launch_mwalk_np(const MwalkArgs &a, bool dep, cudaStream_t s)
{
    if (a.shape.x == 2 && a.shape.y == 4) return launch_mwalk_t<NP, 2, 4, 2>(a, dep, s);
    if (a.shape.x == 1 && a.shape.y == 1) return launch_mwalk_t<NP, 1, 1, 3>(a, dep, s);
    if (a.shape.x == 2 && a.shape.y == 2) return launch_mwalk_t<NP, 2, 2, 2>(a, dep, s);
    return set_error(S2DWC_ERROR_ARG_INVALID, "mwalk: tile shape %d x %d", a.shape.x, a.shape.y);
}

int launch_mwalk(const MwalkArgs &a, bool dep, cudaStream_t s)
{
    switch (a.NP) {
    case 1: return launch_mwalk_np<1>(a, dep, s);
    case 2: return launch_mwalk_np<2>(a, dep, s);
    case 3: return launch_mwalk_np<3>(a, dep, s);
    case 4: return launch_mwalk_np<4>(a, dep, s);
    case 5: return launch_mwalk_np<5>(a, dep, s);
    case 6: return launch_mwalk_np<6>(a, dep, s);
    case 7: return launch_mwalk_np<7>(a, dep, s);
    case 8: return launch_mwalk_np<8>(a, dep, s);
    }
    return set_error(S2DWC_ERROR_SIZE_INVALID, "mwalk: unsupported number of n values %d (N<=%d)", a.NP, S2DW_NMAX);
}

int launch_gpack(const GpackArgs &a, bool transposed, cudaStream_t s)
{
    if (!transposed) {
        const long long total = gpack_row(16 * ((a.B + 15) / 16), 2 * a.NP);
        gpack_kernel<<<(int)std::min<long long>((total + 255) / 256, 148 * 32), 256, 0, s>>>(a);
    } else {
        const dim3 grid(std::max(1, std::min(8, a.Lp / 256)), (a.B + 15) / 16 * 16);
        gtpack_kernel<<<grid, 256, 0, s>>>(a);
    }
    S2DW_CUDA_TRY(cudaGetLastError());
    return S2DWC_OK;
}

}  // namespace s2dw
