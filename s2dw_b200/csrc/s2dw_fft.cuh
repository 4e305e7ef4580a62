// Device helpers shared by the transform stages: complex arithmetic, DFTs of
// 2^k values in registers, short odd DFTs, the beta transforms' input and
// output maps, and the 32-byte accesses of the alpha stages.
#pragma once

#include <cuda_runtime.h>

#include "s2dw_internal.h"

namespace s2dw {

// ---------------------------------------------------------------------------
// Complex helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
// exp(SIGN * 2 pi i k / 16) for k in [0, 8)
template <int SIGN>
__device__ __forceinline__ double2 w16(int k)
{
    const double C[8] = {1.0, 0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173,
                         0.0, -0.38268343236508977173, -0.70710678118654752440, -0.92387953251128675613};
    const double Sn[8] = {0.0, 0.38268343236508977173, 0.70710678118654752440, 0.92387953251128675613,
                          1.0, 0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173};
    return make_double2(C[k], SIGN * Sn[k]);
}

// In-register DFT of size R (R = 1, 2, 4, 8, 16), radix-2 decimation in time.
template <int R, int SIGN>
struct Dft {
    __device__ __forceinline__ static void run(double2 *v)
    {
        double2 ev[R / 2], od[R / 2];
#pragma unroll
        for (int i = 0; i < R / 2; i++) {
            ev[i] = v[2 * i];
            od[i] = v[2 * i + 1];
        }
        Dft<R / 2, SIGN>::run(ev);
        Dft<R / 2, SIGN>::run(od);
#pragma unroll
        for (int k = 0; k < R / 2; k++) {
            double2 t;
            if (k == 0) t = od[k];
            else if (4 * k == R) t = (SIGN < 0) ? make_double2(od[k].y, -od[k].x) : make_double2(-od[k].y, od[k].x);
            else t = cmul(od[k], w16<SIGN>(k * (16 / R)));
            v[k] = cadd(ev[k], t);
            v[k + R / 2] = csub(ev[k], t);
        }
    }
};
template <int SIGN>
struct Dft<1, SIGN> {
    __device__ __forceinline__ static void run(double2 *) {}
};

template <int SIGN>
__device__ __forceinline__ void twiddle_powers16(double2 (&v)[16], double2 w)
{
    if (SIGN > 0) w = cconj(w);
    const double2 w2 = cmul(w, w), w4 = cmul(w2, w2), w8 = cmul(w4, w4);
    const double2 w3 = cmul(w2, w), w5 = cmul(w4, w), w6 = cmul(w4, w2), w7 = cmul(w4, w3);
    v[1] = cmul(v[1], w);
    v[2] = cmul(v[2], w2);
    v[3] = cmul(v[3], w3);
    v[4] = cmul(v[4], w4);
    v[5] = cmul(v[5], w5);
    v[6] = cmul(v[6], w6);
    v[7] = cmul(v[7], w7);
    v[8] = cmul(v[8], w8);
    v[9] = cmul(v[9], cmul(w8, w));
    v[10] = cmul(v[10], cmul(w8, w2));
    v[11] = cmul(v[11], cmul(w8, w3));
    v[12] = cmul(v[12], cmul(w8, w4));
    v[13] = cmul(v[13], cmul(w8, w5));
    v[14] = cmul(v[14], cmul(w8, w6));
    v[15] = cmul(v[15], cmul(w8, w7));
}

// 32-byte accesses of the alpha stages (the two b columns of a b pair at
// one (g, m)): one 256-bit access instead of two 128-bit ones halves the
// L1 wavefronts of these row-strided loads and stores.  The streamed input
// is not kept in L1, which holds the chirp tables.
__device__ __forceinline__ void ld_pair(const double2 *p, double2 &a, double2 &b)
{
    asm volatile("ld.global.L1::no_allocate.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y)
        : "l"(p));
}
__device__ __forceinline__ void st_pair(double2 *p, double2 a, double2 b)
{
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y)
                 : "memory");
}

// Filter spectrum entry k of a Bluestein transform.  The alpha stages' filter
// h(d) = conj(chirp(d)) is even in d (no offsets), so its spectrum is even:
// Hf[k] = Hf[M - k]; reading only k <= M/2 halves the table's cache
// footprint (32 KB instead of 64 KB at M = 4096).
template <int MODE>
__device__ __forceinline__ double2 hf_at(const double2 *Hf, int k, int M)
{
    if (MODE == CZT_ANA_ALPHA || MODE == CZT_SYN_ALPHA) return Hf[k <= (M >> 1) ? k : M - k];
    return Hf[k];
}

// ---- beta transforms as FFTs of length L = 2 bl (Makhoul's algorithm) ----
// Analysis (s2dw_core_mod.f90:708-743), one row X(p), p < bl:
//   cos rows (m+N-1 even): Y(b) = sum_p c_p X(p) cos(p beta_b), c_0 = 1, c_p = 2,
//   sin rows (m+N-1 odd):  Y(b) = X(0) + sum_{p>=1} 2i X(p) sin(p beta_b),
// beta_b = pi (2b+1)/(2L), b < L.  The cos sum is a DCT-III of length L:
//   V_0 = X(0), V_k = e_k X(k) (0 < k < bl), V_bl = 0, V_k = conj(e_{L-k}) X(L-k) (k > bl),
//   v = sum_k V_k e^{+2 pi i k n/L},  Y(2n) = v_n, Y(2n+1) = v_{L-1-n}  (n < bl),
// e_k = exp(i pi k/(2L)) (the czt.pre table).  The sin sum is the same DCT-III
// of the reversed input times i(-1)^b, which moves factors -i (k < bl) and +i
// (k > bl) onto V and i, -i onto the two output halves; its V_0 is 0 and the
// reference's m' = 0 term X(0) (eta = 1) is added to every output.
// Synthesis (:1157-1198), one row u_b, b < L, folded over +-m':
//   cos rows (m+n even): V'(0) = sum_b u_b, V'(m') = 2 sum_b u_b cos(m' beta_b),
//   sin rows (m+n odd):  V'(m') = -2i sum_b u_b sin(m' beta_b),
// a DCT-II of length L: permute v_n = u_{2n}, v_{L-1-n} = u_{2n+1} (n < bl),
// V = sum_n v_n e^{-2 pi i k n/L}, V'(m') = conj(e_m') V_m' +- e_m' V_{L-m'}
// (+ cos, - sin; the sin rows' input carries (-1)^b).  A sin row's V'(0)
// multiplies d^l_{0m}(pi/2) d^l_{0n}(pi/2), which is zero for every l when m+n
// is odd, so it is stored as 0.

// DCT-III input V_k of the analysis beta transform of row X (bl values).
__device__ __forceinline__ double2 ana_beta_in(const double2 *X, int k, int bl, bool sn, const double2 *e)
{
    if (k == 0) return sn ? make_double2(0.0, 0.0) : X[0];
    if (k < bl) {
        const double2 x = cmul(X[k], e[k]);
        return sn ? make_double2(x.y, -x.x) : x;  // -i x
    }
    if (k == bl) return make_double2(0.0, 0.0);
    const int p = 2 * bl - k;
    const double2 x = cmul(X[p], cconj(e[p]));
    return sn ? make_double2(-x.y, x.x) : x;  // i x
}

// Output of the analysis beta transform held at FFT index j: its b, and the
// value (the sin rows' factor i or -i and the m' = 0 term x0 applied).
__device__ __forceinline__ double2 ana_beta_out(double2 y, int j, int bl, bool sn, double2 x0, int *b)
{
    if (j < bl) {
        *b = 2 * j;
        if (sn) y = make_double2(-y.y + x0.x, y.x + x0.y);  // i y + x0
    } else {
        *b = 4 * bl - 1 - 2 * j;
        if (sn) y = make_double2(y.y + x0.x, -y.x + x0.y);  // -i y + x0
    }
    return y;
}

// Folded synthesis beta output V'(m') from the FFT values at m' and L-m'.
__device__ __forceinline__ double2 syn_beta_out(double2 vk, double2 vlk, int mpv, bool sn, const double2 *e)
{
    if (mpv == 0) return sn ? make_double2(0.0, 0.0) : vk;
    const double2 y = cmul(vk, cconj(e[mpv])), z = cmul(vlk, e[mpv]);
    return sn ? csub(y, z) : cadd(y, z);
}

// ===========================================================================
// Transforms of M = 16 ... 2048 points, several rows per CTA of 128 threads
//
// A row of M points has TPR = M/V threads with V values each (V = 4, 8, 16
// for M < 64, < 256, from 256), so a CTA holds 128/TPR rows (32 ... 1) and even
// the rows of a small scale spread over the GPU.  Stockham passes of radix V,
// Q = M/V^2 (if > 1), V: the input and the output of a transform are at
// positions t + i TPR, so that a forward transform, a product and an inverse
// stay in registers, and one or two exchanges through shared memory (padded
// every V values: conflict-free for eight-lane phases) lie between.  Rows of
// up to 32 threads lie in one warp and need no CTA barrier.  Twiddles are
// products of one root per pass from a table of exp(-2 pi i k/2048).
// ===========================================================================
constexpr int ST_THREADS = 128;
constexpr int ST_TW = 2048;  // points of the twiddle table

// VMAX: 16, or 8 to keep a kernel's registers low (up to 512 points).
__host__ __device__ constexpr int row_fft_v(int lg, int vmax) { return lg >= 8 && vmax == 16 ? 16 : lg >= 6 ? 8 : 4; }

template <int LG, int VMAX = 16>
struct RowFft {
    static constexpr int M = 1 << LG;
    static constexpr int V = row_fft_v(LG, VMAX);
    static constexpr int LV = V == 16 ? 4 : V == 8 ? 3 : 2;
    static constexpr int Q = M / (V * V);
    static constexpr int TPR = M / V, ROWS = ST_THREADS / TPR;
    static constexpr int PITCH = M + (M >> LV) + 1;  // shared values per row
    static_assert(Q >= 1 && Q <= 8 && TPR <= ST_THREADS, "row size");

    __device__ __forceinline__ static int pad(int i) { return i + (i >> LV); }
    __device__ __forceinline__ static void sync()
    {
        if (TPR <= 32) __syncwarp();
        else __syncthreads();
    }
    template <int R, int SIGN>
    __device__ __forceinline__ static void twiddle(double2 *v, double2 w)
    {
        if (SIGN > 0) w = cconj(w);
        double2 p[R];
        p[1] = w;
#pragma unroll
        for (int s = 2; s < R; s++) p[s] = cmul(p[s / 2], p[s - s / 2]);
#pragma unroll
        for (int s = 1; s < R; s++) v[s] = cmul(v[s], p[s]);
    }
    // v: values at t + i TPR in, and out; buf: the row's PITCH shared values,
    // free before the call for all threads of the row, and after it
    template <int SIGN>
    __device__ __forceinline__ static void run(double2 (&v)[V], double2 *buf, int t, const double2 *tw)
    {
        Dft<V, SIGN>::run(v);
#pragma unroll
        for (int s = 0; s < V; s++) buf[pad(t * V + s)] = v[s];
        sync();
        if constexpr (Q > 1) {
            const double2 w = __ldg(tw + (t % V) * (ST_TW / (V * Q)));
#pragma unroll
            for (int u = 0; u < V / Q; u++)
#pragma unroll
                for (int s = 0; s < Q; s++) v[u * Q + s] = buf[pad(t + u * TPR + s * (M / Q))];
            sync();
#pragma unroll
            for (int u = 0; u < V / Q; u++) {
                twiddle<Q, SIGN>(v + u * Q, w);
                Dft<Q, SIGN>::run(v + u * Q);
                const int j = t + u * TPR, o = (j >> LV) * (V * Q) + (j & (V - 1));
#pragma unroll
                for (int s = 0; s < Q; s++) buf[pad(o + s * V)] = v[u * Q + s];
            }
            sync();
        }
        const double2 w = __ldg(tw + t * (ST_TW / M));
#pragma unroll
        for (int s = 0; s < V; s++) v[s] = buf[pad(t + s * TPR)];
        sync();
        twiddle<V, SIGN>(v, w);
        Dft<V, SIGN>::run(v);
    }
};

// Asynchronous 16-byte copies of values that the copying thread itself reads.
__device__ __forceinline__ void cp16_own(double2 *smem, const double2 *gmem)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_own_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The entry (scale) of this CTA, and the CTA's index within it.
__device__ __forceinline__ const StageEnt &stage_entry(const StageArgs &a, int &cta)
{
    int e = 0;
    while (e + 1 < a.n && (int)blockIdx.x >= a.e[e + 1].cta0) e++;
    cta = (int)blockIdx.x - a.e[e].cta0;
    return a.e[e];
}

// ---- short DFTs of the prime-factor alpha stages
// cos(2 pi j / R) and sin(2 pi j / R), j < R (local constant tables: with j
// known after unrolling they fold into immediates)
template <int R>
__device__ __forceinline__ void pfa_cs(int j, double &c, double &s);
template <>
__device__ __forceinline__ void pfa_cs<5>(int j, double &c, double &s)
{
    constexpr double C[5] = {1.0, 0.309016994374947424102, -0.809016994374947424102, -0.809016994374947424102, 0.309016994374947424102};
    constexpr double S[5] = {0.0, 0.951056516295153572116, 0.587785252292473129169, -0.587785252292473129169, -0.951056516295153572116};
    c = C[j];
    s = S[j];
}
template <>
__device__ __forceinline__ void pfa_cs<7>(int j, double &c, double &s)
{
    constexpr double C[7] = {1.0, 0.623489801858733530525, -0.222520933956314404289, -0.900968867902419126236, -0.900968867902419126236, -0.222520933956314404289, 0.623489801858733530525};
    constexpr double S[7] = {0.0, 0.781831482468029808708, 0.974927912181823607018, 0.433883739117558120476, -0.433883739117558120476, -0.974927912181823607018, -0.781831482468029808708};
    c = C[j];
    s = S[j];
}
template <>
__device__ __forceinline__ void pfa_cs<9>(int j, double &c, double &s)
{
    constexpr double C[9] = {1.0, 0.766044443118978035202, 0.173648177666930348852, -0.5, -0.939692620785908384054, -0.939692620785908384054, -0.5, 0.173648177666930348852, 0.766044443118978035202};
    constexpr double S[9] = {0.0, 0.642787609686539326323, 0.984807753012208059367, 0.866025403784438646764, 0.342020143325668733044, -0.342020143325668733044, -0.866025403784438646764, -0.984807753012208059367, -0.642787609686539326323};
    c = C[j];
    s = S[j];
}
template <>
__device__ __forceinline__ void pfa_cs<13>(int j, double &c, double &s)
{
    constexpr double C[13] = {1.0, 0.885456025653209895900, 0.568064746731155802512, 0.120536680255323053349, -0.354604887042535625970, -0.748510748171101098635, -0.970941817426052027157, -0.970941817426052027157, -0.748510748171101098635, -0.354604887042535625970, 0.120536680255323053349, 0.568064746731155802512, 0.885456025653209895900};
    constexpr double S[13] = {0.0, 0.464723172043768545656, 0.822983865893656394580, 0.992708874098053992801, 0.935016242685414823440, 0.663122658240795202377, 0.239315664287557767149, -0.239315664287557767149, -0.663122658240795202377, -0.935016242685414823440, -0.992708874098053992801, -0.822983865893656394580, -0.464723172043768545656};
    c = C[j];
    s = S[j];
}

// In-place DFT of length R (odd) with exp(SIGN 2 pi i k m / R):
// y_m = x_0 + sum_k (x_k + x_{R-k}) cos + SIGN i sum_k (x_k - x_{R-k}) sin.
template <int R, int SIGN>
__device__ __forceinline__ void pfa_dft(double2 (&x)[R])
{
    constexpr int H = (R - 1) / 2;
    double2 ap[H], am[H];
    double2 y0 = x[0];
#pragma unroll
    for (int k = 1; k <= H; k++) {
        ap[k - 1] = cadd(x[k], x[R - k]);
        am[k - 1] = csub(x[k], x[R - k]);
        y0 = cadd(y0, ap[k - 1]);
    }
    const double2 x0 = x[0];
    x[0] = y0;
#pragma unroll
    for (int m = 1; m <= H; m++) {
        double2 P = x0, Q = make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 1; k <= H; k++) {
            double c, sn;
            pfa_cs<R>((k * m) % R, c, sn);
            P.x = fma(ap[k - 1].x, c, P.x);
            P.y = fma(ap[k - 1].y, c, P.y);
            Q.x = fma(am[k - 1].x, sn, Q.x);
            Q.y = fma(am[k - 1].y, sn, Q.y);
        }
        // SIGN i Q
        const double2 iq = SIGN > 0 ? make_double2(-Q.y, Q.x) : make_double2(Q.y, -Q.x);
        x[m] = cadd(P, iq);
        x[R - m] = csub(P, iq);
    }
}

template <>
__device__ __forceinline__ void pfa_cs<11>(int j, double &c, double &s)
{
    constexpr double C[11] = {
        1.00000000000000000000, 0.841253532831181168862, 0.415415013001886425529, -0.142314838273285140444,
        -0.654860733945285064057, -0.959492973614497389890, -0.959492973614497389890, -0.654860733945285064057,
        -0.142314838273285140444, 0.415415013001886425529, 0.841253532831181168862};
    constexpr double S[11] = {
        0.0, 0.540640817455597582108, 0.909631995354518371412, 0.989821441880932732376, 0.755749574354258283774,
        0.281732556841429697711, -0.281732556841429697711, -0.755749574354258283774, -0.989821441880932732376,
        -0.909631995354518371412, -0.540640817455597582108};
    c = C[j];
    s = S[j];
}
template <>
__device__ __forceinline__ void pfa_cs<23>(int j, double &c, double &s)
{
    constexpr double C[23] = {
        1.00000000000000000000, 0.962917287347799295015, 0.854419404546488552548, 0.682553143218654082875,
        0.460065037731152126042, 0.203456013052633789878, -0.0682424133646709759212, -0.334879612170986151958,
        -0.576680322114867141251, -0.775711290704419807041, -0.917211301505453017844, -0.990685946036330752342,
        -0.990685946036330752342, -0.917211301505453017844, -0.775711290704419807041, -0.576680322114867141251,
        -0.334879612170986151958, -0.0682424133646709759212, 0.203456013052633789878, 0.460065037731152126042,
        0.682553143218654082875, 0.854419404546488552548, 0.962917287347799295015};
    constexpr double S[23] = {
        0.0, 0.269796771157024271245, 0.519583950035433578133, 0.730835964278124101651, 0.887885218402375234984,
        0.979084087682322875633, 0.997668769190539198454, 0.942260922118820495618, 0.816969893010442016973,
        0.631087944326052789367, 0.398401089846241457998, 0.136166649096246590761, -0.136166649096246590761,
        -0.398401089846241457998, -0.631087944326052789367, -0.816969893010442016973, -0.942260922118820495618,
        -0.997668769190539198454, -0.979084087682322875633, -0.887885218402375234984, -0.730835964278124101651,
        -0.519583950035433578133, -0.269796771157024271245};
    c = C[j];
    s = S[j];
}

// In-place-input DFT of length R (odd), outputs written to out[base + m S]:
// the symmetric pairs overwrite x (x_k <- x_k + x_{R-k}, x_{R-k} <- x_k - x_{R-k}),
// which keeps the registers of a long DFT (R = 23) to about R complex values.
template <int R, int SIGN>
__device__ __forceinline__ void pfa_dft_out(double2 (&x)[R], double2 *out, int base, int S)
{
    constexpr int H = (R - 1) / 2;
    const double2 x0 = x[0];
    double2 y0 = x0;
#pragma unroll
    for (int k = 1; k <= H; k++) {
        const double2 p = cadd(x[k], x[R - k]), q = csub(x[k], x[R - k]);
        x[k] = p;
        x[R - k] = q;
        y0 = cadd(y0, p);
    }
    out[base] = y0;
#pragma unroll
    for (int m = 1; m <= H; m++) {
        double2 P = x0, Q = make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 1; k <= H; k++) {
            double c, sn;
            pfa_cs<R>((k * m) % R, c, sn);
            P.x = fma(x[k].x, c, P.x);
            P.y = fma(x[k].y, c, P.y);
            Q.x = fma(x[R - k].x, sn, Q.x);
            Q.y = fma(x[R - k].y, sn, Q.y);
        }
        const double2 iq = SIGN > 0 ? make_double2(-Q.y, Q.x) : make_double2(Q.y, -Q.x);
        out[base + m * S] = cadd(P, iq);
        out[base + (R - m) * S] = csub(P, iq);
    }
}

// The same DFT with the real and the imaginary parts of a column in two
// neighbouring lanes (even: real): the sums over the symmetric pairs act on
// each part alone and only the sine sums are exchanged.  Half the registers per
// thread and twice the threads of pfa_dft_out.  Every lane of the warp calls
// it; x: this lane's part of the inputs, written to out[2 (base + m S)] + part
// if `live` (doubles).
template <int R, int SIGN>
__device__ __forceinline__ void pfa_dft_part(double (&x)[R], double *out, int base, int S, bool live)
{
    constexpr int H = (R - 1) / 2;
    const double sg = (threadIdx.x & 1) ? (double)SIGN : -(double)SIGN;
    const double x0 = x[0];
    double y0 = x0;
#pragma unroll
    for (int k = 1; k <= H; k++) {
        const double p = x[k] + x[R - k], q = x[k] - x[R - k];
        x[k] = p;
        x[R - k] = q;
        y0 += p;
    }
    if (live) out[2 * base] = y0;
#pragma unroll
    for (int m = 1; m <= H; m++) {
        double P = x0, Q = 0.0;
#pragma unroll
        for (int k = 1; k <= H; k++) {
            double c, sn;
            pfa_cs<R>((k * m) % R, c, sn);
            P = fma(x[k], c, P);
            Q = fma(x[R - k], sn, Q);
        }
        const double o = sg * __shfl_xor_sync(0xffffffffu, Q, 1);
        if (live) {
            out[2 * (base + m * S)] = P + o;
            out[2 * (base + (R - m) * S)] = P - o;
        }
    }
}

template <>
__device__ __forceinline__ void pfa_cs<3>(int j, double &c, double &s)
{
    constexpr double C[3] = {
        1.00000000000000000000, -0.500000000000000000000, -0.500000000000000000000};
    constexpr double S[3] = {
        0.0, 0.866025403784438646764, -0.866025403784438646764};
    c = C[j];
    s = S[j];
}
template <>
__device__ __forceinline__ void pfa_cs<31>(int j, double &c, double &s)
{
    constexpr double C[31] = {
        1.00000000000000000000, 0.979529941252494493938, 0.918957811620230629127, 0.820763441207276326364,
        0.688966919075686567801, 0.528964010326962457365, 0.347305252844820285542, 0.151427777504576663657,
        -0.050649168838712712279, -0.250652532258720539315, -0.440394151557634309516,
        -0.612105982547662844147, -0.758758122692790901913, -0.874346616144582118827,
        -0.954139256400048851476, -0.994869323391895146321, -0.994869323391895146321,
        -0.954139256400048851476, -0.874346616144582118827, -0.758758122692790901913,
        -0.612105982547662844147, -0.440394151557634309516, -0.250652532258720539315,
        -0.050649168838712712279, 0.151427777504576663657, 0.347305252844820285542, 0.528964010326962457365,
        0.688966919075686567801, 0.820763441207276326364, 0.918957811620230629127, 0.979529941252494493938};
    constexpr double S[31] = {
        0.0, 0.201298520088660079142, 0.394355855113318580102, 0.571268215094792279157,
        0.724792787229119958865, 0.848644257494750950464, 0.937752132147080458429, 0.988468324328111399162,
        0.998716507171052807146, 0.968077118866204305153, 0.897804539570741657137, 0.790775736937698582078,
        0.651372482722222207454, 0.485301962531081025215, 0.299363122973357954008, 0.101168321987432177786,
        -0.101168321987432177786, -0.299363122973357954008, -0.485301962531081025215,
        -0.651372482722222207454, -0.790775736937698582078, -0.897804539570741657137,
        -0.968077118866204305153, -0.998716507171052807146, -0.988468324328111399162,
        -0.937752132147080458429, -0.848644257494750950464, -0.724792787229119958865,
        -0.571268215094792279157, -0.394355855113318580102, -0.201298520088660079142};
    c = C[j];
    s = S[j];
}

template <>
__device__ __forceinline__ void pfa_cs<17>(int j, double &c, double &s)
{
    constexpr double C[17] = {
        1.00000000000000000000, 0.932472229404355804573, 0.739008917220659115925, 0.445738355776538267396,
        0.092268359463301995240, -0.273662990072082863539, -0.602634636379256389179, -0.850217135729614152134,
        -0.982973099683901778282, -0.982973099683901778282, -0.850217135729614152134, -0.602634636379256389179,
        -0.273662990072082863539, 0.092268359463301995240, 0.445738355776538267396, 0.739008917220659115925,
        0.932472229404355804573};
    constexpr double S[17] = {
        0.0, 0.361241666187152948745, 0.673695643646557211713, 0.895163291355062322067, 0.995734176295034521871,
        0.961825643172819070409, 0.798017227280239503333, 0.526432162877355800245, 0.183749517816570331574,
        -0.183749517816570331574, -0.526432162877355800245, -0.798017227280239503333, -0.961825643172819070409,
        -0.995734176295034521871, -0.895163291355062322067, -0.673695643646557211713, -0.361241666187152948745};
    c = C[j];
    s = S[j];
}

}  // namespace s2dw
