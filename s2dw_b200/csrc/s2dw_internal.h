// Internal declarations shared by the host and device parts of libs2dw_cuda.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <exception>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "../../include/s2dw_cuda.h"

namespace s2dw {

// ---------------------------------------------------------------------------
// Errors: every failing entry point records a code and a message.
// ---------------------------------------------------------------------------
int set_error(int code, const char *fmt, ...);

#define S2DW_CUDA_TRY(call)                                                              \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess)                                                           \
            return ::s2dw::set_error(S2DWC_ERROR_CUDA, "%s failed: %s (%s:%d)", #call,   \
                                     cudaGetErrorString(e_), __FILE__, __LINE__);        \
    } while (0)

// No C++ exception may cross the C ABI (a Fortran or ctypes caller would be
// terminated): the body of every int-returning entry point runs inside
// S2DW_API_TRY ... S2DW_API_CATCH, which turns a failed host allocation into
// S2DWC_ERROR_MEM_ALLOC_FAIL and any other exception into
// S2DWC_ERROR_ARG_INVALID with its message.
#define S2DW_API_TRY try {
#define S2DW_API_CATCH                                                                        \
    }                                                                                         \
    catch (const std::bad_alloc &) {                                                          \
        return ::s2dw::set_error(S2DWC_ERROR_MEM_ALLOC_FAIL, "%s: host allocation failed",    \
                                 __func__);                                                   \
    }                                                                                         \
    catch (const std::exception &ex_) {                                                       \
        return ::s2dw::set_error(S2DWC_ERROR_ARG_INVALID, "%s: %s", __func__, ex_.what());    \
    }                                                                                         \
    catch (...) {                                                                             \
        return ::s2dw::set_error(S2DWC_ERROR_ARG_INVALID, "%s: unexpected exception", __func__); \
    }

// Programmatic dependent launch: the kernels of a call that follow one another
// on one stream are launched with it (`dep`), so that a kernel's CTAs are in
// place, and its tables on their way, when its predecessor ends.  Every such
// kernel calls pdl_start() and, before it touches anything a kernel before it
// reads or writes, pdl_wait() (the alpha kernels, which have nothing to load
// earlier, wait first; the other order measured the same); launched without the
// attribute both do nothing.  A kernel whose predecessor on the stream is not one
// of this call is launched without it.
template <typename... P, typename... A>
inline cudaError_t launch_dep(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool dep,
                              A &&...args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = dep ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

// ---------------------------------------------------------------------------
// Host helpers restating the reference's scalar routines.
// ---------------------------------------------------------------------------
bool assimilate_int(double x, int *y);
int comp_jmax(int B, double alpha);
bool params_valid(int J, int B, double alpha, int N /* <0: absent */);
void band_limits(int jj, int B, double alpha, int *bl_hi, int *bl_lo);
double quad_weight(double theta, int B);

// Positive n set of the transform: n in [0, N) with N+n odd (the k_indicator
// test of s2dw_core_mod.f90:693 / :1146).  Returns its size NP (<= 4 for N<=8).
int positive_nset(int N, int *nq);

// ---------------------------------------------------------------------------
// Recurrence tables for d^l_{m'm}(pi/2), built on the host in long double.
//   l-walk (fixed m', m, stepping l):   e_{l+1} = -a_m(l) a_m'(l) e_l - e_{l-1},
//                                       d = Om_l(m) Om_l(m') e
//   m'-walk (fixed l, m, stepping m' down): e_{m'-1} = m b(l,m') e_{m'} - e_{m'+1},
//                                       d = Gam(l,m') e
// Start values are stored as mantissa (double in [1,2)) and binary exponent.
// All 2-D tables are [l*B + x] with zeros where x > l.
// ---------------------------------------------------------------------------
// Azimuthal band limits: N <= S2DW_NMAX (FP64 form; the split form N <= 8),
// so at most S2DW_NPMAX values n >= 0 with N + n odd.
constexpr int S2DW_NMAX = 16;
constexpr int S2DW_NPMAX = S2DW_NMAX / 2;
// Largest scale index J (scales j = 0..J): per-scale arrays passed to kernels
// by value are sized by it (J+1 entries; MwalkArgs, the largest, is 3.4 KB of the
// 4 KB that kernel arguments may be).
constexpr int S2DW_JMAX = 127;

struct RecTables {
    int B = 0, HN = 8;
    std::vector<double> Om, Acoef;     // l-walk scale chains and coefficients
    std::vector<double> Stm;           // l-walk start E(l0,k)/Om_l0(k) mantissa
    std::vector<int32_t> Ste;          //   ... exponent
    std::vector<double> Gam, Bcoef;    // m'-walk chains and coefficients
    std::vector<double> Em;            // edge values E(l,m)=sqrt(C(2l,l+m))/2^l
    std::vector<int32_t> Ee;
    std::vector<double> H;             // d^l_{m'n}(pi/2), n < HN: [(l*HN+n)*B + m']
};
void build_rec_tables(int B, int hn, RecTables &t);  // H for n < hn

// ---------------------------------------------------------------------------
// Chirp-z (Bluestein) transform specification:
//   y[b] = sum_{k<K} x[k] exp(2 pi i s (k+k0)(b+b0)/L),  b < Bout,
// with k0, b0 integers or half-integers (passed doubled).
// ---------------------------------------------------------------------------
struct CztSpec {
    int K, Bout, L, s, k0x2, b0x2, M;
};
int czt_size(int K, int Bout);  // power of two M >= max(16, K+Bout-1)
void build_czt_tables(const CztSpec &c, std::vector<double2> &pre, std::vector<double2> &post,
                      std::vector<double2> &Hf);
// exp(i pi k / (4 bl)) for k < bl: the pre/post twiddle of the FFT beta modes.
void build_beta_twiddles(int bl, std::vector<double2> &tw);
// Two-level twiddle tables for a power-of-two FFT of size M:
// W_M^x = hi[x >> 6] * lo[x & 63], W_M = exp(-2 pi i / M).
void build_twiddles(int M, std::vector<double2> &hi, std::vector<double2> &lo);

// ---------------------------------------------------------------------------
// Device kernels (s2dw_kernels.cu)
// ---------------------------------------------------------------------------
// Transform modes.  CZT_* are chirp-z (Bluestein) transforms of any length;
// FFT_ANA_BETA / FFT_SYN_BETA are the beta transforms as one power-of-two FFT
// of length L = 2*bl (used when 2*bl is a power of two, bl >= 8): the analysis
// beta sum is a DCT-III of length L (cos rows) or, on the reversed input, a
// DST-III (i sin rows); the synthesis beta sum with its +-m' fold is the
// matching DCT-II / DST-II.  Each runs as one complex FFT of length L with a
// pre-twiddle, an even/odd reordering and a post-twiddle (Makhoul's
// algorithm, complex-linear, so complex rows need no real/imaginary split).
enum CztMode {
    CZT_ANA_BETA = 0,
    CZT_ANA_ALPHA = 1,
    CZT_SYN_ALPHA = 2,
    CZT_SYN_BETA = 3,
    FFT_ANA_BETA = 4,
    FFT_SYN_BETA = 5
};

struct CztDev {
    int M = 0;
    CztSpec spec{};
    double2 *pre = nullptr, *post = nullptr, *Hf = nullptr;
};

struct TwDev {
    int M = 0;
    double2 *hi = nullptr, *lo = nullptr;
};

// Packed triangular tables of the contraction kernels, rows of R values per
// degree.  Analysis, G: row l holds the m' < gpack_len(l) (l rounded up to 32),
// its R rows consecutive.  Synthesis, GT: row m' holds the l >= gtpack_start(m')
// up to the padded Lp.
__host__ __device__ __forceinline__ int gpack_len(int l) { return 32 * ((l >> 5) + 1); }
__host__ __device__ __forceinline__ long long gpack_row(int l, int R)
{
    const long long k = l >> 5;
    return R * (512 * k * (k + 1) + 32 * (l & 31) * (k + 1));
}
// d^l_{m'n_q}(pi/2), m' <= l
__host__ __device__ __forceinline__ size_t hpack(int l, int NP, int q, int mp)
{
    return (size_t)NP * l * (l + 1) / 2 + (size_t)q * (l + 1) + mp;
}
// (a tile of at most 32 l reads the chunks of up to 16 m' that start at or
// below its last l, so 32 values before the chunk's own m' are kept)
__host__ __device__ __forceinline__ int gtpack_start(int mp) { return mp < 32 ? 0 : 16 * ((mp >> 4) - 2); }
__host__ __device__ __forceinline__ int gtpack_len(int mp, int Lp) { return Lp - gtpack_start(mp); }
__host__ __device__ __forceinline__ long long gtpack_row(int mp, int R, int Lp)
{
    const long long k = mp < 32 ? 0 : (mp >> 4) - 2;
    const long long skipped = 8 * k * (k - 1) + (mp & 15) * k;  // /16
    return R * ((long long)mp * Lp - 16 * skipped);
}

// Tables of the plan use a padded row stride Bp = roundup(B, 32); Acoef and F have
// 64 values of slack where tiles of more than 32 m read past the last row
// (lwalk_slack).
struct LwalkArgs {
    int B, Bp, N, NP, J;
    int nq[S2DW_NPMAX];
    const double *Acoef;  // [l*Bp + x]
    const double *Stm;    // [l0*B + k]
    const int32_t *Ste;
    const double *G;      // gpack_row(l, 2 NP): Om(l,m') d^l_{m'n_q} K_j(l) s(l,n_q), row slot NP + q, slot = j & 1
    const double2 *F;     // [l*Bp + m] = i^{-m} Om(l,m) flm(l,m)
    const double2 *ph;    // [g (2N-1) + n+N-1] = exp(i pi n g / N)
    double2 *Tg;          // scale j: Tg + off[j], [g][m][m'] N x bl x bl
    const int2 *tiles;    // (p-tile, m-tile) per CTA, longest walks first
    int ntiles, S;        // S: m per half warp (lwalk_pairs)
    int jsplit;           // first of the small scales with CTAs of their own (lwalk_split)
    int only;             // -1: every scale; else this scale alone
    // 0: Tg = T.  1: G holds the second real part b of S = eta (a + i b)
    // (a general complex Slm): Tg += T with the +n terms times -i and the
    // -n terms times +i (conj(S) for n >= 0, S for n < 0).
    int acc_imag;
    short bl[S2DW_JMAX + 1], blo[S2DW_JMAX + 1];
    long long off[S2DW_JMAX + 1];
};

// Interval lo <= l < hi whose degrees lie in the ranges of scale j and, if
// two, of scale j + 1 (scale j's range may start at lo + 1).
struct MwalkInterval {
    int lo, hi, j;
    bool two;
};

struct MwalkArgs {
    int B, NP, bs, niv;
    const double *Em;     // [l*B + m]
    const int32_t *Ee;
    const double *GT;     // gtpack_row(m', 2 NP + 1, Lp): Gam(l,m') d^l_{m'n_q} c_j(l,n_q), row slot NP + q; row 2 NP: b(l,m')
    int Lp;               // roundup(B, 8) + the tiles' l
    const double2 *V2f;   // scale j: V2f + offV[j], [(q*bl + m)*Vs + m']
    const double2 *scoeff;
    const double *Phi2;
    double2 *flm;         // flm[l + B m], every value written (the scaling part added)
    const int2 *tiles;    // (l0 | interval << 16, m0) per CTA, longest walks first
    int ntiles;
    int2 shape;           // P x S (mwalk_shape)
    // 0: flm = result.  1: GT holds the second real part b of S = eta (a + i b)
    // (a general complex Slm): flm += i * result.
    int acc_imag;
    short iv_lo[2 * S2DW_JMAX + 2], iv_hi[2 * S2DW_JMAX + 2];
    unsigned char iv_j[2 * S2DW_JMAX + 2], iv_two[2 * S2DW_JMAX + 2];
    short bl[S2DW_JMAX + 1], blo[S2DW_JMAX + 1], Vs[S2DW_JMAX + 1];  // Vs: roundup(bl, 8)
    long long offV[S2DW_JMAX + 1];
};
// Tile lists, ordered by decreasing work so that the longest walks start first.
int lwalk_pairs(int B, int NP);
constexpr int lwalk_slack(int S) { return S > 4 ? 64 : 0; }
bool lwalk_per_scale(int B, int NP);
int lwalk_split(const std::vector<int> &bl, int S);
void build_lwalk_tiles(const std::vector<int> &bl, int S, int jsplit, std::vector<int2> &t);
int2 mwalk_shape(int B, int NP);
int build_mwalk_intervals(const std::vector<int> &bl, const std::vector<int> &blo, int B,
                          std::vector<MwalkInterval> &iv);
void build_mwalk_tiles(const std::vector<MwalkInterval> &iv, int2 shape, std::vector<int2> &t);

// The tables G (from T = Om, kappa of the analysis) or, transposed, GT (from
// T = Gam, kappa of the synthesis), built at set_tables time.
struct GpackArgs {
    int B, Bp, NP, J, Lp;
    const double *T, *H, *kappa, *Bcoef;  // H[hpack(l, NP, q, m')], kappa[(j*B + l)*NP + q]
    double *out;
    short bl[S2DW_JMAX + 1], blo[S2DW_JMAX + 1];
};
int launch_gpack(const GpackArgs &a, bool transposed, cudaStream_t s);

// flm(l,m) = sum_j part_j(l,m) + Phi2(l) scoeff(l,m), the scale sum of
// s2dw_core_mod.f90:1228-1253 in scale order followed by :1258-1261.
struct CombineArgs {
    int B, J, bs;
    int bl[S2DW_JMAX + 1], blo[S2DW_JMAX + 1];
    long long off[S2DW_JMAX + 1];  // offset of part_j in `parts` (complex values)
    int maps;                      // map k: parts + k*pstride, scoeff + k*bs^2, flm + k*B^2
    long long pstride;
    const double2 *parts;
    const double2 *scoeff;
    const double *Phi2;
    double2 *flm;
};

// Per-scale factor tables of the split form (see SplitArgs / SplitSynArgs),
// built at set_tables time: out[((l-blo-1)*NP+q)*stride + x] = T[l*Bp+x] *
// H[hpack(l, NP, q, x)] * kappa[l*NP+q] for x <= l, x < bl; zero elsewhere.
struct GprepArgs {
    int B, Bp, NP, bl, blo, stride;
    const double *T, *H, *kappa;
    double *out;
};
struct CztArgs {
    int mode, bl, N, NP, rows;
    bool pfa;              // a prime-factor transform (czt and tw unset)
    int nq[S2DW_NPMAX];
    CztDev czt;
    TwDev tw;
    const double2 *in_c;   // complex input (Tg, Tb, V)
    const double *in_r;    // real input (wavelet coefficients)
    double2 *out_c;        // complex output (Tb, V, V2f)
    int out_stride;        // row stride of V2f (CZT_SYN_BETA)
    double *out_r;         // real output (wavelet coefficients)
    const double *wq;      // quadrature weights (2bl) for CZT_SYN_BETA
    double scale;          // (4 pi^2/N)/(2bl-1) for CZT_SYN_ALPHA
};

// One transform stage of several scales (and maps) in one launch: scale e.g.
// of a group has the CTAs from cta0 on.  Values of map k start k * in_map
// (out_map) values after the first's.
struct StageEnt {
    int cta0;
    short kind;            // CztMode, or STAGE_PFA: prime-factor alpha
    short lg;              // log2 of the transform length (not STAGE_PFA)
    int bl, rows, rows_map;  // rows: of all maps; rows_map: of one
    int out_stride;        // row stride of V2f (synthesis beta)
    const double2 *pre, *post, *Hf;
    const void *in;
    void *out;
    const double *wq;      // quadrature weights (2bl), synthesis beta
    double scale;          // (4 pi^2/N)/(2bl-1), synthesis alpha
    long long in_map, out_map;
};
constexpr int STAGE_PFA = 6;
constexpr int STAGE_MAX = 24;  // entries per launch
struct StageArgs {
    int n, ncta, N, NP;
    int nq[S2DW_NPMAX];
    const double2 *tw;     // exp(-2 pi i k / 2048), k < 2048
    const double2 *ph;     // LwalkArgs::ph
    StageEnt e[STAGE_MAX];
};
enum Stage { STAGE_ANA_BETA, STAGE_ANA_ALPHA, STAGE_SYN_ALPHA, STAGE_SYN_BETA };
// Fills kind, lg and the CTA count of an entry whose mode, bl and transform
// length M are given (pfa: prime-factor alpha stages where there are any); false
// where the stage kernels have no transform of that size (it then runs through
// launch_czt).
bool stage_plan(int mode, int bl, int M, bool pfa, int rows, StageEnt *e, int *ncta);
// Whether an alpha stage of this band limit has a prime-factor transform.
bool pfa_size(int mode, int bl);
int launch_stage(Stage st, const StageArgs &a, bool dep, cudaStream_t s);
int launch_stage_beta(Stage st, const StageArgs &a, bool dep, cudaStream_t s);
// The length-1023 alpha rows have a kernel of their own: a launch holds only
// such entries or none.
bool stage_alone(const StageEnt &e);

int launch_lwalk(const LwalkArgs &a, bool dep, cudaStream_t s);
int launch_gprep(const GprepArgs &a, cudaStream_t s);
// F[l*Bp + m] = i^{-m} Om[l*Bp + m] * flm[l + B*m] for m <= l < B, zero for m > l, and
// scoeff(0:bs-1,0:bs-1) = flm(0:bs-1,0:bs-1) (s2dw_core_mod.f90:773).
int launch_fprep(double2 *F, double2 *scoeff, const double2 *flm, const double *Om, int B, int Bp, int bs,
                 cudaStream_t s);
int launch_mwalk(const MwalkArgs &a, bool dep, cudaStream_t s);
int launch_czt(const CztArgs &a, cudaStream_t s);
// Builds, once per device, the constant tables of the length-2047 and -511
// alpha stages and the stages' twiddles
// (the current device; synchronises).  Plan creation calls it, never a capture.
int pfa_prepare();
// The current device's table exp(-2 pi i k/2048) (built by pfa_prepare).
int stage_twiddles(const double2 **tw);
void set_alpha_prefetch(bool on);  // synthesis alpha / analysis beta stages: persistent kernel with prefetched input (default on)
// scoeff (bs x bs) of `maps` maps
int launch_scoeff_copy(double2 *scoeff, const double2 *flm, int B, int bs, int maps, cudaStream_t s);
int launch_combine(const CombineArgs &a, cudaStream_t s);

// ---------------------------------------------------------------------------
// Split-precision analysis contraction (tcgen05 int8 digits, batches of maps)
// ---------------------------------------------------------------------------
// Start values below 2^S2DW_SCALE_EXP put a warp of l-walk chains in a scaled
// domain; values above 2^S2DW_RENORM_EXP there are scaled back down.
#define S2DW_SCALE_EXP (-600)
#define S2DW_RENORM_EXP 400

struct SplitArgs {
    int B, Bp, N, NP, bl, blo;
    int c0, nch, nmaps;        // first 32-row chunk of l stored in fdig, chunks, maps (<= 32)
    int nq[S2DW_NPMAX];
    const double *Acoef, *Om;  // [l*Bp + x]
    const double *Stm;         // [l0*B + k]
    const int32_t *Ste;
    const double *G;           // [((l-blo-1)*NP + q)*Gs + m'] = Om(l,m') d^l_{m'n_q} K_j(l) s(l,n_q)
    int Gs;                    // roundup(bl, 32)
    int16_t *dexp;             // [(m*bl + m')*NP + q] exponent of max_l |v|
    const int32_t *fexp;       // [m*64 + col] exponent of the map column
    const uint8_t *fdig;       // [(m*nch + chunk)*5 + digit][2048] map digits
    double2 *Tg;               // [k][g][m][m'] per map
    const double2 *ph;         // [g*16 + n+N-1] = exp(i pi n g / N)
    const int2 *tiles;         // (m, chain tile)
    int ntiles;
    int *err;                  // set to 1 when a wait gave up
    unsigned long long wait_ns;  // bound on every pipeline wait (the plan's wait limit)
};

struct FdigArgs {
    int B, bl, blo, c0, nch, nmaps;
    const double2 *flm;        // nmaps maps of B*B, flm[l + B*m]
    int32_t *fexp;
    uint8_t *fdig;
};

// Synthesis counterpart: for one m, rows are 128 chains l (m'-walk of
// d^l_{m'm}), K runs over (m', q) with MC m' and NPQ (power of two >= NP)
// values of q per 32-byte K step, columns are (map, re/im).
struct SplitSynArgs {
    int B, Bp, N, NP, bl, blo;
    int nch, nmaps;            // 32-row K chunks per m (MC m' each), maps (<= 32)
    const double *Bcoef;       // [l*Bp + m']
    const double *Em;          // [l*B + m]
    const int32_t *Ee;
    const double *G;           // [((l-blo-1)*NP + q)*Gs + m'] = Gam(l,m') d^l_{m'n_q} c_j(l,n_q)
    int Gs;                    // roundup(bl, 8)
    int16_t *sexp;             // [m*bl + l] exponent of max over (m', q) of |v|
    const int32_t *vexp;       // [m*64 + col]
    const uint8_t *vdig;       // [(m*nch + chunk)*6 + digit][2048] map digits
    double2 *part;             // map k: part + k*pstride, [(l-blo-1)*bl + m]
    long long pstride;
    const int2 *tiles;         // (m, 128-row l tile)
    int ntiles;
    int *err;
    unsigned long long wait_ns;
};

struct VdigArgs {
    int bl, NP, nch, nmaps, Vs;
    const double2 *V2f;        // map k: V2f + k*vstride, [(q*bl + m)*Vs + m']
    long long vstride;
    int32_t *vexp;
    uint8_t *vdig;
};

int split_syn_mc(int NP);       // m' per K chunk
long long split_vdig_bytes(int bl, int nch);
int launch_split_syn_dexp(const SplitSynArgs &a, cudaStream_t s);
int launch_split_vdig(const VdigArgs &a, cudaStream_t s);
int launch_split_syn(const SplitSynArgs &a, cudaStream_t s);

int split_chains(int NP);       // m' per CTA
int split_maps_per_pass();      // maps per CTA
long long split_fdig_bytes(int bl, int nch);
int launch_split_dexp(const SplitArgs &a, cudaStream_t s);
int launch_split_fdig(const FdigArgs &a, cudaStream_t s);
int launch_split(const SplitArgs &a, cudaStream_t s);

// ---------------------------------------------------------------------------
// Moments of the wavelet coefficients per scale (s2dw_stats.cu)
// ---------------------------------------------------------------------------
constexpr int STAT_W = 8;       // partial sums per block: 2 of pass 1, 6 of pass 2
// Maps per pair of passes and blocks per (map, scale) in them.  Without a mask many
// maps fill the GPU with fewer blocks and gain from fewer passes: B=256, N=4, 16
// maps 127 us with 48 blocks, 158 with 96, but 4 maps at B=512 147 and 117.
struct StatSplit {
    int maps, P;
};
__host__ __device__ constexpr StatSplit stat_split(int nmaps, bool mask)
{
    return mask ? StatSplit{16, 96} : nmaps <= 8 ? StatSplit{8, 96} : StatSplit{32, 48};
}
constexpr int STAT_BLOCKS = 16 * 96;  // the largest maps x P of them
struct StatArgs {
    int J, nmaps, P;           // at most stat_split's maps, its P
    long long wtot;            // doubles per map in the packed layout
    long long off[S2DW_JMAX + 2];  // scale offsets (J+2 entries)
    const double *wav;         // map k at wav + k*wtot
    const double *mask;        // packed layout of one map, or null
    double *part, *part2;      // nmaps*(J+1)*P x 2 and x 6 partial sums
    double *mean_nj;           // nmaps*(J+1)*2
    double *out;               // nmaps*(J+1)*6: mean, var, skew, kur, five, six
    int *flags;                // nmaps*(J+1): 1 zero variance, 2 fewer than two samples
};
int launch_stat_moments(const StatArgs &a, cudaStream_t s);

// Address on `device` (which must be current) of the static scratch array of
// s2dwc_plan_analysis_noalloc, looked up once per device.
int noalloc_scratch(int device, void **ptr);
// Drops the cached addresses (s2dwc_finalize): the next call looks them up again.
void noalloc_forget();

}  // namespace s2dw
