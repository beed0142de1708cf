// screen.cu -- learned frequency screening: phase-folded lightcurve features
// per trial frequency and the kernels of a small BF16 multilayer perceptron
// (forward, backward, Adam) that ranks trial frequencies by predicted chi^2.
//
// No counterpart in the reference, which fits every trial frequency.  The
// screen proposes a subset (top-ranked frequencies plus a random audit
// sample); the plain scan of that subset then decides, and the full scan
// stays the fallback.
//
// Features (per frequency, 88 floats): each lightcurve c is folded at the
// trial frequency f (phase = frac(t f)) into 64 phase bins of its brightness
// relative to its mean; per curve 8 statistics: the phase-dispersion ratios
// theta_B = within-bin variance / total variance for B = 64, 32, 16, 8 bins,
// and the shares H_1..H_4 of the first four harmonics in the power of the
// 32-bin mean curve; over the curves 8 aggregates of each statistic: mean
// weighted by points, plain mean, standard deviation, min, 25 %, 50 %,
// 75 % quantiles, max (features 8 * statistic + aggregate, 0..63).  Single
// nights cannot tell neighbouring grid frequencies apart (the grid step is a
// few rotations over the whole time span), so the same 8 statistics follow
// for three folds of all points together: all of them, those before the
// middle of the time span, those after it (features 64 + 8 * fold + stat).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "devmath.cuh"
#include "ps_b200.h"
#include "util.h"

namespace {

constexpr int kBins = 64;
constexpr int kStats = 8;
constexpr int kAggs = 8;
constexpr int kFeatThreads = 256;
constexpr int kFeatWarps = kFeatThreads / 32;
constexpr int kMaxScreenCurves = 256;
constexpr int kGlobalFolds = 3;
constexpr int kFeatures = kStats * kAggs + kGlobalFolds * kStats;

// Bin sums are fixed-point (2^-32 units) integers: shared-memory atomics on
// them add in any order to the same total, so the features -- and the screen's
// choice of frequencies -- are the same on every run.
constexpr double kFix = 4294967296.0;  // 2^32
constexpr int kLimb = 20;              // narrow form: a value is hi * 2^20 + lo, each sum in 32 bits

// The fixed-point brightness and squared brightness of one point: two 64-bit
// integers, or in the narrow form {lo, hi} of each.
struct PointFix {
    int4 v;
};

// cos(2 pi j / 32), passed by value.
struct Cosines {
    double c[32];
};

__device__ __forceinline__ double warp_add(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Totals of 16 values over the warp's lanes: lane l returns that of value l / 2.
// Each step halves the values a lane carries, so 16 exchanges do what 16
// butterflies of 5 would.
__device__ __forceinline__ double warp_totals(double (&v)[16])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 8, o = 16; n >= 1; n >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const double keep = up ? v[i + n] : v[i], give = up ? v[i] : v[i + n];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// The 8 statistics of one fold by one warp: lane l holds bins 2l and 2l + 1
// (count, sum, sum of squares), tw its cosines and sines of the four harmonics.
// Lane 2k gets statistic k.
__device__ __forceinline__ float fold_stats(const long long (&ci)[2], const long long (&ai)[2], const long long (&qi)[2],
                                            const double (&tw)[8])
{
    const int lane = threadIdx.x & 31;
    double c[2], a[2], q[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        c[i] = (double)ci[i];
        a[i] = (double)ai[i] * (1.0 / kFix);
        q[i] = (double)qi[i] * (1.0 / kFix);
    }
    auto within = [](double cc, double aa, double qq) { return cc > 0 ? qq - aa * (aa * psb::rcp_nr(cc)) : 0.0; };
    double v[16];  // sums within 64, 32, 16, 8 bins; real, imaginary parts; count, sum, squares
    v[0] = within(c[0], a[0], q[0]) + within(c[1], a[1], q[1]);
    double C = c[0] + c[1], A = a[0] + a[1], Q = q[0] + q[1];
    const double mean = C > 0 ? A * psb::rcp_nr(C) : 0.0;  // of the 32-bin curve; empty bins are left out
    v[1] = C > 0 ? Q - A * mean : 0.0;
    v[12] = C;
    v[13] = A;
    v[14] = Q;
    v[15] = 0.0;
#pragma unroll
    for (int lev = 2; lev < 4; ++lev) {
        const int d = 1 << (lev - 2);
        C += __shfl_xor_sync(0xffffffffu, C, d);
        A += __shfl_xor_sync(0xffffffffu, A, d);
        Q += __shfl_xor_sync(0xffffffffu, Q, d);
        v[lev] = (lane & (2 * d - 1)) == 0 ? within(C, A, Q) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) v[4 + k] = mean * tw[k];
    const double t = warp_totals(v);
    C = __shfl_sync(0xffffffffu, t, 24);
    A = __shfl_sync(0xffffffffu, t, 26);
    Q = __shfl_sync(0xffffffffu, t, 28);
    const double total = Q - (C > 0 ? A * (A * psb::rcp_nr(C)) : 0.0);
    // power of harmonic k on lanes 8 + 2k; its sum over the four
    const double im = __shfl_down_sync(0xffffffffu, t, 8);
    const double pw = t * t + im * im;
    double tot = pw + __shfl_xor_sync(0xffffffffu, pw, 2);
    tot += __shfl_xor_sync(0xffffffffu, tot, 4);
    const bool harmonic = lane >= 8;
    const double num = harmonic ? pw : t, den = harmonic ? tot : total;
    return den > 0 ? (float)(num / den) : harmonic ? 0.25f : 1.0f;
}

// One block per trial frequency; each warp folds one lightcurve at a time, lane
// l owning bins 2l and 2l + 1 of the fold's statistics.  The folds of all
// points together are the sums of the curves' folds: a curve whose points lie
// on both sides of the middle of the time span (side 2) is folded in two
// parts.  NARROW: every sum of a curve fits two 32-bit limbs, so that the
// shared-memory atomics are native 32-bit ones.
//
// What bounds it: instruction issue (about 500 warp instructions a curve, half
// of them the statistics' FP64 reductions).  5000 frequencies of the production
// object (3698 points, 42 curves): 4.19 -> 0.42 ms.
template <bool NARROW>
__global__ void __launch_bounds__(kFeatThreads, 4) features_kernel(const double *tim, const PointFix *fix,
                                                                 const int *cstart, const int *cside, int n_curves,
                                                                 const double *freqs, int n_freq, double t_mid,
                                                                 Cosines cosines, float *out)
{
    constexpr int kWords = NARROW ? 5 : 6;  // 32-bit words of one bin
    __shared__ __align__(8) unsigned bins[kFeatWarps][kWords * kBins];
    __shared__ union {
        long long halves[kFeatWarps][2][3][kBins];
        float sorted[kStats][kMaxScreenCurves];
    } sh;
    __shared__ float cst[kStats][kMaxScreenCurves];
    const int f = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double fr64 = freqs[f] * kBins;  // exact: a power of two
    unsigned *B = bins[warp];
    unsigned long long *B64 = reinterpret_cast<unsigned long long *>(B);
    auto clear = [&] {
        __syncwarp();
        for (int i = lane; i < kWords * kBins; i += 32) B[i] = 0;
        __syncwarp();
    };
    // phase bin floor(64 frac(t f)): floor(64 t f) modulo 64, by rounding down
    // at the unit bit; absurd phases (2^51 bins and more, NaN) go the long way
    auto bin_of = [&](double t) {
        const double x = __dmul_rn(t, fr64);
        int b = __double2loint(__dadd_rd(x, 6755399441055744.0)) & (kBins - 1);
        if (!(fabs(x) < 2251799813685248.0)) {
            const double ph = x / kBins, frac = ph - floor(ph);
            b = min(kBins - 1, max(0, (int)(frac * kBins)));
        }
        return b;
    };
    auto add = [&](int i) {
        const int b = bin_of(tim[i]);
        const int4 v = fix[i].v;
        if constexpr (NARROW) {
            atomicAdd(&B[b], 1u);
            atomicAdd(&B[kBins + b], (unsigned)v.x);
            atomicAdd(&B[2 * kBins + b], (unsigned)v.y);
            atomicAdd(&B[3 * kBins + b], (unsigned)v.z);
            atomicAdd(&B[4 * kBins + b], (unsigned)v.w);
        } else {
            auto u64 = [](int lo, int hi) { return (unsigned long long)(unsigned)hi << 32 | (unsigned)lo; };
            atomicAdd(&B64[b], 1ull);
            atomicAdd(&B64[kBins + b], u64(v.x, v.y));
            atomicAdd(&B64[2 * kBins + b], u64(v.z, v.w));
        }
    };
    double tw[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        tw[k] = cosines.c[((k + 1) * lane) & 31];
        tw[4 + k] = cosines.c[((k + 1) * lane + 24) & 31];  // sin x = cos(x - pi/2)
    }
    long long half[2][3][2] = {};  // [side][count, sum, squares][own bin]
    for (int c = warp; c < n_curves; c += kFeatWarps) {
        const int p0 = cstart[c], p1 = cstart[c + 1], side = cside[c];
        long long own[3][2];
        auto collect = [&](long long (&into)[3][2]) {  // the folded points' sums of this lane's bins
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int b = 2 * lane + j;
                if constexpr (NARROW) {
                    into[0][j] = B[b];
                    into[1][j] = ((long long)(int)B[2 * kBins + b] << kLimb) + B[kBins + b];
                    into[2][j] = ((long long)(int)B[4 * kBins + b] << kLimb) + B[3 * kBins + b];
                } else {
                    for (int k = 0; k < 3; ++k) into[k][j] = (long long)B64[k * kBins + b];
                }
            }
        };
        auto to_half = [&](int h, const long long (&from)[3][2]) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    half[0][k][j] += h == 0 ? from[k][j] : 0;
                    half[1][k][j] += h == 1 ? from[k][j] : 0;
                }
        };
        clear();
        if (side != 2) {
            for (int i = p0 + lane; i < p1; i += 32) add(i);
            collect(own);
            to_half(side, own);
        } else {
            long long part[3][2];
            for (int i = p0 + lane; i < p1; i += 32)
                if (tim[i] < t_mid) add(i);
            collect(part);
            to_half(0, part);
            clear();
            for (int i = p0 + lane; i < p1; i += 32)
                if (!(tim[i] < t_mid)) add(i);
            collect(own);
            to_half(1, own);
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int j = 0; j < 2; ++j) own[k][j] += part[k][j];
        }
        const float st = fold_stats(own[0], own[1], own[2], tw);
        if (lane < 2 * kStats && !(lane & 1)) cst[lane >> 1][c] = st;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            reinterpret_cast<longlong2 *>(sh.halves[warp][h][k])[lane] = make_longlong2(half[h][k][0], half[h][k][1]);
    __syncthreads();
    float *o = out + (size_t)f * kFeatures;
    if (warp < kGlobalFolds) {  // all points, the first half, the second
        long long own[3][2] = {};
        for (int w = 0; w < kFeatWarps; ++w)
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (warp == 0 || warp == 1 + h) {
                        const longlong2 v = reinterpret_cast<const longlong2 *>(sh.halves[w][h][k])[lane];
                        own[k][0] += v.x;
                        own[k][1] += v.y;
                    }
        const float st = fold_stats(own[0], own[1], own[2], tw);
        if (lane < 2 * kStats && !(lane & 1)) o[kStats * kAggs + warp * kStats + (lane >> 1)] = st;
    }
    // aggregates over the curves: warp k takes statistic k, sorted by counting
    // for every value those before it
    static_assert(kFeatWarps == kStats, "one warp per statistic");
    const float *v = cst[warp];
    __syncthreads();  // the halves have been read
    float *sv = sh.sorted[warp];
    double ws = 0, wsum = 0, s1 = 0, s2 = 0;
    for (int c = lane; c < n_curves; c += 32) {
        const float x = v[c];
        const double w = cstart[c + 1] - cstart[c];
        ws += w * x;
        wsum += w;
        s1 += x;
        s2 += (double)x * x;
        int rank = 0;
        for (int j = 0; j < n_curves; ++j) {
            const float y = v[j];
            rank += (y < x || (y == x && j < c)) ? 1 : 0;
        }
        sv[rank] = x;
    }
    ws = warp_add(ws);
    wsum = warp_add(wsum);
    s1 = warp_add(s1);
    s2 = warp_add(s2);
    __syncwarp();
    if (lane < kAggs) {
        const double mean = s1 / n_curves;
        auto quantile = [&](double fq) {
            const double pos = fq * (n_curves - 1);
            const int lo = (int)floor(pos), hi = min(lo + 1, n_curves - 1);
            return (float)(sv[lo] + (pos - lo) * (sv[hi] - sv[lo]));
        };
        float r;
        if (lane == 0)
            r = (float)(ws / wsum);
        else if (lane == 1)
            r = (float)mean;
        else if (lane == 2)
            r = (float)sqrt(fmax(s2 / n_curves - mean * mean, 0.0));
        else
            r = quantile(0.25 * (lane - 3));
        o[warp * kAggs + lane] = r;
    }
}

// ---------------------------------------------------------------- BF16 GEMM

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi)
{
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One product C[m][n] (+)= sum_k A(m, k) B(k, n) (+ bias[n]) (ReLU) (gated),
// A(m, k) = A[m sam + k sak], B(k, n) = B[k sbk + n sbn], BF16 operands on the
// tensor cores, FP32 accumulation.  gate: results where gate[m][n] <= 0 become
// zero (a ReLU's backward pass).
struct Gemm {
    int M, N, K;
    const __nv_bfloat16 *A, *B;
    long sam, sak, sbk, sbn;
    float *C;
    int ldc, accumulate;
    const float *bias;
    int relu;
    const float *gate;
    int ldg;
    __nv_bfloat16 *Cb;
    int ldcb;
    int a_vec, b_vec;    // 16-byte loads along the contiguous direction are aligned
    int form, tiles_n, tiles;  // filled by the launch
};

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __nv_bfloat16 *p, bool trans)
{
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    if (trans)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(a));
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(a));
}

// Eight operand elements along `in` (stride s_in) at outer index `out` (stride
// s_out), zeros outside n_in x n_out.
__device__ __forceinline__ uint4 load8(const __nv_bfloat16 *base, long s_in, long s_out, int in, int out, int n_in,
                                       int n_out, bool vec)
{
    if (out < n_out && vec && in + 8 <= n_in)
        return *reinterpret_cast<const uint4 *>(base + (long)out * s_out + in);
    __nv_bfloat16 v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e)
        v[e] = (out < n_out && in + e < n_in) ? base[(long)out * s_out + (long)(in + e) * s_in] : __float2bfloat16(0.0f);
    uint4 r;
    r.x = pack_bf16(v[0], v[1]);
    r.y = pack_bf16(v[2], v[3]);
    r.z = pack_bf16(v[4], v[5]);
    r.w = pack_bf16(v[6], v[7]);
    return r;
}

constexpr int kGemmThreads = 256;
constexpr int kGemmSmem = 32768;  // partial sums; the operand stages take less

// One BM x BN tile by 8 warps: a warp computes a WM x WN block over every KS-th
// k-step of 16; with KS > 1 the partial sums meet in shared memory.  Stages of
// BK along k: global loads of the next stage are in flight under this one's
// MMAs.  An operand lies in shared memory as it does in global memory
// (contiguous along k, or transposed: AT, BT) and ldmatrix turns it.
//
// The network's products are small (256 x 256 x a few thousand): what bounds
// them is latency, not the tensor cores, so tiles are small enough to give the
// SMs one each, and where k is long and the tiles few it is split over the
// warps (tcgen05 tiles of 128 rows would leave most SMs idle).  Elsewhere each
// result is one chain of k-steps: a split would round hidden activations to
// other BF16 values.
// Measured cold, 256-wide layers: 5000 rows forward 42 -> 18 us; batch 1024, a
// weight gradient and the gradient below it 55 + 15 -> 15 us.
template <int BM, int BN, int BK, int WM, int WN, int KS, bool AT, bool BT>
__device__ __forceinline__ void gemm_tile(const Gemm &g, int m0, int n0, unsigned char *smem)
{
    static_assert((BM / WM) * (BN / WN) * KS * 32 == kGemmThreads, "8 warps");
    constexpr int SA = AT ? BM + 8 : BK + 8, SB = BT ? BN + 8 : BK + 8;  // padded rows: no ldmatrix conflicts
    constexpr int VA = BM * BK / 8 / kGemmThreads, VB = BN * BK / 8 / kGemmThreads;
    static_assert(((AT ? BK * SA : BM * SA) + (BT ? BK * SB : BN * SB)) * 2 <= kGemmSmem, "stage");
    static_assert(KS * BM * BN * 4 <= kGemmSmem, "partial sums");
    __nv_bfloat16 *As = reinterpret_cast<__nv_bfloat16 *>(smem), *Bs = As + (AT ? BK * SA : BM * SA);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ks = warp % KS, block = warp / KS;
    const int wm = WM * (block / (BN / WN)), wn = WN * (block % (BN / WN));
    uint4 ra[VA], rb[VB];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int v = 0; v < VA; ++v) {
            const int i = tid + v * kGemmThreads;
            if constexpr (AT)
                ra[v] = load8(g.A, 1, g.sak, m0 + i % (BM / 8) * 8, k0 + i / (BM / 8), g.M, g.K, g.a_vec);
            else
                ra[v] = load8(g.A, g.sak, g.sam, k0 + i % (BK / 8) * 8, m0 + i / (BK / 8), g.K, g.M, g.a_vec);
        }
#pragma unroll
        for (int v = 0; v < VB; ++v) {
            const int i = tid + v * kGemmThreads;
            if constexpr (BT)
                rb[v] = load8(g.B, 1, g.sbk, n0 + i % (BN / 8) * 8, k0 + i / (BN / 8), g.N, g.K, g.b_vec);
            else
                rb[v] = load8(g.B, g.sbk, g.sbn, k0 + i % (BK / 8) * 8, n0 + i / (BK / 8), g.K, g.N, g.b_vec);
        }
    };
    float acc[WM / 16][WN / 8][4];
#pragma unroll
    for (int i = 0; i < WM / 16; ++i)
#pragma unroll
        for (int j = 0; j < WN / 8; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0f;
    fetch(0);
    for (int k0 = 0; k0 < g.K; k0 += BK) {
        __syncthreads();  // the previous stage has been read
#pragma unroll
        for (int v = 0; v < VA; ++v) {
            const int i = tid + v * kGemmThreads;
            constexpr int W = AT ? BM / 8 : BK / 8;
            *reinterpret_cast<uint4 *>(As + i / W * SA + i % W * 8) = ra[v];
        }
#pragma unroll
        for (int v = 0; v < VB; ++v) {
            const int i = tid + v * kGemmThreads;
            constexpr int W = BT ? BN / 8 : BK / 8;
            *reinterpret_cast<uint4 *>(Bs + i / W * SB + i % W * 8) = rb[v];
        }
        __syncthreads();
        if (k0 + BK < g.K) fetch(k0 + BK);
        const int j = lane >> 3, r = lane & 7;
#pragma unroll
        for (int kk = 0; kk < BK / 16 / KS; ++kk) {
            const int k = 16 * (kk * KS + ks);
            if (k0 + k >= g.K) break;  // zeros from here on
            uint32_t a[WM / 16][4], b[WN / 16][4];
#pragma unroll
            for (int i = 0; i < WM / 16; ++i) {
                const int m = wm + 16 * i;
                ldmatrix4(a[i], AT ? As + (k + (j >> 1) * 8 + r) * SA + m + (j & 1) * 8
                                   : As + (m + (j & 1) * 8 + r) * SA + k + (j >> 1) * 8, AT);
            }
#pragma unroll
            for (int i = 0; i < WN / 16; ++i) {
                const int n = wn + 16 * i;
                ldmatrix4(b[i], BT ? Bs + (k + (j & 1) * 8 + r) * SB + n + (j >> 1) * 8
                                   : Bs + (n + (j >> 1) * 8 + r) * SB + k + (j & 1) * 8, BT);
            }
#pragma unroll
            for (int i = 0; i < WM / 16; ++i)
#pragma unroll
                for (int jn = 0; jn < WN / 8; ++jn)
                    mma_bf16(acc[i][jn], a[i], b[jn >> 1][2 * (jn & 1)], b[jn >> 1][2 * (jn & 1) + 1]);
        }
    }
    __syncthreads();
    float *red = reinterpret_cast<float *>(smem) + ks * BM * BN;
#pragma unroll
    for (int i = 0; i < WM / 16; ++i)
#pragma unroll
        for (int jn = 0; jn < WN / 8; ++jn)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float2 *>(red + (wm + 16 * i + 8 * h + (lane >> 2)) * BN + wn + 8 * jn + 2 * (lane & 3)) =
                    make_float2(acc[i][jn][2 * h], acc[i][jn][2 * h + 1]);
    __syncthreads();
    const float *sum = reinterpret_cast<const float *>(smem);
#pragma unroll
    for (int e = 0; e < BM * BN / kGemmThreads; ++e) {
        const int i = tid + e * kGemmThreads, m = m0 + i / BN, n = n0 + i % BN;
        if (m >= g.M || n >= g.N) continue;
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < KS; ++w) v += sum[w * BM * BN + i];
        if (g.accumulate) v += g.C[(long)m * g.ldc + n];
        if (g.bias) v += g.bias[n];
        if (g.relu) v = fmaxf(v, 0.0f);
        if (g.gate && !(g.gate[(long)m * g.ldg + n] > 0.0f)) v = 0.0f;
        if (g.C) g.C[(long)m * g.ldc + n] = v;
        if (g.Cb) g.Cb[(long)m * g.ldcb + n] = __float2bfloat16(v);
    }
    __syncthreads();
}

// Up to two independent products in one launch.
struct GemmPair {
    Gemm g[2];
};

// The forms of a product's tiles.
enum { kForm64, kForm32, kFormSplit };
constexpr int kFormBM[3] = {64, 32, 32}, kFormBN[3] = {64, 64, 32};

template <bool AT, bool BT>
__device__ __forceinline__ void gemm_form(const Gemm &g, int t, unsigned char *smem)
{
    if (g.form == kForm64)
        gemm_tile<64, 64, 64, 16, 32, 1, AT, BT>(g, t / g.tiles_n * 64, t % g.tiles_n * 64, smem);
    else if (g.form == kForm32)
        gemm_tile<32, 64, 64, 16, 16, 1, AT, BT>(g, t / g.tiles_n * 32, t % g.tiles_n * 64, smem);
    else
        gemm_tile<32, 32, 128, 32, 32, 8, AT, BT>(g, t / g.tiles_n * 32, t % g.tiles_n * 32, smem);
}

__global__ void __launch_bounds__(kGemmThreads) gemm_bf16_kernel(const GemmPair pair)
{
    __shared__ __align__(16) unsigned char smem[kGemmSmem];
    const int second = (int)blockIdx.x >= pair.g[0].tiles;
    const Gemm &g = pair.g[second];
    const int t = blockIdx.x - (second ? pair.g[0].tiles : 0);
    const bool at = g.sak != 1 && g.sam == 1, bt = g.sbk != 1 && g.sbn == 1;
    if (at && bt)
        gemm_form<true, true>(g, t, smem);
    else if (at)
        gemm_form<true, false>(g, t, smem);
    else if (bt)
        gemm_form<false, true>(g, t, smem);
    else
        gemm_form<false, false>(g, t, smem);
}

// Launches one product, or two independent ones (b).  A product takes 64 x 64
// tiles where they give every SM one (they read half as much per result), else
// 32 x 64 -- and 32 x 32 with k split over the warps where k is 512 or more:
// below that the chain of k-steps is as short as the split's own reduction.
cudaError_t launch_gemm(Gemm a, const Gemm *b, cudaStream_t s)
{
    GemmPair p{};
    p.g[0] = a;
    if (b) p.g[1] = *b;
    long tiles = 0;
    for (int i = 0; i < (b ? 2 : 1); ++i) {
        Gemm &g = p.g[i];
        auto count = [&](int f) {
            return (long)((g.M + kFormBM[f] - 1) / kFormBM[f]) * ((g.N + kFormBN[f] - 1) / kFormBN[f]);
        };
        g.form = count(kForm64) >= 148 ? kForm64 : g.K >= 512 ? kFormSplit : kForm32;
        g.tiles_n = (g.N + kFormBN[g.form] - 1) / kFormBN[g.form];
        g.tiles = (int)count(g.form);
        tiles += g.tiles;
        // the contiguous direction's 16-byte loads: base and outer stride
        const bool at = g.sak != 1 && g.sam == 1, bt = g.sbk != 1 && g.sbn == 1;
        const long ao = at ? g.sak : g.sam, bo = bt ? g.sbk : g.sbn;
        g.a_vec = (at || g.sak == 1) && (uintptr_t)g.A % 16 == 0 && ao % 8 == 0;
        g.b_vec = (bt || g.sbk == 1) && (uintptr_t)g.B % 16 == 0 && bo % 8 == 0;
    }
    if (tiles == 0) return cudaSuccess;
    gemm_bf16_kernel<<<(unsigned)tiles, kGemmThreads, 0, s>>>(p);
    return cudaGetLastError();
}

Gemm make_gemm(int M, int N, int K, const void *A, long sam, long sak, const void *B, long sbk, long sbn, float *C,
               int ldc, const float *bias, int relu, void *Cb, int ldcb)
{
    Gemm g{};
    g.M = M;
    g.N = N;
    g.K = K;
    g.A = (const __nv_bfloat16 *)A;
    g.B = (const __nv_bfloat16 *)B;
    g.sam = sam;
    g.sak = sak;
    g.sbk = sbk;
    g.sbn = sbn;
    g.C = C;
    g.ldc = ldc;
    g.bias = bias;
    g.relu = relu;
    g.Cb = (__nv_bfloat16 *)Cb;
    g.ldcb = ldcb;
    return g;
}

// ---------------------------------------------------------------- network, forward

// All layers of a network in one launch: a CTA takes 16 MB rows through every
// layer, their activations in shared memory (and in global memory for the
// backward pass), the weights streaming past in stages of 64 k's that are
// fetched kFwdStages - 1 ahead, over the layers' borders.  Warp w computes
// columns 16 w .. 16 w + 15.  Every result is the same chain of k-steps, bias
// and rounding as the layers' single products, so the bits are theirs.
//
// What bounds it: a layer alone is latency (launch, one tile's loads, 16
// dependent k-steps), 6 to 13 us for 0.1 to 1 us of tensor work; here the loads
// run ahead of it and what remains is reading the weights once per CTA from L2.
// 16 warps a CTA, since two a scheduler left the copies' latency bare (8 warps of
// 32 columns: 37 us instead of 29 at 5000 rows).
// MB is the smallest that gives each SM one CTA: 1024 rows take 18 us in CTAs of
// 16, 25 of 32 and 29 of 48; 3000 rows 33 us of 16 (two waves), 25 of 32.
// Measured (88-256-256-256-1), layer by layer -> here: 1024 rows 34 -> 18 us,
// 5000 rows 60 -> 29 us, 65536 rows 335 -> 215 us.
constexpr int kFwdThreads = 512, kFwdWidth = 256, kFwdLayers = 8, kFwdStages = 3, kFwdK = 64, kFwdMaxMB = 4;
constexpr int kFwdSW = kFwdK + 8, kFwdSA = kFwdWidth + 8;  // padded rows: no ldmatrix conflicts
static_assert(kFwdThreads / 32 * 16 == kFwdWidth, "16 columns a warp");

struct MlpForward {
    struct {
        int k, n;
        const __nv_bfloat16 *w;  // [n][k]
        const float *bias;
        float *hf;               // [rows][n] FP32 results, or null
        __nv_bfloat16 *hb;       // the same in BF16, or null (the last layer)
    } l[kFwdLayers];
    int n_layers, rows;
    const __nv_bfloat16 *x;
};

constexpr size_t forward_smem(int mb)
{
    return sizeof(__nv_bfloat16) * ((size_t)kFwdStages * kFwdWidth * kFwdSW + 2 * 16 * (size_t)mb * kFwdSA);
}

__device__ __forceinline__ void copy16_async(void *dst, const void *src, bool ok)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

template <int MB>
__global__ void __launch_bounds__(kFwdThreads) mlp_forward_kernel(const MlpForward net)
{
    extern __shared__ __align__(16) __nv_bfloat16 fwd_smem[];
    __nv_bfloat16 *const act = fwd_smem + kFwdStages * kFwdWidth * kFwdSW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = blockIdx.x * 16 * MB;

    // the next stage of weights: rows n, columns k0 .. k0 + 63 of its layer,
    // zeros outside; a thread copies 16 bytes of every kRowStep-th row
    constexpr int kRowStep = kFwdThreads / (kFwdK / 8);
    const int pn = tid / (kFwdK / 8), pc = tid % (kFwdK / 8) * 8;
    int pl = 0, pk = 0, pstage = 0, lk = net.l[0].k, ln = net.l[0].n;
    const __nv_bfloat16 *lw = net.l[0].w, *src = lw + (size_t)pn * lk + pc;
    auto prefetch = [&] {
        if (pl < net.n_layers) {
            __nv_bfloat16 *dst = fwd_smem + (pstage * kFwdWidth + pn) * kFwdSW + pc;
            const bool k_in = pk + pc < lk;
            const size_t step = (size_t)kRowStep * lk;
#pragma unroll
            for (int u = 0; u < kFwdWidth / kRowStep; ++u) {
                const bool ok = k_in && pn + u * kRowStep < ln;
                if (u * kRowStep < ln) copy16_async(dst + u * kRowStep * kFwdSW, ok ? src + u * step : lw, ok);
            }
            pstage = pstage + 1 == kFwdStages ? 0 : pstage + 1;
            pk += kFwdK;
            src += kFwdK;
            if (pk >= lk) {
                pk = 0;
                if (++pl < net.n_layers) {
                    lk = net.l[pl].k;
                    ln = net.l[pl].n;
                    lw = net.l[pl].w;
                    src = lw + (size_t)pn * lk + pc;
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the input rows, zeros outside
    {
        const int k = net.l[0].k, chunks = ((k + 15) & ~15) / 8;
        for (int i = tid; i < 16 * MB * chunks; i += kFwdThreads) {
            const int r = i / chunks, c = i % chunks * 8;
            const bool ok = row0 + r < net.rows && c < k;
            copy16_async(act + r * kFwdSA + c, ok ? net.x + (size_t)(row0 + r) * k + c : net.x, ok);
        }
    }
#pragma unroll
    for (int i = 0; i < kFwdStages - 1; ++i) prefetch();  // the first group holds the input too

    int stage = 0;
    for (int l = 0; l < net.n_layers; ++l) {
        const auto &y = net.l[l];
        const int K = y.k, N = y.n;
        const __nv_bfloat16 *in = act + (l & 1) * 16 * MB * kFwdSA;
        const bool active = 16 * warp < N;
        float acc[MB][2][4];
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
            for (int n = 0; n < 2; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.0f;
        for (int k0 = 0; k0 < K; k0 += kFwdK) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kFwdStages - 2) : "memory");
            __syncthreads();  // this stage has landed, the stage before and the last layer's rows are done
            prefetch();
            const int j = lane >> 3, r = lane & 7;
            const __nv_bfloat16 *wb = fwd_smem + (stage * kFwdWidth + 16 * warp + (j >> 1) * 8 + r) * kFwdSW + (j & 1) * 8;
            const __nv_bfloat16 *ab = in + ((j & 1) * 8 + r) * kFwdSA + k0 + (j >> 1) * 8;
            stage = stage + 1 == kFwdStages ? 0 : stage + 1;
            if (!active) continue;
            // two k-steps' fragments, then their MMAs
            uint32_t a[2][MB][4], b[2][4];
#pragma unroll
            for (int kk = 0; kk < kFwdK; kk += 32) {
                if (k0 + kk >= K) break;
                const bool both = k0 + kk + 16 < K;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (q && !both) break;
                    ldmatrix4(b[q], wb + kk + 16 * q, false);
#pragma unroll
                    for (int m = 0; m < MB; ++m) ldmatrix4(a[q][m], ab + 16 * m * kFwdSA + kk + 16 * q, false);
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (q && !both) break;
#pragma unroll
                    for (int m = 0; m < MB; ++m)
#pragma unroll
                        for (int n = 0; n < 2; ++n) mma_bf16(acc[m][n], a[q][m], b[q][2 * n], b[q][2 * n + 1]);
                }
            }
        }
        if (!active) continue;
        const bool last = l == net.n_layers - 1;
        __nv_bfloat16 *out = act + ((l + 1) & 1) * 16 * MB * kFwdSA;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int c = 16 * warp + 8 * n + 2 * (lane & 3);
            const bool in0 = c < N, in1 = c + 1 < N, pair = in1 && !(N & 1);
            const float b0 = y.bias && in0 ? y.bias[c] : 0.0f, b1 = y.bias && in1 ? y.bias[c + 1] : 0.0f;
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = 16 * m + 8 * h + (lane >> 2);
                    float v0 = 0.0f + acc[m][n][2 * h], v1 = 0.0f + acc[m][n][2 * h + 1];
                    if (y.bias) {
                        v0 += b0;
                        v1 += b1;
                    }
                    if (!last) {
                        v0 = fmaxf(v0, 0.0f);
                        v1 = fmaxf(v1, 0.0f);
                    }
                    const __nv_bfloat162 hv = __halves2bfloat162(__float2bfloat16(v0), __float2bfloat16(v1));
                    if (!last) *reinterpret_cast<__nv_bfloat162 *>(out + r * kFwdSA + c) = hv;
                    if (row0 + r >= net.rows) continue;
                    const size_t at = (size_t)(row0 + r) * N + c;
                    if (pair) {
                        if (y.hf) *reinterpret_cast<float2 *>(y.hf + at) = make_float2(v0, v1);
                        if (y.hb) *reinterpret_cast<__nv_bfloat162 *>(y.hb + at) = hv;
                    } else if (in0) {  // an odd width, which only the last layer has
                        if (y.hf) y.hf[at] = v0;
                        if (y.hf && in1) y.hf[at + 1] = v1;
                    }
                }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <int MB>
cudaError_t launch_forward(const MlpForward &net, cudaStream_t s)
{
    const cudaError_t e = cudaFuncSetAttribute(mlp_forward_kernel<MB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)forward_smem(MB));
    if (e != cudaSuccess) return e;
    mlp_forward_kernel<MB><<<(net.rows + 16 * MB - 1) / (16 * MB), kFwdThreads, forward_smem(MB), s>>>(net);
    return cudaGetLastError();
}

// Whether the one-launch forward pass takes these layers: widths within its
// tile, weights and input readable in 16-byte pieces, FP32 pairs aligned.  Any
// other network goes layer by layer.
bool forward_fits(int n_layers, const int32_t *sizes, const void *const *w, void *const *h, float *const *hf)
{
    if (n_layers > kFwdLayers) return false;
    for (int l = 0; l < n_layers; ++l) {
        const uintptr_t ptrs = (uintptr_t)w[l] | (uintptr_t)h[l];
        if (sizes[l] > kFwdWidth || sizes[l + 1] > kFwdWidth || sizes[l] % 8 || ptrs % 16 || (uintptr_t)hf[l] % 8) return false;
    }
    return true;
}

// dZ = dH * (Z > 0), as BF16 (the next backward GEMM's operand) and FP32.
__global__ void relu_backward_kernel(long n, const float *dh, const float *z, float *dz, __nv_bfloat16 *dzb)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = z[i] > 0.0f ? dh[i] : 0.0f;
    if (dz) dz[i] = v;
    if (dzb) dzb[i] = __float2bfloat16(v);
}

// db[n] = sum over rows of dZ[r][n] for several matrices: blocks of 32 columns,
// 32 threads a column taking every 32nd row, their sums added in order.  (One
// thread a column was 60 us for 1024 x 256: a serial chain of loads.)
struct ColumnSums {
    struct {
        int rows, cols, first;  // first: block where the matrix starts
        const float *x;
        float *out;
    } m[16];
    int n;
};

__global__ void __launch_bounds__(1024) column_sum_kernel(const ColumnSums a)
{
    __shared__ float part[32][33];
    int i = 0;
    while (i + 1 < a.n && (int)blockIdx.x >= a.m[i + 1].first) ++i;
    const auto &m = a.m[i];
    const int c = threadIdx.x & 31, r0 = threadIdx.x >> 5;
    const int n = (blockIdx.x - m.first) * 32 + c;
    float s = 0.0f;
    if (n < m.cols)
#pragma unroll 8
        for (int r = r0; r < m.rows; r += 32) s += m.x[(long)r * m.cols + n];
    part[r0][c] = s;
    __syncthreads();
    if (r0 == 0 && n < m.cols) {
        float t = 0.0f;
#pragma unroll
        for (int k = 0; k < 32; ++k) t += part[k][c];
        m.out[n] = t;
    }
}

// Adam on FP32 master weights, then the BF16 working copy.
struct AdamTensors {
    struct {
        long n;
        int first;  // block where the tensor starts
        float *w, *m, *v;
        const float *grad;
        __nv_bfloat16 *wb;
    } t[32];
    int count;
};

__global__ void __launch_bounds__(256) adam_kernel(const AdamTensors a, float lr, float b1, float b2, float eps, float c1,
                                                   float c2)
{
    int k = 0;
    while (k + 1 < a.count && (int)blockIdx.x >= a.t[k + 1].first) ++k;
    const auto &t = a.t[k];
    const long i = (long)(blockIdx.x - t.first) * 256 + threadIdx.x;
    if (i >= t.n) return;
    const float gr = t.grad[i];
    const float mi = b1 * t.m[i] + (1.0f - b1) * gr;
    const float vi = b2 * t.v[i] + (1.0f - b2) * gr * gr;
    t.m[i] = mi;
    t.v[i] = vi;
    const float wi = t.w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    t.w[i] = wi;
    if (t.wb) t.wb[i] = __float2bfloat16(wi);
}

__global__ void to_bf16_kernel(long n, const float *x, __nv_bfloat16 *y)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16(x[i]);
}

inline unsigned blocks_for(long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

#define SC_CUDA(call)                                          \
    do {                                                       \
        cudaError_t e_ = (call);                               \
        if (e_ != cudaSuccess) return psb_fail_cuda(e_, #call); \
    } while (0)

extern "C" ps_status ps_screen_features(int32_t device, int32_t n_points, const double *tim,
                                        const double *brightness, const ps_curves *curves, int32_t n_freq,
                                        const double *freqs, float *features)
{
    if (n_points <= 0 || !tim || !brightness || !curves || !curves->curve_len || n_freq < 0 ||
        (n_freq > 0 && (!freqs || !features)))
        return psb_fail(PS_ERR_ARG, "ps_screen_features: null argument or n_points <= 0");
    const int nc = curves->n_curves;
    if (nc < 1 || nc > kMaxScreenCurves) return psb_fail(PS_ERR_ARG, "ps_screen_features: 1..256 lightcurves");
    if (n_freq == 0) return PS_OK;
    std::vector<int> cstart(nc + 1);
    std::vector<float> y(n_points);
    int q = 0;
    for (int c = 0; c < nc; ++c) {
        const int len = curves->curve_len[c];
        if (len < 1) return psb_fail(PS_ERR_ARG, "ps_screen_features: empty lightcurve");
        cstart[c] = q;
        if (q + len > n_points) return psb_fail(PS_ERR_ARG, "ps_screen_features: curve lengths exceed n_points");
        double mean = 0;
        for (int i = 0; i < len; ++i) mean += brightness[q + i];
        mean /= len;
        for (int i = 0; i < len; ++i) y[q + i] = (float)(mean != 0 ? brightness[q + i] / mean - 1.0 : 0.0);
        q += len;
    }
    cstart[nc] = q;
    if (q != n_points) return psb_fail(PS_ERR_ARG, "ps_screen_features: curve lengths do not sum to n_points");
    double t_lo = tim[0], t_hi = tim[0];
    for (int i = 1; i < n_points; ++i) {
        t_lo = fmin(t_lo, tim[i]);
        t_hi = fmax(t_hi, tim[i]);
    }
    const double t_mid = 0.5 * (t_lo + t_hi);
    // fixed-point values once per point (not once per point and frequency)
    auto to_fix = [](double x) -> long long {
        x *= kFix;
        if (!(x > -9.2e18)) return LLONG_MIN;  // NaN too, as the device's conversion
        return x < 9.2e18 ? std::llrint(x) : LLONG_MAX;
    };
    std::vector<long long> fix(2 * (size_t)n_points);
    double longest = 0, largest = 0;
    for (int c = 0; c < nc; ++c) longest = std::max(longest, (double)(cstart[c + 1] - cstart[c]));
    for (int i = 0; i < n_points; ++i) {
        fix[2 * i] = to_fix(y[i]);
        fix[2 * i + 1] = to_fix((double)y[i] * (double)y[i]);
        largest = std::max({largest, std::fabs((double)fix[2 * i]), std::fabs((double)fix[2 * i + 1])});
    }
    // the limbs' sums over a curve fit 32 bits: 20 low bits of every point, and
    // what lies above them
    const double limb = (double)(1 << kLimb);
    const bool narrow = longest * limb < 4294967296.0 && longest * (largest / limb + 1.0) < 2147483648.0;
    // one buffer: times, fixed-point values, frequencies, curve starts and
    // sides, then the features
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = (off + bytes + 15) & ~size_t(15);
        return o;
    };
    const size_t o_tim = take(sizeof(double) * n_points), o_fix = take(sizeof(PointFix) * n_points);
    const size_t o_freq = take(sizeof(double) * n_freq), o_cs = take(sizeof(int) * (nc + 1)), o_side = take(sizeof(int) * nc);
    const size_t in_bytes = off, o_out = take(sizeof(float) * (size_t)n_freq * kFeatures);
    std::vector<unsigned char> host(in_bytes);
    std::memcpy(&host[o_tim], tim, sizeof(double) * n_points);
    PointFix *hf = reinterpret_cast<PointFix *>(&host[o_fix]);
    for (int i = 0; i < n_points; ++i) {
        const long long v[2] = {fix[2 * i], fix[2 * i + 1]};
        int w[4];
        for (int k = 0; k < 2; ++k) {
            w[2 * k] = narrow ? (int)(v[k] & ((1 << kLimb) - 1)) : (int)(unsigned)(unsigned long long)v[k];
            w[2 * k + 1] = narrow ? (int)(v[k] >> kLimb) : (int)(v[k] >> 32);
        }
        hf[i].v = make_int4(w[0], w[1], w[2], w[3]);
    }
    std::memcpy(&host[o_freq], freqs, sizeof(double) * n_freq);
    std::memcpy(&host[o_cs], cstart.data(), sizeof(int) * (nc + 1));
    int *side = reinterpret_cast<int *>(&host[o_side]);
    for (int c = 0; c < nc; ++c) {
        int before = 0;
        for (int i = cstart[c]; i < cstart[c + 1]; ++i) before += tim[i] < t_mid ? 1 : 0;
        side[c] = before == cstart[c + 1] - cstart[c] ? 0 : before == 0 ? 1 : 2;
    }
    Cosines cosines;
    for (int j = 0; j < 32; ++j) cosines.c[j] = j % 8 == 0 ? (j == 0 ? 1.0 : j == 16 ? -1.0 : 0.0)
                                                         : std::cos(2.0 * 3.14159265358979323846 * j / 32.0);
    SC_CUDA(cudaSetDevice(device));
    unsigned char *d = nullptr;
    cudaError_t e = (cudaError_t)psb_pool_alloc(device, (void **)&d, off, nullptr);
    if (e == cudaSuccess) e = cudaMemcpy(d, host.data(), in_bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        auto *k = narrow ? features_kernel<true> : features_kernel<false>;
        k<<<n_freq, kFeatThreads>>>((const double *)(d + o_tim), (const PointFix *)(d + o_fix), (const int *)(d + o_cs),
                                    (const int *)(d + o_side), nc, (const double *)(d + o_freq), n_freq, t_mid,
                                    cosines, (float *)(d + o_out));
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpy(features, d + o_out, sizeof(float) * (size_t)n_freq * kFeatures, cudaMemcpyDeviceToHost);
    psb_pool_free(d, nullptr);
    if (e != cudaSuccess) return psb_fail_cuda(e, "ps_screen_features");
    return PS_OK;
}

extern "C" ps_status ps_gemm_bf16(int32_t M, int32_t N, int32_t K, const void *A, int64_t sam, int64_t sak,
                                  const void *B, int64_t sbk, int64_t sbn, float *C, int32_t ldc, int32_t accumulate,
                                  const float *bias, int32_t relu, void *Cb, int32_t ldcb, void *stream)
{
    if (M < 0 || N < 0 || K < 0 || !A || !B || (!C && !Cb) || (accumulate && !C))
        return psb_fail(PS_ERR_ARG, "ps_gemm_bf16: bad arguments");
    if (M == 0 || N == 0) return PS_OK;
    Gemm g = make_gemm(M, N, K, A, sam, sak, B, sbk, sbn, C, ldc, bias, relu, Cb, ldcb);
    g.accumulate = accumulate;
    SC_CUDA(launch_gemm(g, nullptr, (cudaStream_t)stream));
    return PS_OK;
}

extern "C" ps_status ps_relu_backward(int64_t n, const float *dh, const float *z, float *dz, void *dzb, void *stream)
{
    if (n < 0 || !dh || !z || (!dz && !dzb)) return psb_fail(PS_ERR_ARG, "ps_relu_backward: bad arguments");
    if (n == 0) return PS_OK;
    relu_backward_kernel<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(n, dh, z, dz, (__nv_bfloat16 *)dzb);
    SC_CUDA(cudaGetLastError());
    return PS_OK;
}

extern "C" ps_status ps_column_sum(int32_t rows, int32_t cols, const float *x, float *out, void *stream)
{
    if (rows < 0 || cols < 0 || !x || !out) return psb_fail(PS_ERR_ARG, "ps_column_sum: bad arguments");
    if (cols == 0) return PS_OK;
    ColumnSums a{};
    a.n = 1;
    a.m[0] = {rows, cols, 0, x, out};
    column_sum_kernel<<<blocks_for(cols, 32), 1024, 0, (cudaStream_t)stream>>>(a);
    SC_CUDA(cudaGetLastError());
    return PS_OK;
}

extern "C" ps_status ps_adam_step(int64_t n, float *w, const float *grad, float *m, float *v, float lr, float beta1,
                                  float beta2, float eps, int32_t step, void *wb, void *stream)
{
    if (n < 0 || !w || !grad || !m || !v || step < 1) return psb_fail(PS_ERR_ARG, "ps_adam_step: bad arguments");
    if (n == 0) return PS_OK;
    const int64_t sizes[1] = {n};
    float *ws[1] = {w}, *ms[1] = {m}, *vs[1] = {v};
    const float *gs[1] = {grad};
    void *wbs[1] = {wb};
    return ps_adam_steps(1, sizes, ws, gs, ms, vs, wbs, lr, beta1, beta2, eps, step, stream);
}

extern "C" ps_status ps_adam_steps(int32_t count, const int64_t *n, float *const *w, const float *const *grad,
                                   float *const *m, float *const *v, void *const *wb, float lr, float beta1,
                                   float beta2, float eps, int32_t step, void *stream)
{
    if (count < 0 || count > 32 || (count > 0 && (!n || !w || !grad || !m || !v || !wb)) || step < 1)
        return psb_fail(PS_ERR_ARG, "ps_adam_steps: bad arguments (at most 32 tensors)");
    AdamTensors a{};
    long blocks = 0;
    for (int i = 0; i < count; ++i) {
        if (n[i] < 0 || (n[i] > 0 && (!w[i] || !grad[i] || !m[i] || !v[i])))
            return psb_fail(PS_ERR_ARG, "ps_adam_steps: bad arguments (null tensor)");
        if (n[i] == 0) continue;
        auto &t = a.t[a.count++];
        t.n = n[i];
        t.first = (int)blocks;
        t.w = w[i];
        t.grad = grad[i];
        t.m = m[i];
        t.v = v[i];
        t.wb = (__nv_bfloat16 *)wb[i];
        blocks += blocks_for(n[i], 256);
    }
    if (blocks == 0) return PS_OK;
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    adam_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(a, lr, beta1, beta2, eps, c1, c2);
    SC_CUDA(cudaGetLastError());
    return PS_OK;
}

extern "C" ps_status ps_mlp_forward(int32_t n_layers, const int32_t *sizes, int32_t rows, const void *const *w,
                                    const float *const *bias, void *const *h, float *const *hf, void *stream)
{
    if (n_layers < 1 || !sizes || rows < 0 || !w || !bias || !h || !hf)
        return psb_fail(PS_ERR_ARG, "ps_mlp_forward: bad arguments");
    for (int l = 0; l < n_layers; ++l) {
        const bool last = l == n_layers - 1;
        if (sizes[l] < 1 || sizes[l + 1] < 1 || !w[l] || !h[l] || (!last && !h[l + 1]) || (last && !hf[l]))
            return psb_fail(PS_ERR_ARG, "ps_mlp_forward: bad layer");
    }
    if (rows == 0) return PS_OK;
    if (forward_fits(n_layers, sizes, w, h, hf)) {
        MlpForward net{};
        net.n_layers = n_layers;
        net.rows = rows;
        net.x = (const __nv_bfloat16 *)h[0];
        for (int l = 0; l < n_layers; ++l)
            net.l[l] = {sizes[l], sizes[l + 1], (const __nv_bfloat16 *)w[l], bias[l], hf[l],
                        l == n_layers - 1 ? nullptr : (__nv_bfloat16 *)h[l + 1]};
        const long blocks = ((long)rows + 15) / 16;
        const int mb = (int)std::min<long>(kFwdMaxMB, (blocks + 147) / 148);
        SC_CUDA(mb == 1   ? launch_forward<1>(net, (cudaStream_t)stream)
                : mb == 2 ? launch_forward<2>(net, (cudaStream_t)stream)
                : mb == 3 ? launch_forward<3>(net, (cudaStream_t)stream)
                          : launch_forward<4>(net, (cudaStream_t)stream));
        return PS_OK;
    }
    for (int l = 0; l < n_layers; ++l) {
        const int k = sizes[l], n = sizes[l + 1];
        const bool last = l == n_layers - 1;
        SC_CUDA(launch_gemm(make_gemm(rows, n, k, h[l], k, 1, w[l], 1, k, hf[l], n, bias[l], last ? 0 : 1,
                                      last ? nullptr : h[l + 1], n),
                            nullptr, (cudaStream_t)stream));
    }
    return PS_OK;
}

extern "C" ps_status ps_mlp_backward(int32_t n_layers, const int32_t *sizes, int32_t rows, const void *const *w,
                                     const void *const *h, const float *const *hf, float *const *dz, void *const *dzb,
                                     float *const *gw, float *const *gb, void *stream)
{
    if (n_layers < 1 || !sizes || rows < 0 || !w || !h || !hf || !dz || !dzb || !gw || !gb)
        return psb_fail(PS_ERR_ARG, "ps_mlp_backward: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    const int last = n_layers - 1;
    ColumnSums cs{};
    unsigned blocks = 0;
    auto sum_columns = [&]() -> ps_status {
        if (blocks) column_sum_kernel<<<blocks, 1024, 0, s>>>(cs);
        SC_CUDA(cudaGetLastError());
        cs.n = 0;
        blocks = 0;
        return PS_OK;
    };
    for (int l = last; l >= 0; --l) {
        const int k = sizes[l], n = sizes[l + 1];
        if (k < 1 || n < 1 || !w[l] || !gw[l] || !gb[l] || !h[l] || !dz[l] || !dzb[l] || (l > 0 && !hf[l - 1]))
            return psb_fail(PS_ERR_ARG, "ps_mlp_backward: bad layer");
        if (l == last && rows > 0) {
            const long all = (long)rows * n;
            to_bf16_kernel<<<blocks_for(all, 256), 256, 0, s>>>(all, dz[l], (__nv_bfloat16 *)dzb[l]);
            SC_CUDA(cudaGetLastError());
        }
        // the weight gradient, and beside it the gradient of the layer below
        const Gemm grad = make_gemm(n, k, rows, dzb[l], 1, n, h[l], k, 1, gw[l], k, nullptr, 0, nullptr, 0);
        if (l > 0) {
            Gemm down = make_gemm(rows, k, n, dzb[l], n, 1, w[l], k, 1, dz[l - 1], k, nullptr, 0, dzb[l - 1], k);
            down.gate = hf[l - 1];
            down.ldg = k;
            SC_CUDA(launch_gemm(down, &grad, s));
        } else {
            SC_CUDA(launch_gemm(grad, nullptr, s));
        }
        cs.m[cs.n] = {rows, n, (int)blocks, dz[l], gb[l]};
        cs.n += 1;
        blocks += blocks_for(n, 32);
        if (cs.n == 16 && l > 0) {
            const ps_status st = sum_columns();
            if (st != PS_OK) return st;
        }
    }
    return sum_columns();
}

extern "C" ps_status ps_to_bf16(int64_t n, const float *x, void *y, void *stream)
{
    if (n < 0 || !x || !y) return psb_fail(PS_ERR_ARG, "ps_to_bf16: bad arguments");
    if (n == 0) return PS_OK;
    to_bf16_kernel<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(n, x, (__nv_bfloat16 *)y);
    SC_CUDA(cudaGetLastError());
    return PS_OK;
}

extern "C" ps_status ps_screen_rank(int32_t device, int32_t n_points, const double *tim, const double *brightness,
                                    const ps_curves *curves, int32_t n_freq, const double *freqs_per_hour,
                                    int32_t n_layers, const int32_t *sizes, const float *params, float *score)
{
    if (n_freq < 0 || (n_freq > 0 && (!freqs_per_hour || !score)) || n_layers < 1 || n_layers > 16 || !sizes ||
        !params)
        return psb_fail(PS_ERR_ARG, "ps_screen_rank: bad arguments");
    if (sizes[0] != kFeatures || sizes[n_layers] != 1)
        return psb_fail(PS_ERR_ARG, "ps_screen_rank: the network must map 88 features to 1 score");
    for (int l = 1; l < n_layers; ++l)
        if (sizes[l] < 1 || sizes[l] > 4096) return psb_fail(PS_ERR_ARG, "ps_screen_rank: layer width 1..4096");
    if (n_freq == 0) return PS_OK;
    // features (1/day), then standardised per feature over this object's frequencies
    std::vector<double> fday(n_freq);
    for (int f = 0; f < n_freq; ++f) fday[f] = 24.0 * freqs_per_hour[f];
    std::vector<float> feat((size_t)n_freq * kFeatures);
    ps_status st = ps_screen_features(device, n_points, tim, brightness, curves, n_freq, fday.data(), feat.data());
    if (st != PS_OK) return st;
    for (int k = 0; k < kFeatures; ++k) {
        double m = 0, m2 = 0;
        for (int f = 0; f < n_freq; ++f) m += feat[(size_t)f * kFeatures + k];
        m /= n_freq;
        for (int f = 0; f < n_freq; ++f) {
            const double d = feat[(size_t)f * kFeatures + k] - m;
            m2 += d * d;
        }
        const double sd = std::sqrt(m2 / n_freq);
        const double inv = sd > 1e-6 ? 1.0 / sd : 1.0;
        for (int f = 0; f < n_freq; ++f) {
            float &v = feat[(size_t)f * kFeatures + k];
            v = (float)((v - m) * inv);
        }
    }
    // device buffers: parameters (FP32 + BF16 copies), two activation buffers
    size_t n_par = 0, widest = kFeatures;
    for (int l = 0; l < n_layers; ++l) {
        n_par += (size_t)sizes[l + 1] * sizes[l] + sizes[l + 1];
        widest = std::max<size_t>(widest, (size_t)sizes[l + 1]);
    }
    float *d_par = nullptr, *d_out = nullptr;
    __nv_bfloat16 *d_parb = nullptr, *d_h[2] = {nullptr, nullptr};
    cudaError_t e = cudaMalloc(&d_par, sizeof(float) * n_par);
    if (e == cudaSuccess) e = cudaMalloc(&d_parb, sizeof(__nv_bfloat16) * n_par);
    if (e == cudaSuccess) e = cudaMalloc(&d_out, sizeof(float) * ((size_t)n_freq * widest + n_freq * kFeatures));
    if (e == cudaSuccess) e = cudaMalloc(&d_h[0], sizeof(__nv_bfloat16) * (size_t)n_freq * widest);
    if (e == cudaSuccess) e = cudaMalloc(&d_h[1], sizeof(__nv_bfloat16) * (size_t)n_freq * widest);
    float *d_feat = d_out + (size_t)n_freq * widest;
    if (e == cudaSuccess) e = cudaMemcpy(d_par, params, sizeof(float) * n_par, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(d_feat, feat.data(), sizeof(float) * feat.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        to_bf16_kernel<<<blocks_for((long)n_par, 256), 256>>>((long)n_par, d_par, d_parb);
        to_bf16_kernel<<<blocks_for((long)feat.size(), 256), 256>>>((long)feat.size(), d_feat, d_h[0]);
        e = cudaGetLastError();
    }
    size_t off = 0;
    int cur = 0;
    for (int l = 0; l < n_layers && e == cudaSuccess; ++l) {
        const int k = sizes[l], n = sizes[l + 1];
        const __nv_bfloat16 *W = d_parb + off;
        const float *b = d_par + off + (size_t)n * k;
        off += (size_t)n * k + n;
        const bool last = l == n_layers - 1;
        e = launch_gemm(make_gemm(n_freq, n, k, d_h[cur], k, 1, W, 1, k, last ? d_out : nullptr, n, b, last ? 0 : 1,
                                  last ? nullptr : d_h[1 - cur], n),
                        nullptr, nullptr);
        cur = 1 - cur;
    }
    if (e == cudaSuccess) e = cudaMemcpy(score, d_out, sizeof(float) * n_freq, cudaMemcpyDeviceToHost);
    cudaFree(d_par);
    cudaFree(d_parb);
    cudaFree(d_out);
    cudaFree(d_h[0]);
    cudaFree(d_h[1]);
    if (e != cudaSuccess) return psb_fail_cuda(e, "ps_screen_rank");
    return PS_OK;
}
