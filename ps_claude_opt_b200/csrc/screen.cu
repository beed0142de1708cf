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

// C[m][n] (+)= sum_k A(m, k) B(k, n) (+ bias[n]) (ReLU), A(m, k) = A[m sam + k sak],
// B(k, n) = B[k sbk + n sbn], BF16 operands on the tensor cores, FP32
// accumulation.  A block of 4 warps computes a 64 x 32 tile; operands are
// read element by element with bounds checks, so any strides (transposes)
// and any sizes work.
constexpr int kGemmTM = 64, kGemmTN = 32;

__global__ void __launch_bounds__(128) gemm_bf16_kernel(int M, int N, int K, const __nv_bfloat16 *A, long sam,
                                                        long sak, const __nv_bfloat16 *B, long sbk, long sbn,
                                                        float *C, int ldc, int accumulate, const float *bias,
                                                        int relu, __nv_bfloat16 *Cb, int ldcb)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int m0 = blockIdx.y * kGemmTM + warp * 16;
    const int n0 = blockIdx.x * kGemmTN;
    const __nv_bfloat16 zero = __float2bfloat16(0.0f);
    auto ld_a = [&](int m, int k) { return (m < M && k < K) ? A[(long)m * sam + (long)k * sak] : zero; };
    auto ld_b = [&](int k, int n) { return (k < K && n < N) ? B[(long)k * sbk + (long)n * sbn] : zero; };
    float acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += 16) {
        uint32_t a[4];
        a[0] = pack_bf16(ld_a(m0 + g, k0 + 2 * t), ld_a(m0 + g, k0 + 2 * t + 1));
        a[1] = pack_bf16(ld_a(m0 + g + 8, k0 + 2 * t), ld_a(m0 + g + 8, k0 + 2 * t + 1));
        a[2] = pack_bf16(ld_a(m0 + g, k0 + 2 * t + 8), ld_a(m0 + g, k0 + 2 * t + 9));
        a[3] = pack_bf16(ld_a(m0 + g + 8, k0 + 2 * t + 8), ld_a(m0 + g + 8, k0 + 2 * t + 9));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + 8 * j + g;
            const uint32_t b0 = pack_bf16(ld_b(k0 + 2 * t, n), ld_b(k0 + 2 * t + 1, n));
            const uint32_t b1 = pack_bf16(ld_b(k0 + 2 * t + 8, n), ld_b(k0 + 2 * t + 9, n));
            mma_bf16(acc[j], a, b0, b1);
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int m = m0 + g + (e >= 2 ? 8 : 0);
            const int n = n0 + 8 * j + 2 * t + (e & 1);
            if (m >= M || n >= N) continue;
            float v = acc[j][e];
            if (accumulate) v += C[(long)m * ldc + n];
            if (bias) v += bias[n];
            if (relu) v = fmaxf(v, 0.0f);
            if (C) C[(long)m * ldc + n] = v;
            if (Cb) Cb[(long)m * ldcb + n] = __float2bfloat16(v);
        }
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

// db[n] = sum over rows of dZ[r][n] (one thread per column, rows in order).
__global__ void column_sum_kernel(int rows, int cols, const float *dz, float *db)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= cols) return;
    float s = 0.0f;
    for (int r = 0; r < rows; ++r) s += dz[(long)r * cols + n];
    db[n] = s;
}

// Adam on FP32 master weights, then the BF16 working copy.
__global__ void adam_kernel(long n, float *w, const float *grad, float *m, float *v, float lr, float b1, float b2,
                            float eps, float c1, float c2, __nv_bfloat16 *wb)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gr = grad[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gr;
    const float vi = b2 * v[i] + (1.0f - b2) * gr * gr;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    if (wb) wb[i] = __float2bfloat16(wi);
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
    dim3 grid((N + kGemmTN - 1) / kGemmTN, (M + kGemmTM - 1) / kGemmTM);
    gemm_bf16_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(
        M, N, K, (const __nv_bfloat16 *)A, sam, sak, (const __nv_bfloat16 *)B, sbk, sbn, C, ldc, accumulate, bias,
        relu, (__nv_bfloat16 *)Cb, ldcb);
    SC_CUDA(cudaGetLastError());
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
    column_sum_kernel<<<blocks_for(cols, 128), 128, 0, (cudaStream_t)stream>>>(rows, cols, x, out);
    SC_CUDA(cudaGetLastError());
    return PS_OK;
}

extern "C" ps_status ps_adam_step(int64_t n, float *w, const float *grad, float *m, float *v, float lr, float beta1,
                                  float beta2, float eps, int32_t step, void *wb, void *stream)
{
    if (n < 0 || !w || !grad || !m || !v || step < 1) return psb_fail(PS_ERR_ARG, "ps_adam_step: bad arguments");
    if (n == 0) return PS_OK;
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    adam_kernel<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(n, w, grad, m, v, lr, beta1, beta2, eps, c1,
                                                                       c2, (__nv_bfloat16 *)wb);
    SC_CUDA(cudaGetLastError());
    return PS_OK;
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
        dim3 grid((n + kGemmTN - 1) / kGemmTN, (n_freq + kGemmTM - 1) / kGemmTM);
        gemm_bf16_kernel<<<grid, 128>>>(n_freq, n, k, d_h[cur], k, 1, W, 1, k, last ? d_out : nullptr, n, 0, b,
                                        last ? 0 : 1, last ? nullptr : d_h[1 - cur], n);
        e = cudaGetLastError();
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
