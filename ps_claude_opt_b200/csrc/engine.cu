// engine.cu -- template dispatch and launch wrappers of the fit kernel.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "engine.h"
#include "fit_kernel.cuh"

namespace psb {

using KernelFn = void (*)(DevObject, DevParams, const FitItem *, int, int *, FitOut *, double *, size_t,
                          int *, EvalOut, int, const DevObject *, const DevParams *);

// The shape-derivative accumulators live in registers, so the kernel is
// compiled per padded coefficient count.
#define PSB_NCP_LIST(X) X(16) X(24) X(32) X(40) X(48) X(56) X(64) X(72) X(80) X(88)

int padded_ncoef(int n_coef)
{
#define PSB_PICK(N) if (n_coef <= N) return N;
    PSB_NCP_LIST(PSB_PICK)
#undef PSB_PICK
    return -1;
}

size_t fit_smem_bytes(int n_fac, int mfit, int ncp, int n_curves, int row_stride, int tile_rows, int cstat_smem,
                      int mixed)
{
    return kStaticSmem +
           carve_bytes(n_fac, mfit, ncp, n_curves, row_stride, tile_rows, cstat_smem, mixed, nullptr, nullptr);
}

size_t fit_dynamic_smem(const DevObject &o)
{
    return carve_bytes(o.n_fac, o.mfit, o.ncp, o.n_curves, o.row_stride, o.tile_rows, o.cstat_smem, o.mixed, nullptr,
                       nullptr);
}

int chunk_facets_of(int ncp) { return chunk_facets(ncp); }

size_t fit_scratch_doubles(const DevObject &o)
{
    size_t n = scratch_perm(o.n_points, o.row_stride, o.n_curves, o.ma) + (size_t)o.n_points;
    return (n + 31) & ~size_t(31);
}

// The mixed-precision sweep is built for the smaller bases (chunks of 32
// facets, ncp <= kMaxMixedNcp).
#define PSB_MIXED_LIST(X) X(16) X(24) X(32) X(40) X(48) X(56) X(64)

// One translation unit per instance (fit_inst.cu) exports its kernel.
#define PSB_DECL(N) KernelFn fit_kernel_ptr_##N();
PSB_NCP_LIST(PSB_DECL)
#undef PSB_DECL
#define PSB_DECLM(N) KernelFn fit_kernel_mixed_ptr_##N();
PSB_MIXED_LIST(PSB_DECLM)
#undef PSB_DECLM
#define PSB_DECLB(N) KernelFn fit_kernel_batch_ptr_##N();
PSB_NCP_LIST(PSB_DECLB)
#undef PSB_DECLB

#define PSB_DECLT(N) KernelFn fit_kernel_team_ptr_##N();
PSB_NCP_LIST(PSB_DECLT)
#undef PSB_DECLT
#define PSB_DECLMT(N) KernelFn fit_kernel_mixed_team_ptr_##N();
PSB_MIXED_LIST(PSB_DECLMT)
#undef PSB_DECLMT

static KernelFn team_kernel_for(int ncp, int mixed)
{
    if (mixed) {
        switch (ncp) {
#define PSB_CASEMT(N) \
    case N:           \
        return fit_kernel_mixed_team_ptr_##N();
            PSB_MIXED_LIST(PSB_CASEMT)
#undef PSB_CASEMT
        default:
            return nullptr;
        }
    }
    switch (ncp) {
#define PSB_CASET(N) \
    case N:          \
        return fit_kernel_team_ptr_##N();
        PSB_NCP_LIST(PSB_CASET)
#undef PSB_CASET
    default:
        return nullptr;
    }
}

static KernelFn batch_kernel_for(int ncp)
{
    switch (ncp) {
#define PSB_CASEB(N) \
    case N:          \
        return fit_kernel_batch_ptr_##N();
        PSB_NCP_LIST(PSB_CASEB)
#undef PSB_CASEB
    default:
        return nullptr;
    }
}

static KernelFn kernel_for(int ncp, int mixed)
{
    if (mixed) {
        switch (ncp) {
#define PSB_CASEM(N) \
    case N:          \
        return fit_kernel_mixed_ptr_##N();
            PSB_MIXED_LIST(PSB_CASEM)
#undef PSB_CASEM
        default:
            return nullptr;
        }
    }
    switch (ncp) {
#define PSB_CASE(N) \
    case N:         \
        return fit_kernel_ptr_##N();
        PSB_NCP_LIST(PSB_CASE)
#undef PSB_CASE
    default:
        return nullptr;
    }
}

// Every use of a kernel allows it what the largest layout takes, not its own
// object's: the allowance belongs to the kernel, and with the object's own size
// a handle in another thread, of a smaller object, took it away between this and
// the launch.
static int allow_smem(KernelFn fn)
{
    return (int)cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kBlockSmem - kStaticSmem));
}

static int prepare_kernel(const DevObject &o, KernelFn *fn, size_t *smem)
{
    *fn = kernel_for(o.ncp, o.mixed);
    if (!*fn) return (int)cudaErrorInvalidValue;
    *smem = fit_dynamic_smem(o);
    return allow_smem(*fn);
}

int fit_ctas_per_sm(const DevObject &o)
{
    KernelFn fn;
    size_t smem;
    if (prepare_kernel(o, &fn, &smem) != 0) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kThreads, smem) != cudaSuccess) return 0;
    return n;
}

int launch_fits(const DevObject &o, const DevParams &p, const FitItem *items, int n_items, int *queue,
                FitOut *out, double *scratch, size_t scratch_per_cta, int n_ctas, int *status, void *stream)
{
    KernelFn fn;
    size_t smem;
    int e = prepare_kernel(o, &fn, &smem);
    if (e) return e;
    EvalOut ev{};
    fn<<<n_ctas, kThreads, smem, (cudaStream_t)stream>>>(o, p, items, n_items, queue, out, scratch,
                                                         scratch_per_cta, status, ev, 0, nullptr, nullptr);
    return (int)cudaGetLastError();
}

int prepare_batch_kernel(const DevObject &env)
{
    KernelFn fn = batch_kernel_for(env.ncp);
    if (!fn || env.mixed) return (int)cudaErrorInvalidValue;
    return allow_smem(fn);
}

int fit_batch_ctas_per_sm(const DevObject &env)
{
    if (prepare_batch_kernel(env) != 0) return 0;
    const size_t smem = fit_dynamic_smem(env);
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_kernel_for(env.ncp), kThreads, smem) != cudaSuccess)
        return 0;
    return n;
}

int launch_fits_batch(const DevObject &env, const DevObject *d_objs, const DevParams *d_prms, const FitItem *items,
                      int n_items, int *queue, FitOut *out, double *scratch, size_t scratch_per_cta, int n_ctas,
                      int *status, void *stream)
{
    KernelFn fn = batch_kernel_for(env.ncp);
    if (!fn || env.mixed) return (int)cudaErrorInvalidValue;
    const size_t smem = fit_dynamic_smem(env);
    DevParams p{};
    EvalOut ev{};
    fn<<<n_ctas, kThreads, smem, (cudaStream_t)stream>>>(env, p, items, n_items, queue, out, scratch,
                                                         scratch_per_cta, status, ev, 0, d_objs, d_prms);
    return (int)cudaGetLastError();
}

// Launch configuration of `groups` teams of team_size CTAs.
struct TeamLaunch {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    KernelFn fn = nullptr;
    int prepare(const DevObject &o, int groups, int team_size, void *stream)
    {
        fn = team_kernel_for(o.ncp, o.mixed);
        if (!fn) return (int)cudaErrorInvalidValue;
        const size_t smem = fit_dynamic_smem(o);
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = team_size;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(groups * team_size);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = (cudaStream_t)stream;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        return allow_smem(fn);
    }
};

// Teams of this size the GPU holds at a time (0 if none).
static int max_teams(const DevObject &o, int team_size)
{
    TeamLaunch l;
    int n = 0;
    if (l.prepare(o, 1, team_size, nullptr) != 0 ||
        cudaOccupancyMaxActiveClusters(&n, l.fn, &l.cfg) != cudaSuccess) {
        cudaGetLastError();  // not the next launch's
        return 0;
    }
    return n;
}

void load_team_kernel(const DevObject &o)
{
    TeamLaunch l;
    if (l.prepare(o, 1, 2, nullptr) != 0) cudaGetLastError();  // the launch itself will say so
}

constexpr int kTeamSizes[3] = {2, 4, 8};
// Time of one fit by a team, as a share of its time by one CTA.  Measured, FP64,
// teams of 2 / 4 / 8: production object 0.73 / 0.42 / 0.27, largest models
// 0.78 / 0.48 / 0.31, config 1 0.91 / 0.64 / 0.45; mixed precision 0.88 / 0.53 /
// 0.33.  (The solve and the barriers do not divide, and a team's few tiles a
// warp leave the sweep's rounds uneven.)
constexpr double kTeamTime[3] = {0.78, 0.46, 0.31};

FitPlan plan_fits(const DevObject &o, int n, int resident, int max_slabs, bool mixable)
{
    FitPlan pl;
    const int slabs = max_slabs > 0 ? max_slabs : INT_MAX;
    const int wave = std::max(1, std::min(resident, slabs));  // fits one wave of single CTAs holds
    const int waves = n / wave, rest = n - waves * wave;
    pl.main_items = n;
    pl.main_ctas = std::min(n, wave);
    // with nothing but whole waves, or a last wave too full to split, single
    // CTAs are best; without a second stream all fits go one way.  A wave of
    // single CTAs takes 1, so teams must make the rest cheaper.  B200's 148 SMs
    // hold 15 teams of 8, 33 of 4 or 74 of 2 at a time, so production fits go by
    // teams of 8 up to 15 (10 fits: 56.3 -> 15.4 ms), of 4 up to 33 (30 fits: 23.8
    // ms), of 2 up to 74 (70 fits: 41.7 ms), and by single CTAs above (140 fits:
    // 56.3 ms)
    const int items = mixable ? rest : n;
    if (items == 0) return pl;
    double best = mixable ? 1.0 : (n + wave - 1) / wave;
    best *= 0.95;
    for (int k = 0; k < 3; ++k) {
        // teams that this number of fits could use at once
        if (mixable && (double)((items * kTeamSizes[k] + resident - 1) / resident) * kTeamTime[k] >= best) continue;
        const int teams = std::min({max_teams(o, kTeamSizes[k]), slabs, items});
        if (teams < 1) continue;
        const double t = ((items + teams - 1) / teams) * kTeamTime[k];
        if (t < best) {
            best = t;
            pl.teams = teams;
            pl.team_size = kTeamSizes[k];
        }
    }
    if (pl.teams) {
        pl.team_items = items;
        pl.main_items = n - items;
        pl.main_ctas = std::min(pl.main_items, wave);
    }
    return pl;
}

int launch_fit_teams(const DevObject &o, const DevParams &p, const FitItem *items, int n_items, int *queue,
                     FitOut *out, double *scratch, size_t scratch_per_cta, int groups, int team_size, int *status,
                     void *stream)
{
    TeamLaunch l;
    const int e = l.prepare(o, groups, team_size, stream);
    if (e) return e;
    EvalOut ev{};
    return (int)cudaLaunchKernelEx(&l.cfg, l.fn, o, p, items, n_items, queue, out, scratch, scratch_per_cta, status, ev,
                                   0, (const DevObject *)nullptr, (const DevParams *)nullptr);
}

int launch_eval(const DevObject &o, const DevParams &p, EvalOut ev, double *scratch, int *status, void *stream)
{
    // the largest team the GPU holds; where one CTA of a layout fits, a pair does:
    // the layout was chosen with the teams' static shared memory counted in
    for (int k = 2; k >= 0; --k) {
        if (max_teams(o, kTeamSizes[k]) < 1) continue;
        TeamLaunch l;
        const int e = l.prepare(o, 1, kTeamSizes[k], stream);
        if (e) return e;
        return (int)cudaLaunchKernelEx(&l.cfg, l.fn, o, p, (const FitItem *)nullptr, 1, (int *)nullptr,
                                       (FitOut *)nullptr, scratch, (size_t)0, status, ev, 1,
                                       (const DevObject *)nullptr, (const DevParams *)nullptr);
    }
    return (int)cudaErrorLaunchOutOfResources;
}

}  // namespace psb
