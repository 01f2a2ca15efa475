/*
 * pt_api.cu -- the C ABI (include/particles_gb300.h): errors, argument
 * checking, parameter unpacking, kernel dispatch, device-buffer runs, the
 * autotuner and the debug entry points.  Field handles live in pt_fields.cu,
 * host-buffer runs (the drop-in pt_integrate) in pt_hostio.cu, ensembles in
 * pt_ensemble.cu.  Nothing here calls a CPU fallback: without a usable GPU
 * every entry point returns PT_ERR_CUDA.
 */
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <math.h>
#include <stdio.h>
#include <string.h>
#include <strings.h>

#include "pt_common.cuh"
#include "pt_detmath.h"
#include "pt_tableau.h"
#include "pt_internal.h"
#include "pt_tableau.h"

/* Device blob of a learned-controller model (pt_mlp_train.cu). */
const unsigned char *pt_mlp_blob(const pt_mlp *m);

/* ---------------------------------------------------------------------- */
/* errors                                                                 */
/* ---------------------------------------------------------------------- */

namespace pt_internal {

thread_local char g_err[512] = "";

int set_err(int code, const char *fmt, const char *detail)
{
    snprintf(g_err, sizeof g_err, fmt, detail ? detail : "");
    return code;
}

int cuda_err(cudaError_t e, const char *where)
{
    snprintf(g_err, sizeof g_err, "%s: %s", where, cudaGetErrorString(e));
    return (e == cudaErrorMemoryAllocation) ? PT_ERR_NOMEM : PT_ERR_CUDA;
}

}  // namespace pt_internal

using namespace pt_internal;

/* SMs of the device that is current at the first call. */
int pt_coop_sms()
{
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n < 1 ? 1 : n;
    }();
    return sms;
}

/* pt_debug_machines of the calling thread; -1: the library's own */
static thread_local int64_t g_coop_limit = -1;
static thread_local int g_hand_cap = -1;

int64_t pt_coop_max()
{
    return g_coop_limit >= 0 ? g_coop_limit : (int64_t)PT_COOP_PER_SM * pt_coop_sms();
}

int pt_hand_cap() { return g_hand_cap >= 0 ? g_hand_cap : PT_HAND_CAP; }

extern "C" int64_t pt_debug_machines(int64_t limit, int32_t hand_cap)
{
    g_coop_limit = limit < 0 ? -1 : limit;
    g_hand_cap = hand_cap < 0 || hand_cap > PT_HAND_CAP ? -1 : hand_cap;
    return pt_coop_max();
}

extern "C" const char *pt_last_error(void) { return g_err; }
extern "C" int32_t pt_abi_version(void) { return PT_ABI_VERSION; }

extern "C" int64_t pt_carry_bytes(int64_t np)
{
    return np > 0 ? np * PT_CARRY_BYTES_PER_PARTICLE : 0;
}

extern "C" int32_t pt_method_from_name(const char *name)
{
    if (!name) return 0;
    /* particles.F90:337-347 compares trim(method) case-sensitively */
    char b[33];
    size_t n = strlen(name);
    while (n > 0 && name[n - 1] == ' ') --n;
    if (n == 0 || n > 32) return 0;
    memcpy(b, name, n);
    b[n] = 0;
    if (!strcmp(b, "rk5")) return PT_METHOD_RK5;
    if (!strcmp(b, "dop853") || !strcmp(b, "dp853") || !strcmp(b, "rk8")) return PT_METHOD_DOP853;
    return 0;
}

/* ---------------------------------------------------------------------- */
/* runs                                                                   */
/* ---------------------------------------------------------------------- */

namespace pt_internal {

void unpack_params(const double *p, const RunShape &g, PtRun &R)
{
    memset(&R, 0, sizeof R);
    R.qom = p[0]; R.vun = p[1]; R.tmx = p[2]; R.dtm = p[4];
    R.atol = p[5]; R.rtol = p[6]; R.fcmn = p[7]; R.fcmx = p[8]; R.safe = p[9];
    R.beta = p[10];
    R.expo = 2.0e-01 * R.beta - 1.25e-01;                     /* integrations.F90:348 */
    bool unit = true;
    for (int i = 0; i < 3; ++i) {
        R.xl[i] = p[11 + i];
        R.xs[i] = p[14 + i];
        R.dm[i] = g.dm[i];
        R.dmr[i] = (double)g.dm[i];
        R.inv_dm[i] = 1.0 / (double)g.dm[i];
        R.dm_mask[i] = ((g.dm[i] & (g.dm[i] - 1)) == 0) ? g.dm[i] - 1 : 0;
        R.gsx[i] = (double)g.dm[i] / R.xs[i];
        R.gox[i] = -R.xl[i] * R.gsx[i];
        R.gsxf[i] = (float)R.gsx[i];
        R.inv_xs[i] = 1.0 / R.xs[i];
        unit = unit && (R.xl[i] == 0.0) && !signbit(R.xl[i]) && (R.xs[i] == 1.0);
    }
    R.unit_map = unit ? 1 : 0;
    R.inv_vun = 1.0 / R.vun;
    R.inv_atol = 1.0 / R.atol;
    R.ivunf = (float)R.inv_vun;
    R.qomf = (float)R.qom;
}

/* PT_CTL_NOISE: the embedded error estimate is a combination sum_j e_j k_j of
 * the stage derivatives, and an FP32 evaluation (trilinear sums and force
 * in FP32) carries a rounding error of a few units in the last place of the
 * largest component of its group (positions, momenta).  The stages round
 * independently, so with PT_NOISE_ULP such units per stage the estimate's
 * noise is nu = PT_NOISE_ULP 2^-24 sqrt(sum_j e_j^2) |f|_max.  The norm adds
 * twice that to each component's scale sr, so that an estimate made of
 * noise alone scores at most about 1/2 and the controller responds to
 * truncation errors only:
 *   RK5 (del = max |er / sr| / atol, k = dt f):  sr += 2 nu / atol with
 *       dt |f|_max read as |k1|_max, coefficient 2 PT_NOISE_ULP 2^-24 |d|_2 / atol;
 *   DOP853 (err = |dt| ||e / sr|| with e in units of f):  sr += 2 |dt| nu,
 *       with |dt| |f|_max read as the largest component of the step's
 *       increment dt k4 (in registers), coefficient 2 PT_NOISE_ULP 2^-24 |er|_2.
 * Without it the reference's per-component scales (RK5: |si| + |k1|) become
 * tiny where a momentum component crosses zero during a gyration, an
 * estimate made of FP32 rounding exceeds them at every step size, and the
 * controller shrinks dt without end (measured: 17,535 attempts in a
 * 0.1-gyro-period window for a particle the FP64 kernel takes in 365). */
#define PT_NOISE_ULP 8.0
static double noise_floor(int method, double atol)
{
    using namespace pt_tab;
    const double u = PT_NOISE_ULP * 5.9604644775390625e-08;     /* 2^-24 */
    if (method == PT_METHOD_DOP853) {
        const double e[8] = { ER01, ER06, ER07, ER08, ER09, ER10, ER11, ER12 };
        double s = 0.0;
        for (double x : e) s += x * x;
        return 2.0 * u * sqrt(s);
    }
    const double d[5] = { CK_D1, CK_D3, CK_D4, CK_D5, CK_D6 };
    double s = 0.0;
    for (double x : d) s += x * x;
    return 2.0 * u * sqrt(s) / atol;
}

/* Face-cap constants (PT_CTL_FACE) per method [RK5, DOP853]: faces reached
 * within skip x the proposed step are crossed; steps end `over` cells of the
 * fastest axis past the capping face.  pt_debug_face_params sets them.
 * Tuned on the benchmark workloads (FMA / FP32 builds), simulated time per
 * second relative to the same build without the cap:
 *   RK5 (rtol 1e-8, 512^3): skip 0.05 / 0.1 / 0.15 -> 1.52x / 1.62x / 1.60x;
 *     overshoot 1e-2 / 1e-3 / 1e-4 / 3e-5 at skip 0.1 -> 1.09x / 1.46x /
 *     1.62x / 1.63x;
 *   DOP853 (rtol 1e-10, 256^3): skip 0 / 0.005 / 0.01 / 0.02 / 0.1 / 0.3
 *     -> 2.91x / 3.50x / 3.43x / 3.32x / 2.86x / 2.24x at overshoot 3e-5. */
static float g_face_skip[2] = { 0.1f, 0.01f }, g_face_over[2] = { 3.0e-5f, 3.0e-5f };

/* pt_options.threads_per_block, read only from callers whose struct has it
 * (struct_size 0 means the current layout). */
int32_t pt_opt_threads_per_block(const pt_options *opt)
{
    if (!opt) return 0;
    const int32_t need = (int32_t)(offsetof(pt_options, threads_per_block) + sizeof(int32_t));
    return (opt->struct_size == 0 || opt->struct_size >= need) ? opt->threads_per_block : 0;
}

/* pt_options.open_x_margin under the same rule. */
double pt_opt_open_x_margin(const pt_options *opt)
{
    if (!opt) return 0.0;
    const int32_t need = (int32_t)(offsetof(pt_options, open_x_margin) + sizeof(double));
    return (opt->struct_size == 0 || opt->struct_size >= need) ? opt->open_x_margin : 0.0;
}

int prepare_run(int32_t method, int64_t np, int32_t m, const RunShape &g,
                       const double *params, const pt_options *opt, PtRun &R)
{
    if (method != PT_METHOD_RK5 && method != PT_METHOD_DOP853)
        return set_err(PT_ERR_ARG, "unknown method%s");
    if (np < 0 || m < 1) return set_err(PT_ERR_ARG, "np < 0 or m < 1%s");
    if (!params) return set_err(PT_ERR_ARG, "params is NULL%s");
    if ((int64_t)m * np > ((int64_t)1 << 56)) return set_err(PT_ERR_ARG, "state too large%s");
    for (int i = 0; i < 17; ++i)
        if (i != 3 && !isfinite(params[i])) return set_err(PT_ERR_ARG, "non-finite params%s");
    if (params[14] == 0.0 || params[15] == 0.0 || params[16] == 0.0)
        return set_err(PT_ERR_ARG, "zero domain size%s");
    double eta = 0.0, t_stop = 0.0, budget = 0.0;
    int32_t open_x = 0;
    int64_t max_steps = 0;
    if (opt) {
        if (opt->precision != g.precision)
            return set_err(PT_ERR_ARG, "options precision differs from the field handle%s");
        if (opt->controller < 0 || opt->controller > (PT_CTL_LEARNED | PT_CTL_FACE | PT_CTL_NOISE))
            return set_err(PT_ERR_ARG, "unknown controller%s");
        if ((opt->controller & PT_CTL_NOISE) && g.precision != PT_PREC_FP32 &&
            g.precision != PT_PREC_BF16)
            return set_err(PT_ERR_UNSUPPORTED, "the error norm's rounding floor is for the FP32 "
                                               "evaluation (PT_PREC_FP32 / PT_PREC_BF16)%s");
        if ((opt->controller & PT_CTL_LEARNED) && !opt->model)
            return set_err(PT_ERR_ARG, "the learned controller needs opt->model%s");
        if ((opt->controller & PT_CTL_FACE) && g.precision == PT_PREC_FP64)
            return set_err(PT_ERR_UNSUPPORTED, "PT_PREC_FP64 keeps the reference's controller; "
                                               "face-capped steps need another precision%s");
        if (opt->records && opt->record_capacity < 0)
            return set_err(PT_ERR_ARG, "negative record capacity%s");
        if (opt->blocks_per_sm != 0 && (opt->blocks_per_sm < 2 || opt->blocks_per_sm > 4))
            return set_err(PT_ERR_ARG, "blocks_per_sm must be 0, 2, 3 or 4%s");
        const int32_t tpb = pt_opt_threads_per_block(opt);
        if (tpb != 0 && tpb != 64 && tpb != 128 && tpb != 256)
            return set_err(PT_ERR_ARG, "threads_per_block must be 0, 64, 128 or 256%s");
        if (opt->interpolation != 0 && opt->interpolation != 1)
            return set_err(PT_ERR_ARG, "interpolation must be 0 (trilinear) or 1 (nearest node)%s");
        if (opt->interpolation == 1 && (opt->controller & PT_CTL_LEARNED))
            return set_err(PT_ERR_UNSUPPORTED, "the learned controller's features need the trilinear gather%s");
        eta = opt->eta;
        t_stop = opt->t_stop;
        budget = opt->time_budget_s;
        open_x = opt->open_x;
        max_steps = opt->max_steps;
    }
    const double margin = pt_opt_open_x_margin(opt);
    if (!isfinite(eta) || !isfinite(t_stop) || !isfinite(budget) || !isfinite(margin))
        return set_err(PT_ERR_ARG, "non-finite option%s");
    if (margin < 0.0) return set_err(PT_ERR_ARG, "open_x_margin must be >= 0%s");
    if (eta != 0.0 && !g.has_j)
        return set_err(PT_ERR_ARG, "eta != 0 needs a field handle created with J%s");
    if (eta == 0.0 && g.has_j)
        return set_err(PT_ERR_ARG, "field handle holds J but eta == 0%s");
    unpack_params(params, g, R);
    R.eta = eta;
    R.etaf = (float)eta;
    R.has_j = g.has_j;
    R.open_x = open_x ? 1 : 0;
    /* the same expressions as the oracle, so the escape test matches bit for bit */
    R.xo_lo = (margin == 0.0) ? R.xl[0] : R.xl[0] - margin * R.xs[0];
    R.xo_hi = (margin == 0.0) ? R.xl[0] + R.xs[0] : R.xl[0] + R.xs[0] + margin * R.xs[0];
    R.max_steps = max_steps > 0 ? max_steps : 1000000000LL;
    R.tend = (t_stop > 0.0 && t_stop < R.tmx) ? t_stop : R.tmx;
    R.budget_ns = (uint64_t)((budget > 0.0 ? budget : 600.0) * 1e9);
    R.m = m;
    R.np = np;
    R.few = pt_coop_max();
    if (opt) {
        R.mlp = (opt->controller & PT_CTL_LEARNED)
                    ? pt_mlp_blob(static_cast<const pt_mlp *>(opt->model)) : nullptr;
        R.face = (opt->controller & PT_CTL_FACE) ? 1 : 0;
        R.face_skip = g_face_skip[method == PT_METHOD_DOP853];
        R.face_over = g_face_over[method == PT_METHOD_DOP853];
        R.noise = (opt->controller & PT_CTL_NOISE) ? noise_floor(method, R.atol) : 0.0;
        R.rec = static_cast<float *>(opt->records);
        R.rec_cap = opt->record_capacity;
        R.order = opt->order;
        R.minb = opt->blocks_per_sm;
        R.block = pt_opt_threads_per_block(opt);
        R.near = opt->interpolation;
    }
    return PT_OK;
}

/* Launch variants chosen by pt_autotune, per kernel family
 * [precision][method - 1][with J][learned]: blocks_per_sm | threads_per_block
 * << 8; 0 = not tuned. */
static std::atomic<int> g_tuned[4][2][2][2];

std::atomic<int> &tuned_slot(int32_t method, const pt_fields *f, const PtRun &R)
{
    return g_tuned[f->precision & 3][method - 1][f->has_j ? 1 : 0][(R.mlp || R.rec) ? 1 : 0];
}

RunShape shape_of(const pt_fields *f)
{
    RunShape g;
    for (int i = 0; i < 3; ++i) g.dm[i] = f->dm[i];
    g.precision = f->precision;
    g.has_j = f->has_j;
    return g;
}

cudaError_t launch_run(int32_t method, const pt_fields *f, const PtRun &R, cudaStream_t s)
{
    if (f->precision == PT_PREC_FP64)
        return method == PT_METHOD_RK5 ? pt_launch_rk5_exact(R, f->nc, s) : pt_launch_dp853_exact(R, f->nc, s);
    if (f->precision == PT_PREC_FP64_FMA)
        return method == PT_METHOD_RK5 ? pt_launch_rk5_fma(R, f->nc, s) : pt_launch_dp853_fma(R, f->nc, s);
    if (f->precision == PT_PREC_BF16)
        return method == PT_METHOD_RK5 ? pt_launch_rk5_bf16(R, f->nc16, s)
                                       : pt_launch_dp853_bf16(R, f->nc16, s);
    return method == PT_METHOD_RK5 ? pt_launch_rk5_mixed(R, f->nc32, s)
                                   : pt_launch_dp853_mixed(R, f->nc32, s);
}

void attach_fields(const pt_fields *f, PtRun &R)
{
    R.fld = f->rec64;
    R.fld32 = f->rec32;
    R.fld16 = f->rec16;
    R.bscale = f->bscale;
    for (int i = 0; i < 3; ++i) R.nb[i] = f->nb[i];
    const int64_t nbk = (int64_t)f->nb[0] * f->nb[1] * f->nb[2];
    R.nrec = f->precision == PT_PREC_BF16 ? nbk * 729                 /* halo bricks */
           : f->precision == PT_PREC_FP32 ? nbk * 512                 /* compact bricks */
           : f->nodes;
    R.oob = f->scratch + 2;
}

void attach_hand(const pt_fields *fc, PtRun &R)
{
    pt_fields *f = const_cast<pt_fields *>(fc);
    if (R.np <= R.few) return;
    if (!f->hand) {
        /* In the default mode of a stream capture, here or in another thread, an
         * allocation invalidates the capture, be it of another stream than this
         * run's.  It is no part of any graph, so the relaxed mode fits. */
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
        if (e == cudaSuccess) {
            e = cudaMalloc(&f->hand, (size_t)PT_HAND_CAP * PT_HAND_WORDS * 8);
            const cudaError_t back = cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) f->hand = nullptr;
            else e = back;
        }
        if (e != cudaSuccess) (void)cudaGetLastError();
        if (!f->hand) return;                  /* the run goes without */
    }
    R.hand.ctl = f->scratch + 3;
    R.hand.rec = f->hand;
    R.hand.lanes = pt_hand_lanes(R.np, f->precision);
    R.hand.cap = pt_hand_cap();
}

int run_impl(int32_t method, int64_t np, int32_t m, const pt_fields *f,
                    const double *params, const double *d_time, double *d_state, int64_t *d_cnt,
                    int32_t *d_status, void *d_carry, const pt_options *opt, cudaStream_t s, bool fresh)
{
    if (!f) return set_err(PT_ERR_ARG, "fields handle is NULL%s");
    if (np > 0 && (!d_time || !d_state || !d_cnt)) return set_err(PT_ERR_ARG, "NULL buffer%s");
    PtRun R;
    int rc = prepare_run(method, np, m, shape_of(f), params, opt, R);
    if (rc != PT_OK) return rc;
    attach_fields(f, R);
    R.time = d_time;
    R.state = d_state;
    R.cnt = d_cnt;
    R.status = d_status;
    R.carry = static_cast<unsigned char *>(d_carry);
    R.fresh = fresh || !d_carry;
    R.queue = f->scratch;
    R.flags = reinterpret_cast<int32_t *>(f->scratch + 1);
    if (R.minb == 0 || R.block == 0) {
        const int t = tuned_slot(method, f, R).load(std::memory_order_relaxed);
        if (R.minb == 0) R.minb = (t & 0xff) ? (t & 0xff) : PT_MINB_DEFAULT;
        if (R.block == 0) R.block = (t >> 8) ? (t >> 8) : PT_BLOCK_DEFAULT;
    }

    attach_hand(f, R);

    cudaError_t e;
    if (d_status && np > 0) {
        e = cudaMemsetAsync(d_status, 0xff, (size_t)np * sizeof(int32_t), s);
        if (e != cudaSuccess) return cuda_err(e, "status reset");
    }
    e = cudaMemsetAsync(f->scratch, 0, 5 * sizeof(unsigned long long), s);
    if (e != cudaSuccess) return cuda_err(e, "scratch reset");
    e = launch_run(method, f, R, s);
    if (e != cudaSuccess) return cuda_err(e, "kernel launch");
    return PT_OK;
}

}  // namespace pt_internal

extern "C" int pt_autotune(int32_t method, int64_t np, int32_t m, const pt_fields *f,
                           const double params[17], const double *d_time, const double *d_state,
                           const pt_options *opt, int64_t sample, void *stream, int32_t chosen[2],
                           double ms_out[9])
{
    if (!f) return set_err(PT_ERR_ARG, "fields handle is NULL%s");
    if (np < 1 || !d_time || !d_state) return set_err(PT_ERR_ARG, "autotune needs np >= 1 and buffers%s");
    PtRun R;
    int rc = prepare_run(method, np, m, shape_of(f), params, opt, R);
    if (rc != PT_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return cuda_err(e, "pt_autotune");
    const int64_t dflt = (int64_t)sms * 4 * 128 * 2;
    const int64_t want = sample < 0 ? np : (sample == 0 ? dflt : sample);
    const int64_t ns = np < want ? np : want;
    const bool windowed = opt && opt->t_stop > 0.0;   /* a real window, else an attempt cap */
    const int32_t mt = m < 2 ? m : 2;
    double *t_state = nullptr;
    int64_t *t_cnt = nullptr;
    float *t_rec = nullptr;            /* a record header with no room: counted, not written */
    cudaEvent_t ev[2] = { nullptr, nullptr };
    static const int kBlocks[3] = { 64, 128, 256 };
    double ms[9];
    for (int v = 0; v < 9; ++v) ms[v] = -1.0;
    e = cudaMalloc(&t_state, (size_t)ns * mt * 8 * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&t_cnt, (size_t)ns * 3 * sizeof(int64_t));
    if (e == cudaSuccess && R.rec) e = cudaMalloc(&t_rec, 16);
    if (e == cudaSuccess && t_rec) e = cudaMemsetAsync(t_rec, 0, 16, s);
    if (e == cudaSuccess) e = cudaEventCreate(&ev[0]);
    if (e == cudaSuccess) e = cudaEventCreate(&ev[1]);
    R.np = ns;
    R.m = mt;
    R.time = d_time;
    R.state = t_state;
    R.cnt = t_cnt;
    R.status = nullptr;
    R.carry = nullptr;
    R.fresh = 1;
    R.order = nullptr;
    R.rec = t_rec;
    R.rec_cap = 0;
    attach_fields(f, R);
    R.queue = f->scratch;
    R.flags = reinterpret_cast<int32_t *>(f->scratch + 1);
    /* Variants are of the machine with one lane per particle, and the choice is for
     * the runs that start on it: a smaller sample is timed there too, to its end. */
    attach_hand(f, R);
    R.few = 0;
    if (!windowed && !(opt && opt->max_steps > 0)) R.max_steps = 32;
    /* One trial of variant (minb, block index) on fresh copies of the states. */
    auto trial = [&](int minb, int bi, bool keep) {
        R.minb = minb;
        R.block = kBlocks[bi];
        e = cudaMemcpy2DAsync(t_state, (size_t)mt * 64, d_state, (size_t)m * 64, 64, (size_t)ns,
                              cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) e = cudaMemsetAsync(f->scratch, 0, 5 * sizeof(unsigned long long), s);
        if (e == cudaSuccess) e = cudaEventRecord(ev[0], s);
        if (e == cudaSuccess) e = launch_run(method, f, R, s);
        if (e == cudaSuccess) e = cudaEventRecord(ev[1], s);
        if (e == cudaSuccess) e = cudaEventSynchronize(ev[1]);
        float t = 0.0f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&t, ev[0], ev[1]);
        if (e == cudaSuccess && keep) ms[(minb - 2) * 3 + bi] = t;
    };
    /* Coordinate search: the register cap (2, 3, 4 resident 128-thread
     * blocks) at 128 threads per block, then 64 and 256 threads per block at
     * the best cap.  Short attempt-capped trials get a warm-up round; window
     * trials last long enough that the first launch's set-up does not
     * matter. */
    int best_m = 3, best_b = 1;
    for (int round = windowed ? 1 : 0; round < 2 && e == cudaSuccess; ++round)
        for (int v = 0; v < 3 && e == cudaSuccess; ++v) trial(2 + v, 1, round == 1);
    for (int v = 0; v < 3; ++v)
        if (ms[v * 3 + 1] >= 0.0 && ms[v * 3 + 1] < ms[(best_m - 2) * 3 + 1]) best_m = 2 + v;
    for (int bi = 0; bi < 3 && e == cudaSuccess; bi += 2) trial(best_m, bi, true);
    for (int bi = 0; bi < 3; ++bi) {
        const double t = ms[(best_m - 2) * 3 + bi];
        if (t >= 0.0 && t < ms[(best_m - 2) * 3 + best_b]) best_b = bi;
    }
    if (ev[0]) cudaEventDestroy(ev[0]);
    if (ev[1]) cudaEventDestroy(ev[1]);
    cudaFree(t_state);
    cudaFree(t_cnt);
    cudaFree(t_rec);
    if (e != cudaSuccess) return cuda_err(e, "pt_autotune");
    R.minb = 0;
    tuned_slot(method, f, R).store(best_m | (kBlocks[best_b] << 8), std::memory_order_relaxed);
    if (chosen) {
        chosen[0] = best_m;
        chosen[1] = kBlocks[best_b];
    }
    if (ms_out)
        for (int v = 0; v < 9; ++v) ms_out[v] = ms[v];
    return PT_OK;
}

/* Access for the no-allocation entry point (pt_noalloc.cu). */
int pt_prepare_run_public(int32_t method, int64_t np, int32_t m, const int32_t dm[3],
                          int32_t precision, int32_t has_j, const double *params,
                          const pt_options *opt, PtRun &R)
{
    RunShape g;
    for (int i = 0; i < 3; ++i) g.dm[i] = dm[i];
    g.precision = precision;
    g.has_j = has_j;
    return prepare_run(method, np, m, g, params, opt, R);
}

void pt_set_last_error(const char *msg) { snprintf(g_err, sizeof g_err, "%s", msg); }

/* Launch-parameter echo: out (device, 8 doubles) = what the kernel receives;
 * host_out (host, 2 doubles) = host sizeof(PtRun), offsetof(tend). */
extern "C" int pt_debug_echo(int32_t method, int64_t np, int32_t m, const int32_t dm[3],
                             int32_t precision, int32_t has_j, const double params[17],
                             const pt_options *opt, double *d_out, double *host_out)
{
    RunShape g;
    for (int i = 0; i < 3; ++i) g.dm[i] = dm[i];
    g.precision = precision;
    g.has_j = has_j;
    PtRun R;
    int rc = prepare_run(method, np, m, g, params, opt, R);
    if (rc != PT_OK) return rc;
    host_out[0] = (double)sizeof(PtRun);
    host_out[1] = (double)offsetof(PtRun, tend);
    cudaError_t e = pt_launch_echo_exact(R, d_out, (cudaStream_t)0);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_debug_echo");
}

extern "C" int pt_debug_unpack(int32_t method, int64_t np, int32_t m, const int32_t dm[3],
                               int32_t precision, int32_t has_j, const double params[17],
                               const pt_options *opt, double out[8])
{
    if (!dm || !out) return set_err(PT_ERR_ARG, "NULL argument%s");
    RunShape g;
    for (int i = 0; i < 3; ++i) g.dm[i] = dm[i];
    g.precision = precision;
    g.has_j = has_j;
    PtRun R;
    int rc = prepare_run(method, np, m, g, params, opt, R);
    if (rc != PT_OK) return rc;
    out[0] = R.tend;
    out[1] = R.tmx;
    out[2] = R.expo;
    out[3] = (double)R.unit_map;
    out[4] = (double)R.budget_ns * 1e-9;
    out[5] = (double)R.max_steps;
    out[6] = R.eta;
    out[7] = (double)R.open_x;
    return PT_OK;
}

extern "C" int pt_run_device(int32_t method, int64_t np, int32_t m, const pt_fields *f,
                             const double params[17], const double *d_time, double *d_state,
                             int64_t *d_cnt, int32_t *d_status, void *d_carry,
                             const pt_options *opt, void *stream)
{
    return run_impl(method, np, m, f, params, d_time, d_state, d_cnt, d_status, d_carry, opt,
                    (cudaStream_t)stream);
}

extern "C" int pt_run_check(const pt_fields *f)
{
    if (!f) return set_err(PT_ERR_ARG, "fields handle is NULL%s");
    unsigned long long w[2] = { 0, 0 };             /* flags (2 x int32), out-of-range count */
    cudaError_t e = cudaMemcpy(w, f->scratch + 1, sizeof w, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_err(e, "pt_run_check");
    int32_t flags[2];
    memcpy(flags, &w[0], sizeof flags);
    if (w[1]) {
        snprintf(g_err, sizeof g_err, "%llu index(es) out of range (gathers outside the field records or queue-order entries outside [0, np))", w[1]);
        return PT_ERR_BOUNDS;
    }
    if (flags[0]) return set_err(PT_ERR_TIMEOUT, "time budget expired%s");
    if (flags[1]) {
        snprintf(g_err, sizeof g_err, "%d particle(s) ended with a negative status", flags[1]);
        return PT_ERR_PARTICLE;
    }
    return PT_OK;
}

extern "C" int32_t pt_tableau(int32_t which, double *out)
{
    using namespace pt_tab;
    if (which == 1) {
        const double v[37] = {
            CK_B2_1, 0, 0, 0, 0,
            CK_B3_1, CK_B3_2, 0, 0, 0,
            CK_B4_1, CK_B4_2, CK_B4_3, 0, 0,
            CK_B5_1, CK_B5_2, CK_B5_3, CK_B5_4, 0,
            CK_B6_1, CK_B6_2, CK_B6_3, CK_B6_4, CK_B6_5,
            CK_C1, CK_C2, CK_C3, CK_C4, CK_C5, CK_C6,
            CK_D1, CK_D2, CK_D3, CK_D4, CK_D5, CK_D6 };
        if (out) memcpy(out, v, sizeof v);
        return 37;
    }
    if (which == 2) {
        const double v[] = {
            A0201, A0301, A0302, A0401, A0403, A0501, A0503, A0504, A0601, A0604, A0605,
            A0701, A0704, A0705, A0706, A0801, A0804, A0805, A0806, A0807,
            A0901, A0904, A0905, A0906, A0907, A0908,
            A1001, A1004, A1005, A1006, A1007, A1008, A1009,
            A1101, A1104, A1105, A1106, A1107, A1108, A1109, A1110,
            A1201, A1204, A1205, A1206, A1207, A1208, A1209, A1210, A1211,
            B01, B06, B07, B08, B09, B10, B11, B12, BH1, BH2, BH3,
            ER01, ER06, ER07, ER08, ER09, ER10, ER11, ER12 };
        if (out) memcpy(out, v, sizeof v);
        return (int32_t)(sizeof v / sizeof v[0]);
    }
    return 0;
}

__global__ void k_debug_pow(int64_t n, const double *x, const double *y, double *o)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        o[i] = pt_det_pow(x[i], y[i]);
}

extern "C" int pt_debug_pow(int64_t n, const double *d_x, const double *d_y, double *d_out,
                            void *stream)
{
    if (n <= 0) return PT_OK;
    if (!d_x || !d_y || !d_out) return set_err(PT_ERR_ARG, "NULL buffer%s");
    const int grid = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
    k_debug_pow<<<grid, 256, 0, (cudaStream_t)stream>>>(n, d_x, d_y, d_out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_debug_pow");
}

extern "C" int pt_debug_intpipe(int64_t n, const double *d_x, int32_t d, double *d_out,
                                int32_t *d_idx, void *stream)
{
    if (n < 0 || (n > 0 && (!d_x || !d_out || !d_idx))) return set_err(PT_ERR_ARG, "bad argument%s");
    const cudaError_t e = pt_launch_intpipe(n, d_x, d, d_out, d_idx, (cudaStream_t)stream);
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_debug_intpipe");
}

extern "C" int pt_debug_axis(int64_t n, const double *d_x, int32_t d, double *d_xd, int32_t *d_lr,
                             void *stream)
{
    if (n < 0 || d < 1 || (n > 0 && (!d_x || !d_xd || !d_lr))) return set_err(PT_ERR_ARG, "bad argument%s");
    const cudaError_t e = pt_launch_axis(n, d_x, d, d_xd, d_lr, (cudaStream_t)stream);
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_debug_axis");
}

extern "C" int pt_debug_qdiv(int64_t n, const double *d_a, const double *d_b, double *d_out,
                             void *stream)
{
    if (n < 0 || (n > 0 && (!d_a || !d_b || !d_out))) return set_err(PT_ERR_ARG, "bad argument%s");
    const cudaError_t e = pt_launch_qdiv(n, d_a, d_b, d_out, (cudaStream_t)stream);
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_debug_qdiv");
}

extern "C" int pt_debug_smul(int64_t n, const double *d_a, const double *d_b, double *d_out,
                             void *stream)
{
    if (n < 0 || (n > 0 && (!d_a || !d_b || !d_out))) return set_err(PT_ERR_ARG, "bad argument%s");
    const cudaError_t e = pt_launch_smul(n, d_a, d_b, d_out, (cudaStream_t)stream);
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_debug_smul");
}

extern "C" int pt_debug_ctl_pow(int64_t n, const double *d_x, const double *d_y, double *d_out,
                                void *stream)
{
    if (n < 0 || (n > 0 && (!d_x || !d_y || !d_out))) return set_err(PT_ERR_ARG, "bad argument%s");
    const cudaError_t e = pt_launch_ctl_pow(n, d_x, d_y, d_out, (cudaStream_t)stream);
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_debug_ctl_pow");
}

extern "C" int pt_debug_accel(const pt_fields *f, int64_t n, const double params[17],
                              const double *d_vec, double *d_acc, void *stream)
{
    if (!f || !params) return set_err(PT_ERR_ARG, "NULL argument%s");
    if (n <= 0) return PT_OK;
    PtRun R;
    RunShape g = shape_of(f);
    unpack_params(params, g, R);
    attach_fields(f, R);
    R.has_j = f->has_j;
    R.eta = 0.0;
    cudaError_t e;
    if (f->precision == PT_PREC_FP64)
        e = pt_launch_accel_exact(R, f->nc, n, d_vec, d_acc, (cudaStream_t)stream);
    else if (f->precision == PT_PREC_FP64_FMA)
        e = pt_launch_accel_fma(R, f->nc, n, d_vec, d_acc, (cudaStream_t)stream);
    else if (f->precision == PT_PREC_BF16)
        e = pt_launch_accel_mixed(R, f->nc16, 1, n, d_vec, d_acc, (cudaStream_t)stream);
    else
        e = pt_launch_accel_mixed(R, f->nc32, 0, n, d_vec, d_acc, (cudaStream_t)stream);
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_debug_accel");
}


extern "C" int pt_debug_face_params(int32_t method, float skip, float over)
{
    if (method != PT_METHOD_RK5 && method != PT_METHOD_DOP853)
        return set_err(PT_ERR_ARG, "pt_debug_face_params: unknown method%s");
    if (!(skip >= 0.0f && skip < 1.0f) || !(over > 0.0f && over < 1.0f))
        return set_err(PT_ERR_ARG, "pt_debug_face_params: skip in [0, 1), over in (0, 1)%s");
    g_face_skip[method == PT_METHOD_DOP853] = skip;
    g_face_over[method == PT_METHOD_DOP853] = over;
    return PT_OK;
}

extern "C" int pt_debug_face_cap(const pt_fields *f, int32_t method, int64_t n,
                                 const double params[17], const double *d_si, const double *d_h,
                                 double *d_out, void *stream)
{
    if (!f || !params) return set_err(PT_ERR_ARG, "NULL argument%s");
    if (method != PT_METHOD_RK5 && method != PT_METHOD_DOP853)
        return set_err(PT_ERR_ARG, "pt_debug_face_cap: unknown method%s");
    if (n <= 0) return PT_OK;
    if (!d_si || !d_h || !d_out) return set_err(PT_ERR_ARG, "NULL buffer%s");
    PtRun R;
    RunShape g = shape_of(f);
    unpack_params(params, g, R);
    attach_fields(f, R);
    R.face = 1;
    R.face_skip = g_face_skip[method == PT_METHOD_DOP853];
    R.face_over = g_face_over[method == PT_METHOD_DOP853];
    const cudaError_t e = pt_launch_face_cap(R, n, d_si, d_h, d_out, (cudaStream_t)stream);
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_debug_face_cap");
}
