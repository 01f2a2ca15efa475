/*
 * pt_common.cuh -- definitions shared by the kernels and the C ABI.
 *
 * Device data layout (all in HBM, written once per field handle):
 *   FP64 field records: for node (i,j,k), x fastest, one record of NC doubles
 *     { Ux, Uy, Uz, Bx, By, Bz }            NC = 6  (48 B, 3 x 16-B loads)
 *     { Ux, Uy, Uz, Bx, By, Bz, Jx, Jy, Jz, 0 } NC = 10 (80 B, with eta J)
 *   so one trilinear corner is 2-3 contiguous 32-B sectors instead of the 6
 *   separate planes of the reference layout uu(dm1,dm2,dm3,3), bb(...).
 *   Particle state keeps the reference layout state(8,m,np); each output
 *   sample is one aligned 64-B row.  The controller memory (carry) is SoA.
 */
#ifndef PT_COMMON_CUH
#define PT_COMMON_CUH

#include <stddef.h>
#include <stdint.h>
#include <cuda_runtime.h>

#include "../../include/particles_gb300.h"
#include "pt_detmath.h"
#include "pt_hand.h"
#include "pt_smul.h"

/* Particles handed from the lane-per-particle machine to the eight-lane one
 * (pt_coop.cuh) when a launch runs out of queued particles: ctl[0] counts the
 * records (pt_hand.h), ctl[1] is the head they are taken from; a record holds a
 * particle between two attempts. */
#define PT_HAND_WORDS 22
/* 16 warps on each of 152 SMs (the kernels' register counts allow no more) with
 * 12 particles each, or the warps of 240 particles per SM with 24 each; a warp
 * whose particles do not fit any more keeps them */
#define PT_HAND_CAP 32768
struct PtHand {
    unsigned long long *ctl;  /* 2 words, zeroed before a launch; NULL: no hand-over */
    double *rec;              /* PT_HAND_WORDS words per record */
    int lanes;                /* lanes a warp still has at work when it hands over */
    int cap;                  /* records that fit */
};

/* Everything a particle-integration kernel reads, by value in the launch. */
struct PtRun {
    /* params(1:17) unpacked as integrations.F90:103-118,330-346 */
    double qom, vun, tmx, dtm, atol, rtol, fcmn, fcmx, safe, beta, expo;
    double xl[3], xs[3];
    /* grid */
    double inv_dm[3], dmr[3];
    double gsx[3], gox[3];  /* node coordinate = x * gsx + gox = (x - xl) / xs * dm */
    double inv_vun;         /* 1 / vun, correctly rounded */
    double inv_xs[3];       /* 1 / xs, correctly rounded */
    double inv_atol;        /* 1 / atol, correctly rounded */
    float gsxf[3];          /* gsx rounded to FP32 (mixed precision) */
    float ivunf, qomf, etaf;
    int32_t dm[3];
    int32_t dm_mask[3];     /* dm - 1 when dm is a power of two, else 0 */
    int32_t unit_map;      /* xl == +0 and xs == 1: (pos - xl) / xs == pos exactly */
    int32_t fresh;         /* 1: no particle resumes from a carry */
    int32_t near;          /* 1: interpolate_near (the node at the cell's lower corner) */
    int32_t face;          /* 1: trial steps capped just past the next cell face */
    float face_skip;       /* faces within face_skip x the proposed step are crossed */
    float face_over;       /* overshoot past the capping face, in cells of the fastest axis */
    double noise;          /* PT_CTL_NOISE: rounding floor of the FP32 evaluation in the error
                              norm, per unit of the largest dt |f| component of a group
                              (positions, momenta); 0 = the reference's norm */
    /* extensions */
    double eta;
    int32_t has_j;
    int32_t open_x;
    double xo_lo, xo_hi;   /* open x faces: xl and xl + xs moved out by the margin */
    int64_t max_steps;
    double tend;           /* min(t_stop, tmx) */
    uint64_t budget_ns;
    /* sizes */
    int32_t m;
    int64_t np;
    int64_t few;           /* a run of at most this many starts on eight lanes per particle */
    /* device pointers */
    const double *fld;     /* FP64 records */
    const float *fld32;    /* FP32 brick records (mixed precision) */
    const uint4 *fld16;    /* BF16 brick records (PT_PREC_BF16) */
    const float *bscale;   /* per brick: FP32 offsets then scales of each component */
    int32_t nb[3];         /* bricks per axis, ceil(dm / 8) */
    const double *time;
    double *state;
    int64_t *cnt;
    int32_t *status;
    unsigned char *carry;  /* SoA carry or NULL */
    const int32_t *order;  /* queue order (particle index per queue slot) or NULL */
    const unsigned char *mlp;  /* learned-controller weight blob or NULL */
    float *rec;            /* accepted-step records (see PT_REC_*) or NULL */
    int64_t rec_cap;       /* record capacity */
    unsigned long long *queue;  /* work-queue head */
    int32_t *flags;        /* [0] time budget hit, [1] particles with negative status */
    int32_t minb;          /* launch variant: register cap of 2, 3 or 4 resident 128-thread
                              blocks per SM (255, 168, 128 registers) */
    int32_t block;         /* threads per block: 64, 128 or 256 (0 = 128) */
    unsigned long long *oob;  /* checked builds: count of out-of-range record indices */
    int64_t nrec;          /* records of the field store (index bound of the gathers) */
    int32_t *work;         /* per particle: attempts made in this run, or NULL */
    const int64_t *qlen;   /* ensembles: device queue length (else np) */
    const double *tstop;   /* ensembles: device window end (else tend) */
    PtHand hand;
};

/* Launch variant of an integrator: the same kernel compiled with the
 * register cap of 2, 3 or 4 resident 128-thread blocks per SM (255 / 168 /
 * 128 registers, __maxnreg__), launched with 64, 128 or 256 threads per
 * block (one particle per lane; the k rows in shared memory scale with the
 * block).  The register cap is the trade: more resident warps hide more
 * latency, fewer avoid spills (the learned controller's MLP, DOP853's k rows
 * in flight); the block size sets how shared memory and the register file
 * are carved into blocks.  Results do not depend on either. */
#define PT_MINB_DEFAULT 3
#define PT_BLOCK_DEFAULT 128
#define PT_BLOCK_MAX 256
#define PT_REGS_OF_MINB(b) ((b) == 2 ? 255 : (b) == 3 ? 168 : 128)

/* Carry (controller memory) SoA layout inside one buffer of 128*np bytes:
 *   double t[np], dt[np], errold[np], si[6][np], k1[6][np]; int32 n[np], flags[np]
 * flags bit0 = started, bit1 = the previous DOP853 attempt was rejected,
 * bit2 = k1 holds f(si), so a resumed particle needs no evaluation. */
struct PtCarry {
    double *t, *dt, *errold, *si, *k1;
    int32_t *n, *flags;
};

__host__ __device__ inline PtCarry pt_carry_view(unsigned char *base, int64_t np)
{
    PtCarry c;
    double *d = reinterpret_cast<double *>(base);
    c.t = d;
    c.dt = d + np;
    c.errold = d + 2 * np;
    c.si = d + 3 * np;
    c.k1 = d + 9 * np;
    int32_t *i = reinterpret_cast<int32_t *>(d + 15 * np);
    c.n = i;
    c.flags = i + np;
    return c;
}

#define PT_CARRY_BYTES_PER_PARTICLE 128

/* Accepted-step record buffer: a 16-byte header whose first 8 bytes count
 * the records written, then records of PT_REC_FLOATS floats: the nine
 * controller features at the start of an accepted step, log(dt) and
 * log(error ratio) of that step. */
#define PT_REC_NFEAT 9
#define PT_REC_FLOATS 11
#define PT_REC_HEADER_FLOATS 4

/* A double whose +, - and * are separately rounded operations issued as FMAs
 * (pt_fadd, pt_fsub, pt_fmul): the exact build's expressions keep the
 * reference's operand order and bits at the FMA rate of the FP64 pipe.  The
 * other builds write PtR too, as a plain double that contracts. */
#ifdef PT_EXACT
struct PtR {
    double v;
    __device__ __forceinline__ PtR() {}
    __device__ __forceinline__ PtR(double x) : v(x) {}
    __device__ __forceinline__ operator double() const { return v; }
};
#define PT_R_OP(op, fn)                                                                              \
    __device__ __forceinline__ PtR operator op(PtR a, PtR b) { return PtR(fn(a.v, b.v)); }           \
    __device__ __forceinline__ PtR operator op(PtR a, double b) { return PtR(fn(a.v, b)); }          \
    __device__ __forceinline__ PtR operator op(double a, PtR b) { return PtR(fn(a, b.v)); }
PT_R_OP(+, pt_fadd)
PT_R_OP(-, pt_fsub)
PT_R_OP(*, pt_fmul)
#undef PT_R_OP
#else
using PtR = double;
#endif

/* Fortran MIN/MAX with the NaN rule of the oracle (a NaN first operand
 * propagates). */
__device__ __forceinline__ double pt_max(double a, double b) { return (b > a) ? b : a; }
__device__ __forceinline__ double pt_min(double a, double b) { return (b < a) ? b : a; }

/* Comparisons on the integer pipe (an FP64 comparison takes an FP64 slot: with
 * them, the floors' hidden ones and the unused FP64 stage state gone, 262,144
 * particles RK5 FP32 25.6 -> 23.2 ms, DOP853 FP32 43.0 -> 39.8, RK5 exact
 * 57.5 -> 55.2).
 * pt_isnan for any x; pt_le: a <= b for b >= +0 and any a but NaN;
 * pt_max_pos: pt_max of magnitudes (a NaN may win where pt_max keeps a number). */
__device__ __forceinline__ bool pt_isnan(double x)
{
    const uint32_t h = (uint32_t)__double2hiint(x) & 0x7fffffffu;
    return h > 0x7ff00000u || (h == 0x7ff00000u && __double2loint(x) != 0);
}
__device__ __forceinline__ bool pt_le(double a, double b)
{
    return __double_as_longlong(a) <= __double_as_longlong(b);
}
__device__ __forceinline__ double pt_max_pos(double a, double b) { return pt_le(b, a) ? a : b; }

/* floor(xp) as a 0-based node index; dm (only reachable when x - floor(x)
 * rounds up to 1 for a tiny negative x, where the reference indexes past the
 * array) wraps to 0, NaN maps to 0.  Identical rule in the oracle.  q is an
 * integral double (a floor), read off its bits on the integer pipe. */
__device__ __forceinline__ int32_t pt_node_index(double q, int32_t d)
{
    const uint32_t hi = (uint32_t)__double2hiint(q), lo = (uint32_t)__double2loint(q);
    const uint32_t e = (hi >> 20) - 1023u;                 /* with the sign bit: > 30 if negative */
    if (e > 30u) return 0;                                 /* negative, < 1, huge, inf, NaN */
    const uint32_t m = (hi & 0xfffffu) | 0x100000u;
    const int32_t v = (int32_t)(e < 20u ? m >> (20u - e) : __funnelshift_l(lo, m, e - 20u));
    return v < d ? v : 0;
}

/* The exact build's cell of one axis (interpolations.F90:140-149): left and
 * right node of the scaled position x on d nodes, and the offset xd from the
 * left one.  The reference forms the right node from x + 1/d the way it forms
 * the left one from x; that is the left one's neighbour unless xd comes within
 * rounding of 0 or 1.  With |x| < 2^10 and d <= 2^18 the two ways' coordinates
 * differ from one node by at most d 2^-43 + d 2^-51 < 2^-24 (1/d rounded, x + 1/d
 * rounded, then the fraction and the product), so for xd in [2^-20, 1 - 2^-20) the
 * neighbour it is, at three FP64 operations, two floors and an index less per
 * axis; else the reference's own steps decide.  mask = d - 1 for a power of two
 * (else 0): the product by d is then an addition to the exponent. */
__device__ __forceinline__ void pt_axis_exact(double x, int32_t d, int32_t mask, double dmr,
                                              double inv_d, int32_t &l, int32_t &r, double &xd)
{
    auto times_d = [&](double fr) {
        const uint32_t hi = (uint32_t)__double2hiint(fr);
        if (mask && hi - 0x00100000u <= 0x3ff00000u - 0x00100000u)   /* normal, at most 1 */
            return __hiloint2double((int)(hi + ((uint32_t)__popc(mask) << 20)), __double2loint(fr));
        return pt_fmul(dmr, fr);
    };
    const double xp = times_d(pt_fsub(x, pt_floor(x)));
    const double pl = pt_floor(xp);
    l = pt_node_index(pl, d);
    xd = pt_fsub(xp, pl);
    const uint32_t hx = (uint32_t)__double2hiint(x) & 0x7fffffffu, hd = (uint32_t)__double2hiint(xd);
    if (hx < 0x40900000u && hd - 0x3eb00000u < 0x3feffffeu - 0x3eb00000u) {
        r = (l + 1 == d) ? 0 : l + 1;
    } else {
        const double xr = pt_fadd(x, inv_d);
        r = pt_node_index(pt_floor(times_d(pt_fsub(xr, pt_floor(xr)))), d);
    }
}

/* The IEEE division for quotients and reciprocals outside the fast forms'
 * domains, out of line: inlined at every use its own slow path makes the
 * compiler spill around code that physical states never reach. */
static __device__ __noinline__ double pt_div_cold(double a, double b) { return a / b; }

/* 1 / b correctly rounded: the hardware's approximation (20 bits and more),
 * two Newton steps to within an ulp, and a third that rounds correctly unless
 * the significand of b is all ones (P. Markstein, IBM J. Res. Develop. 34(1),
 * 1990, for fused multiply-add).  That case, and b whose reciprocal's steps could
 * leave the normal range (also zero, infinity, NaN), take the division.  Six
 * FP64 operations against about nine. */
__device__ __forceinline__ double pt_recip(double b)
{
    const uint32_t hi = (uint32_t)__double2hiint(b), e = (hi >> 20) & 0x7ffu;
    if (e - 24u > 1998u || ((hi & 0xfffffu) == 0xfffffu && __double2loint(b) == -1)) return pt_div_cold(1.0, b);
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = fma(fma(-b, y, 1.0), y, y);
    y = fma(fma(-b, y, 1.0), y, y);
    return fma(fma(-b, y, 1.0), y, y);
}

/* a / b correctly rounded from y = RN(1/b) (Markstein's quotient correction,
 * P. Markstein, IBM J. Res. Develop. 34(1), 1990): q0 = RN(a y) is within an
 * ulp of a / b, so the remainder r = a - b q0 is exact in one FMA and
 * RN(q0 + r y) is the correctly rounded quotient -- bit-identical to IEEE
 * a / b while the quotient and the remainder stay inside the normal range.
 * Three FP64 operations instead of a division sequence, and one reciprocal
 * serves every quotient by the same b.  Zeros, quotients outside [2^-960,
 * 2^961), dividends below 2^-907 (whose remainder could be subnormal),
 * infinities and NaN take the IEEE division (never on physical states; the
 * exponent tests run on the integer pipe). */
__device__ __forceinline__ double pt_qdiv(double a, double b, double y)
{
    const double q0 = pt_fmul(a, y);
    const uint32_t e = (uint32_t)((unsigned long long)__double_as_longlong(q0) >> 52) & 0x7ffu;
    const uint32_t ea = (uint32_t)((unsigned long long)__double_as_longlong(a) >> 52) & 0x7ffu;
    if (e - 63u > 1920u || ea < 116u) return pt_div_cold(a, b);
    const double r = fma(-b, q0, a);
    return fma(r, y, q0);
}

/* a * b on the integer pipes where pt_smul_bits covers it (normal operands,
 * normal product), else on the FPU: the correctly rounded product either
 * way, so the exact build may route any multiply here.  The FP64 pipe is the
 * GB300 kernels' bottleneck; this form spends integer-pipe issue slots,
 * which those kernels leave idle, instead. */
__device__ __forceinline__ double pt_smul(double a, double b)
{
    uint32_t rh, rl;
    if (pt_smul_bits((uint32_t)__double2hiint(a), (uint32_t)__double2loint(a),
                     (uint32_t)__double2hiint(b), (uint32_t)__double2loint(b), rh, rl))
        return __hiloint2double((int)rh, (int)rl);
    return __dmul_rn(a, b);
}

/* The integer-pipe product alone: `ok` is cleared when the operands or the
 * product lie outside pt_smul_bits' domain (the value is then meaningless
 * and the caller recomputes on the FPU).  No branch, so a run of such
 * products schedules as one straight-line block. */
__device__ __forceinline__ double pt_smul_raw(double a, double b, bool &ok)
{
    uint32_t rh, rl;
    ok &= pt_smul_bits((uint32_t)__double2hiint(a), (uint32_t)__double2loint(a),
                       (uint32_t)__double2hiint(b), (uint32_t)__double2loint(b), rh, rl);
    return __hiloint2double((int)rh, (int)rl);
}

__device__ __forceinline__ uint64_t pt_globaltimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

/* Checked builds (PT_CHECKED, the bounds-checking variant of the library):
 * every record index of a gather is tested against the store; an index out
 * of range is counted in P.oob and replaced by record 0, so the access stays
 * inside the allocation and the host reports the count (PT_ERR_BOUNDS).
 * Other builds compile the test away. */
#ifdef PT_CHECKED
__device__ __forceinline__ int64_t pt_chk(unsigned long long *oob, int64_t i, int64_t n)
{
    if (i < 0 || i >= n) {
        atomicAdd(oob, 1ULL);
        return 0;
    }
    return i;
}
#define PT_CHK(P, i, n) pt_chk((P).oob, (i), (n))
#else
#define PT_CHK(P, i, n) (i)
#endif

/* Internal "keep integrating" word of the step loops; distinct from every
 * PT_ST_* status (PT_ST_RUNNING is 1). */
#define PT_GO 0x7fff

/* Loop guard shared with the oracle: < 0 stops the particle before an attempt. */
__device__ __forceinline__ int32_t pt_attempt_guard(double t, double dt, int64_t attempts,
                                                    int64_t max_steps)
{
    if (max_steps > 0 && attempts >= max_steps) return PT_ST_STEP_LIMIT;
    if (pt_isnan(dt)) return PT_ST_NONFINITE;
    /* dt > 0, and t >= 0 moves: on the bits */
    if (pt_le(dt, 0.0) || __double_as_longlong(t + dt) == __double_as_longlong(t)) return PT_ST_DT_UNDERFLOW;
    return PT_GO;
}

/* Launchers implemented by the kernel translation units. */
struct PtLaunch {
    int grid, block;
    cudaStream_t stream;
};

/* Particles up to which a run goes to the eight-lane machine from the start,
 * PT_COOP_PER_SM per SM.  Exact build, one against eight lanes per particle:
 * 1,024 particles DOP853 11.8 / 3.6 ms, RK5 10.1 / 3.4 ms; 9,728 11.8 / 7.7
 * and 10.6 / 7.2; 12,160 (80 per SM) 11.8 / 9.4 and 10.6 / 8.6, where one lane
 * with hand-over takes 10.7 and 8.9; 16,384 11.8 / 12.2 and 10.7 / 11.4. */
#ifndef PT_COOP_PER_SM
#define PT_COOP_PER_SM 80
#endif
int pt_coop_sms();
int64_t pt_coop_max();                /* particles; pt_debug_machines may change both */
int pt_hand_cap();                    /* records of a hand-over list */
/* Lanes a warp still has at work when it hands over.  One lane per particle
 * costs a scheduler ~2,400 FP64 slots per DOP853 attempt for up to 32 particles,
 * eight lanes ~900 for 4: equal at about 11 where the schedulers are full.
 * Exact build, 65,536 particles, never / 4 / 8 / 12 / 16 / 24: DOP853 25.3 / 21.9
 * / 20.2 / 20.0 / 26.8 / 29.2 ms, RK5 21.4 / 18.3 / 17.3 / 17.2 / 23.9 / 26.0.
 * Where one warp per scheduler holds the whole run, the eight-lane machine's
 * shorter attempt counts instead.  12 / 16 / 20 / 24 lanes: exact DOP853 16,384
 * particles 9.5 / 8.9 / 8.9 / 8.9 ms, 20,001 10.6 / 10.1 / 10.1 / 10.3, 32,768
 * 11.5 / 11.4 / 11.9 / 12.3; FP32 DOP853 16,384 9.5 / 8.8 / 8.5 / 8.2, 32,768
 * 10.8 / 10.5 / 10.3 / 9.9. */
inline int pt_hand_lanes(int64_t np, int precision)
{
    const bool mixed = precision == PT_PREC_FP32 || precision == PT_PREC_BF16;
    return np <= (mixed ? 240 : 160) * (int64_t)pt_coop_sms() ? (mixed ? 24 : 20) : 12;
}

#define PT_DECLARE_FP64_LAUNCHERS(sfx)                                            \
    cudaError_t pt_launch_rk5_##sfx(const PtRun &P, int nc, cudaStream_t s);     \
    cudaError_t pt_launch_dp853_##sfx(const PtRun &P, int nc, cudaStream_t s);   \
    cudaError_t pt_launch_accel_##sfx(const PtRun &P, int nc, int64_t n,         \
                                      const double *vec, double *acc, cudaStream_t s); \
    cudaError_t pt_launch_echo_##sfx(const PtRun &P, double *out, cudaStream_t s);    \
    cudaError_t pt_launch_rk5_ens_##sfx(const PtRun *tab, int nmem, int nc, int minb, \
                                        int block, int64_t ntot, cudaStream_t s);   \
    cudaError_t pt_launch_dp853_ens_##sfx(const PtRun *tab, int nmem, int nc, int minb, \
                                          int block, int64_t ntot, cudaStream_t s);

PT_DECLARE_FP64_LAUNCHERS(exact)
PT_DECLARE_FP64_LAUNCHERS(fma)

/* Readies the exact kernels of a method for later runs without options (NC = 6). */
cudaError_t pt_ready_rk5(const PtRun &P, cudaStream_t s);
cudaError_t pt_ready_dp853(const PtRun &P, cudaStream_t s);

cudaError_t pt_launch_rk5_mixed(const PtRun &P, int nc, cudaStream_t s);
cudaError_t pt_launch_rk5_ens_mixed(const PtRun *tab, int nmem, int nc, int minb, int block,
                                    int64_t ntot, cudaStream_t s);
cudaError_t pt_launch_dp853_ens_mixed(const PtRun *tab, int nmem, int nc, int minb, int block,
                                      int64_t ntot, cudaStream_t s);
cudaError_t pt_launch_dp853_mixed(const PtRun &P, int nc, cudaStream_t s);
cudaError_t pt_launch_rk5_bf16(const PtRun &P, int nc, cudaStream_t s);
cudaError_t pt_launch_dp853_bf16(const PtRun &P, int nc, cudaStream_t s);
cudaError_t pt_launch_rk5_ens_bf16(const PtRun *tab, int nmem, int nc, int minb, int block,
                                   int64_t ntot, cudaStream_t s);
cudaError_t pt_launch_dp853_ens_bf16(const PtRun *tab, int nmem, int nc, int minb, int block,
                                     int64_t ntot, cudaStream_t s);
cudaError_t pt_launch_accel_mixed(const PtRun &P, int nc, int brick, int64_t n, const double *vec,
                                  double *acc, cudaStream_t s);

cudaError_t pt_launch_debug_pow(int64_t n, const double *x, const double *y, double *out,
                                cudaStream_t s);
cudaError_t pt_launch_smul(int64_t n, const double *a, const double *b, double *out,
                           cudaStream_t s);
cudaError_t pt_launch_qdiv(int64_t n, const double *a, const double *b, double *out,
                           cudaStream_t s);
cudaError_t pt_launch_ctl_pow(int64_t n, const double *x, const double *y, double *out,
                              cudaStream_t s);
cudaError_t pt_launch_face_cap(const PtRun &P, int64_t n, const double *si, const double *h,
                               double *out, cudaStream_t s);
cudaError_t pt_launch_axis(int64_t n, const double *x, int32_t d, double *xd, int32_t *lr,
                           cudaStream_t s);
cudaError_t pt_launch_intpipe(int64_t n, const double *x, int32_t d, double *out, int32_t *idx,
                              cudaStream_t s);

#endif /* PT_COMMON_CUH */
