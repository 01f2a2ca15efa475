/*
 * pt_coop.cuh -- the step machine with eight lanes per particle, for runs too
 * small to fill the GPU with one particle per lane.
 *
 * What bounds such a run is not throughput but the time of one attempt: a
 * GB300 scheduler takes one FP64 warp instruction every 64 cycles, whatever
 * its active lanes and its independent work, so a particle advances at the
 * count of FP64 instructions its warp issues, ~2,400 per DOP853 attempt
 * (170 us) in the lane-per-particle machine of pt_integrator.cuh.  Here a
 * group of eight lanes shares them:
 *   - lane c < 6 owns component c of the state and its k rows: stage sums,
 *     final combination, error terms and output rows are one component wide;
 *   - the axes' cell maps run side by side on lanes 0-2, the momenta's on
 *     lanes 3-5;
 *   - lane q gathers corner q's record and forms its products by the weight;
 *     a transpose through shared memory hands lane c the eight products of
 *     component c, which it adds in the reference's corner order;
 *   - the force runs on lanes 3-5 while lanes 0-2 divide by vun.
 * Every component sees the same operations on the same operands in the same
 * order as in pt_integrator.cuh, so a particle's bits do not depend on which
 * machine integrated it.  In the non-exact builds that includes which product
 * of a sum the compiler contracts there; where its choice is not the only one
 * it is written out here (tests/test_gpu_coop.py compares the two machines).
 */
#ifndef PT_COOP_CUH
#define PT_COOP_CUH

#include "pt_integrator.cuh"

namespace pt_sm {

constexpr int kGroup = 8;                 /* lanes per particle */

/* What every lane of a group knows about itself. */
struct Group {
    int gl;                               /* lane in the group */
    int c;                                /* component it owns (lanes 6, 7 idle along with 5) */
    int ax;                               /* axis of that component */
    unsigned mask;                        /* the group's lanes in its warp */
    __device__ __forceinline__ Group()
    {
        const int lane = threadIdx.x & 31;
        gl = lane & (kGroup - 1);
        c = gl < 6 ? gl : 5;
        ax = c < 3 ? c : c - 3;
        mask = 0xffu << (lane & ~(kGroup - 1));
    }
    template <class V> __device__ __forceinline__ V get(V v, int src) const
    {
        return __shfl_sync(mask, v, src, kGroup);
    }
};

/* k rows of the lane's component in shared memory. */
struct KOwn {
    double *base;
    int stride;
    __device__ __forceinline__ double &operator()(int row) const { return base[row * stride]; }
};

/* Shared memory per block: k rows, then the gather's transpose area (per
 * group NV rows of 8 products, rows padded to 9). */
template <int METHOD, class EV>
__host__ __device__ constexpr int coop_rows_bytes(int block)
{
    return Traits<METHOD>::ROWS * 8 * block + EV::kCoopRows * 9 * 8 * (block / kGroup);
}
/* ... and, with a learned controller, its weight blob. */
template <int METHOD, class EV>
__host__ __device__ constexpr int coop_smem_bytes(int block, bool learn)
{
    return coop_rows_bytes<METHOD, EV>(block) + (learn ? PT_MLP_BLOB_BYTES : 0);
}

template <int METHOD>
__device__ __forceinline__ void coop_open(const PtRun &P, const Group &G, const KOwn &K, Lane &L,
                                          double &si, int &how)
{
    const PtCarry C = pt_carry_view(P.carry, P.np);
    const int32_t fl = (P.carry != nullptr) ? C.flags[L.p] : 0;
    if (!(fl & 1)) {
        si = P.state[(int64_t)8 * P.m * L.p + G.c];
        L.t = 0.0; L.n = 1; L.errold = 1.0e-04; L.rejected = false;
        L.c0 = L.c1 = L.c2 = 0;
        L.w0 = 0;
        how = 0;
        return;
    }
    L.t = C.t[L.p]; L.dt = C.dt[L.p]; L.errold = C.errold[L.p]; L.n = C.n[L.p];
    L.rejected = (fl & 2) != 0;
    si = C.si[(int64_t)G.c * P.np + L.p];
    L.c0 = P.cnt[3 * L.p]; L.c1 = P.cnt[3 * L.p + 1]; L.c2 = P.cnt[3 * L.p + 2];
    L.w0 = (int32_t)L.c0;
    how = 1;
    if (fl & 4) {
        K(Traits<METHOD>::F1) = C.k1[(int64_t)G.c * P.np + L.p];
        how = 2;
    }
}

/* Takes over a particle that lane_hand left. */
template <int METHOD>
__device__ __forceinline__ void coop_take(const double *r, const Group &G, const KOwn &K, Lane &L,
                                          double &si, uint64_t &t_start, int &mi)
{
    const long long *w = reinterpret_cast<const long long *>(r);
    L.t = r[HandRec::T]; L.dt = r[HandRec::DT]; L.errold = r[HandRec::ERROLD];
    si = r[HandRec::SI + G.c];
    K(Traits<METHOD>::F1) = r[HandRec::K1 + G.c];
    L.c0 = w[HandRec::C0]; L.c1 = w[HandRec::C1]; L.c2 = w[HandRec::C2];
    L.p = w[HandRec::P];
    t_start = (uint64_t)w[HandRec::START];
    L.n = (int32_t)(uint32_t)w[HandRec::N_W0];
    L.w0 = (int32_t)(w[HandRec::N_W0] >> 32);
    L.rejected = (w[HandRec::FLAGS] & 1) != 0;
    mi = (int)(w[HandRec::FLAGS] >> 1);
}

template <int METHOD>
__device__ __forceinline__ void coop_close(const PtRun &P, const Group &G, const KOwn &K,
                                           const Lane &L, double si, int32_t st)
{
    const PtCarry C = pt_carry_view(P.carry, P.np);
    if (P.carry && G.gl < 6) {
        C.si[(int64_t)G.c * P.np + L.p] = si;
        C.k1[(int64_t)G.c * P.np + L.p] = K(Traits<METHOD>::F1);
    }
    if (G.gl != 0) return;
    P.cnt[3 * L.p] = L.c0;
    P.cnt[3 * L.p + 1] = L.c1;
    P.cnt[3 * L.p + 2] = L.c2;
    if (P.status) P.status[L.p] = st;
    if (P.work) P.work[L.p] = (int32_t)L.c0 - L.w0;
    if (P.carry) {
        C.t[L.p] = L.t; C.dt[L.p] = L.dt; C.errold[L.p] = L.errold; C.n[L.p] = L.n;
        C.flags[L.p] = 1 | (L.rejected ? 2 : 0) | 4;
    }
    if (st < 0) atomicAdd(P.flags + 1, 1);
    if (st == PT_ST_TIMEOUT) atomicExch(P.flags, 1);
}

/* dti_guess, as dti_finish. */
__device__ __forceinline__ double coop_dti(const PtRun &P, const Group &G, int iord, double si,
                                           double ki)
{
    const double sr = P.atol + P.rtol * fabs(si);
    const double q0 = si / sr, q1 = ki / sr;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) { const double q = G.get(q0, i); s0 = s0 + q * q; }
#pragma unroll
    for (int i = 0; i < 6; ++i) { const double q = G.get(q1, i); s1 = s1 + q * q; }
    const double d0 = sqrt(s0 / 6.0);
    const double d1 = sqrt(s1 / 6.0);
    double dti;
    if (pt_min(d0, d1) < 1.0e-10) dti = 1.0e-06;
    else dti = 1.0e-01 * (d0 / d1);
    const double sf = si + dti * ki;
    const double q2 = (sf - si) / sr;
    double s2 = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) { const double q = G.get(q2, i); s2 = s2 + q * q; }
    const double d2 = pt_max(d1, sqrt(s2 / 6.0) / dti);
    double dtf;
    if (d2 <= 1.0e-15) dtf = pt_max(1.0e-06, 1.0e-03 * dti);
    else dtf = pt_det_pow(1.0e-02 / d2, 1.0 / (double)iord);
    return pt_min(pt_min(1.0e+02 * dti, dtf), P.dtm);
}

/* One output row, as dense_row: lane c < 6 writes component c, lane 6 gamma,
 * lane 7 the step. */
__device__ __forceinline__ void coop_row(const Group &G, double t, double dt, double tn, double si,
                                         double sf, double ka, double kb, bool scale, double *row)
{
    const double fr = (t - tn) / dt;
    const double fl = 1.0 - fr;
    const double ds = sf - si;
    const double a = scale ? dt * ka : ka;
    const double b = scale ? dt * kb : kb;
#ifdef PT_EXACT
    const double st = fr * si + fl * sf + fl * fr * ((a - ds) * fr + (ds - b) * fl);
#else
    /* which of two products contracts as in dense_row */
    const double in = scale ? fma(a - ds, fr, __dmul_rn(ds - b, fl)) : (a - ds) * fr + (ds - b) * fl;
    const double st = fr * si + fl * sf + fl * fr * in;
#endif
    const double s3 = G.get(st, 3), s4 = G.get(st, 4), s5 = G.get(st, 5);
    const double gam = sqrt(s3 * s3 + s4 * s4 + s5 * s5 + 1.0);
    row[G.gl] = G.gl < 6 ? st : (G.gl == 6 ? gam : dt);
}

/* s = si + d with the increment d = h k.  The non-exact builds' lane-per-
 * particle machine contracts the two where the increment itself is not used
 * (the FMA build), and rounds it where it is (DELTA); so do these lanes. */
template <bool DELTA>
__device__ __forceinline__ void coop_step(double h, double k, double si, double &s, double &d)
{
#ifdef PT_EXACT
    const PtR x = PtR(h) * k;
    d = x;
    s = si + x;
#else
    d = __dmul_rn(h, k);
    s = DELTA ? __dadd_rn(si, d) : fma(h, k, si);   /* (unused, and dropped, in DELTA stages) */
#endif
}

/* The lane's component of the stage state and its increment, as stage_state. */
template <int METHOD, bool DELTA>
__device__ __forceinline__ void coop_stage(int j, const KOwn &K, double si, double dt, double &ss,
                                           double &dl)
{
    if (METHOD == PT_METHOD_DOP853) {
        const Stage &S = kDop[j];
        if (j == 1) {
            coop_step<DELTA>(PtR(dt) * S.a[0], K(0), si, ss, dl);
        } else {
            PtR acc = PtR(S.a[0]) * K(S.r[0]);
            /* the next term's coefficient and row are on their way during this one */
            double a = S.a[1], k = K(S.r[1]);
            for (int i = 1; i < S.n; ++i) {
                const double an = S.a[i + 1], kn = K(S.r[i + 1]);
                acc = acc + PtR(a) * k;
                a = an;
                k = kn;
            }
            coop_step<DELTA>(dt, acc, si, ss, dl);
        }
    } else {
        const Stage &S = kCk[j];
        if (DELTA) {
            double acc = S.a[0] * K(S.r[0]);
            double a = S.a[1], k = K(S.r[1]);
            for (int i = 1; i < S.n; ++i) {
                const double an = S.a[i + 1], kn = K(S.r[i + 1]);
                acc = acc + a * k;
                a = an;
                k = kn;
            }
            dl = acc;
        } else {
            PtR acc = si;
            double a = S.a[0], k = K(S.r[0]);
            for (int i = 0; i < S.n; ++i) {
                const double an = S.a[i + 1], kn = K(S.r[i + 1]);
                acc = acc + PtR(a) * k;
                a = an;
                k = kn;
            }
            ss = acc;
        }
    }
}

#ifndef PT_EXACT
/* The largest |v| of the lane's group of components (positions, momenta). */
__device__ __forceinline__ double coop_group_max(const Group &G, double v)
{
    const int b = G.c < 3 ? 0 : 3;
    const double a = fabs(v);
    const double v0 = G.get(a, b), v1 = G.get(a, b + 1), v2 = G.get(a, b + 2);
    return pt_max_pos(v0, pt_max_pos(v1, v2));
}
#endif

/* Final combination and error norm, as finish_attempt: sf, dsf of the lane's
 * component; the norm on every lane. */
template <int METHOD, bool DELTA>
__device__ __forceinline__ double coop_finish(const PtRun &P, const Group &G, const KOwn &K,
                                              double si, double dt, double &sf, double &dsf)
{
    if (METHOD == PT_METHOD_DOP853) {
        const PtR k4 = PtR(B01) * K(0) + PtR(B06) * K(5) + PtR(B07) * K(6) + PtR(B08) * K(7)
                     + PtR(B09) * K(8) + PtR(B10) * K(9) + PtR(B11) * K(1) + PtR(B12) * K(2);
        coop_step<DELTA>(dt, k4, si, sf, dsf);
        double sr = PtR(P.atol) + PtR(P.rtol) * pt_max_pos(fabs(si), fabs(sf));
        const PtR e3 = k4 - PtR(BH1) * K(0) - PtR(BH2) * K(8) - PtR(BH3) * K(2);
        const PtR e5 = PtR(ER01) * K(0) + PtR(ER06) * K(5) + PtR(ER07) * K(6) + PtR(ER08) * K(7)
                     + PtR(ER09) * K(8) + PtR(ER10) * K(9) + PtR(ER11) * K(1) + PtR(ER12) * K(2);
#ifdef PT_EXACT
        const double ysr = pt_recip(sr);
        const PtR q3 = pt_qdiv(e3, sr, ysr), q5 = pt_qdiv(e5, sr, ysr);
        const double t3 = q3 * q3, t5 = q5 * q5;       /* squared before they are handed round */
#else
        if (P.noise != 0.0) sr = fma(P.noise, coop_group_max(G, dsf), sr);
        const double ysr = pt_rcp(sr);
        const double t3 = e3 * ysr, t5 = e5 * ysr;
#endif
        /* the two sums side by side: err3 on even lanes, err5 on odd ones */
        PtR s = 0.0;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const double a = G.get(t3, i), b = G.get(t5, i);
            const double v = (G.gl & 1) ? b : a;
#ifdef PT_EXACT
            s = (i == 0) ? PtR(v) : s + v;
#else
            s = (i == 0) ? v : (i == 1) ? fma(s, s, __dmul_rn(v, v)) : fma(v, v, s);
#endif
        }
        const PtR err3 = G.get((double)s, 0), err5 = G.get((double)s, 1);
        const double deno = err5 + 1.0e-02 * err3;
#ifdef PT_EXACT
        const double num = PtR(fabs(dt)) * err5;
        return num / sqrt(pt_le(deno, 0.0) ? 6.0 : (double)(PtR(6.0) * deno));
#else
        if (pt_le(deno, 1.0e-300))
            return (deno <= 0.0) ? fabs(dt) * err5 * 0.40824829046386307
                                 : fabs(dt) * err5 / sqrt(6.0 * deno);
        return fabs(dt) * err5 * pt_rsqrt(6.0 * deno);
#endif
    } else {
#ifdef PT_EXACT
        PtR a = 0.0, e = 0.0;
        a = a + PtR(CK_C1) * K(0); a = a + PtR(CK_C2) * K(1); a = a + PtR(CK_C3) * K(2);
        a = a + PtR(CK_C4) * K(3); a = a + PtR(CK_C5) * K(4); a = a + PtR(CK_C6) * K(5);
        e = e + PtR(CK_D1) * K(0); e = e + PtR(CK_D2) * K(1); e = e + PtR(CK_D3) * K(2);
        e = e + PtR(CK_D4) * K(3); e = e + PtR(CK_D5) * K(4); e = e + PtR(CK_D6) * K(5);
        const double sr = PtR(fabs(si)) + fabs(K(0)) + 2.2250738585072014e-308;
#else
        const double a = CK_C1 * K(0) + CK_C3 * K(2) + CK_C4 * K(3) + CK_C6 * K(5);
        const double e = CK_D1 * K(0) + CK_D3 * K(2) + CK_D4 * K(3) + CK_D5 * K(4) + CK_D6 * K(5);
        double sr = fabs(si) + fabs(K(0));
        if (P.noise != 0.0) sr += __dmul_rn(P.noise, coop_group_max(G, K(0)));
        if (__double_as_longlong(sr) == 0) sr = 2.2250738585072014e-308;
#endif
        dsf = a;
        sf = si + a;
        /* the largest |e / sr| by its bits (NaN above infinity: it propagates) */
        const double r = PT_DIV((double)e, sr);
        const unsigned long long q =
            (unsigned long long)__double_as_longlong(r) & 0x7fffffffffffffffULL;
        unsigned long long del = G.get(q, 0);
#pragma unroll
        for (int i = 1; i < 6; ++i) {
            const unsigned long long v = G.get(q, i);
            del = v > del ? v : del;
        }
#ifdef PT_EXACT
        return pt_qdiv(__longlong_as_double((long long)del), P.atol, P.inv_atol);
#else
        return PT_DIV(__longlong_as_double((long long)del), P.atol);
#endif
    }
}

/* from_queue: particles come from the work queue; then, and otherwise only,
 * from the hand-over list of the launch before (complete: that launch is over). */
template <int METHOD, class EV, bool LEARN, bool ENS = false>
__device__ __forceinline__ void run_coop(const Members<ENS> &MB, bool from_queue)
{
    using T = Traits<METHOD>;
    extern __shared__ double pt_ksm[];
    const Group G;
    const KOwn K{ pt_ksm + threadIdx.x, (int)blockDim.x };
    double *const tr = pt_ksm + T::ROWS * blockDim.x + (threadIdx.x / kGroup) * (EV::kCoopRows * 9);
    int mi = 0;
#define PT_Q (MB.q(mi))
    unsigned char *const blob = reinterpret_cast<unsigned char *>(pt_ksm) + coop_rows_bytes<METHOD, EV>(blockDim.x);
    if (LEARN) (void)pt_mlp_load(PT_Q.mlp, blob);
    uint64_t t_start = pt_globaltimer();
    const PtHand H = MB.q(0).hand;
    const unsigned long long handed = H.ctl ? pt_hand_written(H.ctl[0], H.cap) : 0ULL;
    Lane L;
    L.p = 0; L.t = 0.0; L.dt = 0.0; L.errold = 0.0; L.tnext = 0.0; L.n = 0;
    L.rejected = false; L.c0 = L.c1 = L.c2 = 0; L.w0 = 0;
    double si = 0.0;
    typename EV::CoopOrigin O;
    bool active = false, drained = false, dry = !from_queue;
    int j = 0;
    for (;;) {
        double pt = si, dl = 0.0;
        bool need = false, fresh = false, handed_over = false;
        int mode = M_IDLE;
        double q = 0.0;
        if (j == 0) {
            if (active) {
                q = coop_finish<METHOD, EV::kDelta>(PT_Q, G, K, si, L.dt, pt, dl);
                if (pt_isnan(q)) {
                    coop_close<METHOD>(PT_Q, G, K, L, si, PT_ST_NONFINITE);
                    active = false;
                } else if (pt_le(q, 1.0)) {
                    mode = M_ACCEPT;
                    need = true;
                } else {
                    mode = M_REJECT;
                }
            }
            if (!active && !drained) {
                unsigned long long qi = 0;
                bool got = false;
                while (!dry && !got && mi < MB.count()) {
                    if (G.gl == 0) qi = atomicAdd(PT_Q.queue, 1ULL);
                    qi = G.get(qi, 0);
                    got = (int64_t)qi < MB.queue_len(mi);
                    if (!got) {
                        ++mi;
                    } else if (PT_Q.order) {
                        const int64_t p = (int64_t)PT_Q.order[qi];
                        if (p < 0 || p >= PT_Q.np) {
                            if (PT_Q.oob && G.gl == 0) atomicAdd(PT_Q.oob, 1ULL);
                            got = false;
                        }
                    }
                }
                if (!got) {
                    dry = true;
                    mi = 0;
                    if (handed && G.gl == 0) qi = atomicAdd(H.ctl + 1, 1ULL);
                    qi = G.get(qi, 0);
                    if (handed && qi < handed) {
                        const double *const r = H.rec + qi * PT_HAND_WORDS;
                        /* (the next tail tries again after a slot marked as empty) */
                        if (reinterpret_cast<const long long *>(r)[HandRec::P] >= 0) {
                            coop_take<METHOD>(r, G, K, L, si, t_start, mi);
                            mode = M_READY;
                            handed_over = true;
                            active = true;
                        }
                    } else {
                        drained = true;
                    }
                } else {
                    L.p = PT_Q.order ? (int64_t)PT_Q.order[qi] : (int64_t)qi;
                    int how;
                    coop_open<METHOD>(PT_Q, G, K, L, si, how);
                    if (how == 2) {
                        mode = M_READY;
                    } else {
                        mode = M_INIT;
                        need = true;
                        pt = si;
                        dl = 0.0;
                        EV::coop_begin(PT_Q, G, si, O);
                    }
                    active = true;
                    fresh = (how == 0);
                }
            }
        } else if (active) {
            coop_stage<METHOD, EV::kDelta>(j, K, si, L.dt, pt, dl);
            need = true;
        }

        double a = 0.0;
        if (need) a = EV::coop_f(PT_Q, G, tr, pt, dl, O);       /* the one evaluation site */

        if (j != 0) {
            if (active) {
                if (METHOD == PT_METHOD_DOP853) K(kDop[j].dst) = a;
                else K(kCk[j].dst) = PtR(L.dt) * a;
            }
        } else {
            const double dt = L.dt;
            const bool was_rejected = L.rejected;
            double fpow = 0.0;
            if (mode == M_ACCEPT || mode == M_REJECT) {
                const double y = (METHOD == PT_METHOD_DOP853) ? PT_Q.expo
                               : (mode == M_ACCEPT ? -0.20 : -0.25);
                fpow = PT_Q.safe * pt_ctl_pow(q, y);
            }
            if (mode == M_ACCEPT) {
                L.t = L.t + dt;
                while (L.n < PT_Q.m && L.t >= L.tnext) {
                    double *row = PT_Q.state + (int64_t)8 * ((int64_t)L.n + (int64_t)PT_Q.m * L.p);
                    if (METHOD == PT_METHOD_DOP853)
                        coop_row(G, L.t, dt, L.tnext, si, pt, K(0), a, true, row);
                    else
                        coop_row(G, L.t, dt, L.tnext, si, pt, K(0), K(5), false, row);
                    L.n++;
                    next_time(PT_Q, L);
                }
                si = pt;
                K(T::F1) = a;
                L.c1++;
                if (METHOD == PT_METHOD_DOP853) {
                    double dtn = pt_max(PT_Q.fcmn, fpow * pt_det_pow(L.errold, PT_Q.beta));
                    dtn = L.rejected ? dt * pt_min(dtn, 1.0) : dt * pt_min(dtn, PT_Q.fcmx);
                    L.errold = pt_max(q, 1.0e-04);
                    L.rejected = false;
                    L.dt = dtn;
                } else {
                    L.dt = dt * pt_min(PT_Q.fcmx, fpow);
                }
                L.c0++;
                L.dt = pt_min(L.dt, PT_Q.dtm);
                if (escaped_x(PT_Q, G.get(si, 0))) {
                    coop_close<METHOD>(PT_Q, G, K, L, si, PT_ST_ESCAPED);
                    active = false;
                }
            } else if (mode == M_REJECT) {
                L.c2++;
                L.dt = dt * pt_max(PT_Q.fcmn, fpow);
                if (METHOD == PT_METHOD_DOP853) L.rejected = true;
                L.c0++;
                L.dt = pt_min(L.dt, PT_Q.dtm);
            } else if (mode == M_INIT) {
                K(T::F1) = a;
                if (fresh) {
                    L.dt = coop_dti(PT_Q, G, T::IORD, si, a);
                    const double s3 = G.get(si, 3), s4 = G.get(si, 4), s5 = G.get(si, 5);
                    double *row = PT_Q.state + (int64_t)8 * PT_Q.m * L.p;
                    if (G.gl == 6) row[6] = sqrt(s3 * s3 + s4 * s4 + s5 * s5 + 1.0);
                    if (G.gl == 7) row[7] = L.dt;
                }
                next_time(PT_Q, L);
            } else if (mode == M_READY) {
                next_time(PT_Q, L);
            }
            if (active && (mode == M_ACCEPT || mode == M_READY)) EV::coop_begin(PT_Q, G, si, O);
            if constexpr (LEARN) {
                /* as in run_machine: the group's lanes form the features alike,
                 * its first lane is the row of the network's input */
                const bool want = (mode == M_ACCEPT) && active;
                float feat[PT_REC_NFEAT] = { 0, 0, 0, 0, 0, 0, 0, 0, 0 };
                if (want) {
                    double s6[6];
#pragma unroll
                    for (int c = 0; c < 6; ++c) s6[c] = G.get(si, c);
                    int32_t fl_[3], fr_[3];
                    float fx_[3];
                    EV::feature_cell(PT_Q, s6, O, fl_, fr_, fx_);
                    const auto ld_ = EV::feature_loader(PT_Q, fl_, fr_);
                    pt_field_features(PT_Q, ld_, s6, fx_, feat);
                    const float om = PT_Q.qomf * __expf(feat[0] - feat[2]);
                    const float dtf = pt_d2f(dt);
                    feat[5] = __logf(om * dtf + 1e-30f);
                    feat[6] = __logf(pt_d2f(q) + 1e-30f);
                    feat[7] = __logf(dtf);
                    feat[8] = __logf(fminf(pt_face_time(PT_Q, s6, fx_) / dtf, 1.0e6f) + 1e-30f);
                }
                if (__any_sync(0xffffffffu, want)) {
                    const float y = G.get(pt_mlp_warp(pt_mlp_view(blob), feat, want && G.gl == 0), 0);
                    if (want) {
                        const double lo = PT_Q.fcmn * dt;
                        const double hi = (METHOD == PT_METHOD_DOP853 && was_rejected) ? dt : PT_Q.fcmx * dt;
                        const double h = pt_f2d(__expf(y));
                        L.dt = pt_min(pt_max(h, lo), hi);
                        L.dt = pt_min(L.dt, PT_Q.dtm);
                    }
                }
            }
#ifndef PT_EXACT
            /* a handed-over step is capped already */
            if (PT_Q.face && active && !handed_over) L.dt = EV::coop_face_cap(PT_Q, G, si, O, L.dt);
#endif
            if (active) {
                int32_t st = lane_check(PT_Q, L, t_start);
                st = G.get(st, 0);                  /* one clock reading for the group */
                if (st != PT_GO) {
                    coop_close<METHOD>(PT_Q, G, K, L, si, st);
                    active = false;
                } else if (METHOD == PT_METHOD_RK5) {
                    K(0) = PtR(L.dt) * K(T::F1);
                }
            }
            if (!__any_sync(0xffffffffu, active)) {
                if (!__any_sync(0xffffffffu, !drained)) break;
                continue;
            }
        }
        j = (j + 1 < T::SLOTS) ? j + 1 : 0;
    }
}
#undef PT_Q

/* Launch of an eight-lane kernel for n particles at most (n < 0: unknown, fill
 * the GPU).  Runs of under four groups per scheduler take one-warp blocks,
 * which spread over all SMs. */
template <int METHOD, class EV, class KERN, class... Args>
cudaError_t launch_coop(KERN kern, int64_t n, bool learn, cudaStream_t s, Args... args)
{
    const int sms = pt_coop_sms();
    const int block = (n >= 0 && n < 16 * (int64_t)sms) ? 32 : 128;
    const int64_t full = (int64_t)sms * 3;
    int64_t grid = n < 0 ? full : (n * kGroup + block - 1) / block;
    if (block == 128 && grid > full) grid = full;
    kern<<<(int)(grid < 1 ? 1 : grid), block, coop_smem_bytes<METHOD, EV>(block, learn), s>>>(args...);
    return cudaGetLastError();
}

}  // namespace pt_sm

#endif /* PT_COOP_CUH */
