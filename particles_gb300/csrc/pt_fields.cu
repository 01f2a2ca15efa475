/*
 * pt_fields.cu -- field handles of the C ABI: the snapshot converted once on
 * the device into the store of the handle's precision (FP64 node records,
 * compact FP32 bricks, BF16 halo bricks), freed with the handle.  The reference keeps uu, bb
 * in module fields (sources/fields.F90:35, :51-76); the GPU holds this copy.
 */
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <math.h>
#include <stdio.h>
#include <string.h>

#include "pt_internal.h"

using namespace pt_internal;

/* Planar reference layout -> node records { U, B, (J, 0) }. */
__global__ void k_pack_records64(int64_t nn, const double *__restrict__ uu,
                                 const double *__restrict__ bb, const double *__restrict__ jj,
                                 int nc, double *__restrict__ rec)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nn;
         i += (int64_t)gridDim.x * blockDim.x) {
        double v[10];
        for (int c = 0; c < 3; ++c) { v[c] = uu[i + c * nn]; v[3 + c] = bb[i + c * nn]; }
        if (nc == 10) {
            for (int c = 0; c < 3; ++c) v[6 + c] = jj[i + c * nn];
            v[9] = 0.0;
        }
        double2 *o = reinterpret_cast<double2 *>(rec + i * nc);
        for (int c = 0; c < nc / 2; ++c) o[c] = make_double2(v[2 * c], v[2 * c + 1]);
    }
}

/* Planar reference layout -> the FP32 store: 8^3-node bricks without a halo
 * (bricks x-fastest, nodes x-fastest inside a brick; node n of brick b is
 * store node 512 b + n), per node a 32-B record {Ux, Uy, Uz, Bx, By, Bz, 0, 0}
 * or, with J, {Ux, Uy, Uz, Bx, By, Bz, Jx, Jy} and Jz in a second plane.
 * Padding nodes of partial bricks (beyond dm) hold zeros and are never
 * gathered.  One thread per store node. */
__global__ void k_pack_f32(int32_t d0, int32_t d1, int32_t d2, int32_t nbx, int32_t nby,
                           int64_t nrec, const double *__restrict__ uu,
                           const double *__restrict__ bb, const double *__restrict__ jj,
                           float *__restrict__ rec)
{
    const int64_t nn = (int64_t)d0 * d1 * d2;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrec;
         r += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = r >> 9;
        const int t = (int)(r & 511);
        const int bx = (int)(b % nbx), by = (int)((b / nbx) % nby), bz = (int)(b / ((int64_t)nbx * nby));
        const int i = bx * 8 + (t & 7), j = by * 8 + ((t >> 3) & 7), k = bz * 8 + (t >> 6);
        const bool in = i < d0 && j < d1 && k < d2;
        const int64_t g = in ? i + (int64_t)d0 * (j + (int64_t)d1 * k) : 0;
        float v[9];
        for (int c = 0; c < 3; ++c) {
            v[c] = in ? (float)uu[g + c * nn] : 0.f;
            v[3 + c] = in ? (float)bb[g + c * nn] : 0.f;
            v[6 + c] = (in && jj) ? (float)jj[g + c * nn] : 0.f;
        }
        float4 *o = reinterpret_cast<float4 *>(rec + 8 * r);
        o[0] = make_float4(v[0], v[1], v[2], v[3]);
        o[1] = make_float4(v[4], v[5], v[6], v[7]);
        if (jj) rec[8 * nrec + r] = v[8];
    }
}

/* Doubles in the order of their values as unsigned integers (-0 below +0):
 * the high and the low word of the key, and its value again. */
__device__ __forceinline__ uint32_t pt_key_hi(double x)
{
    const int32_t hi = __double2hiint(x);
    return (uint32_t)hi ^ ((uint32_t)(hi >> 31) | 0x80000000u);
}
__device__ __forceinline__ uint32_t pt_key_lo(double x)
{
    return (uint32_t)__double2loint(x) ^ (uint32_t)(__double2hiint(x) >> 31);
}
__device__ __forceinline__ double pt_key_value(uint32_t hi, uint32_t lo)
{
    const uint32_t s = (hi >> 31) ? 0u : 0xffffffffu;      /* negative: all bits inverted */
    return __hiloint2double((int)(hi ^ (s | 0x80000000u)), (int)(lo ^ s));
}

/* The rarely needed FP64 quotient, out of line: inlined, parts of the division
 * run ahead of the test that decides on it. */
__noinline__ __device__ float pt_pack_quotient(double v, float off, float sc)
{
    return (float)((v - (double)off) / (double)sc);
}

/* Planar reference layout -> BF16 8^3 bricks with a one-node halo on the
 * high faces (9^3 records per brick; record (lx, ly, lz) of brick (bx, by,
 * bz) holds node ((8 bx + lx) mod d0, ...)), one block per brick.  Per component the brick's offset is the
 * midpoint and its scale the half-range of the component over the records a
 * stencil can reach (8 b + l <= d on every axis), both rounded to FP32; a
 * record stores q = (v - offset) / scale rounded to BF16 (|q| <= 1).
 *
 * The bound is HBM (with eta J 1.97 GB at 256^3, 0.29 ms); the FP64 pipe, at one
 * instruction per 64 cycles and scheduler, must stay out of the way.  So the
 * extremes are taken on integer keys, the high words first and the low words
 * among the few values that share the extreme high word, and the quotient --
 * FP64 division, rounded to FP32, rounded to BF16 -- is formed in FP32 from
 * v split into two floats, offset and 1/scale: within 7 FP32 ulps of the twice
 * rounded one, so their BF16 roundings agree unless a BF16 midpoint lies
 * within 8 ulps, and then (also where v nearly cancels the offset, or leaves
 * the FP32 normal range, as a zero does) the division decides.  256^3: 0.75 ms
 * (0.45 without J); with FP64 reductions and divisions it was 9.95 (6.91).  With
 * zeros the whole pt_fields_create_device call at 256^3 without J takes 0.62 ms
 * (no component zero; 7.1 with FP64 reductions), 1.27 (Bz = 0; 7.6), 3.4 (U = 0;
 * 8.6), 6.5 (all zero; 10.2). */
template <int NV> struct PackShape {
    /* records per thread, blocks per SM; 1 x 2, 2 x 3, 3 x 3, 4 x 4 measured 944,
     * 748, 764, 868 us with J and 1 x 2, 2 x 3, 3 x 3, 3 x 4, 4 x 4 601, 535,
     * 492, 452, 462 us without (256^3) */
    static constexpr int kRecords = NV == 9 ? 2 : 3, kBlocks = NV == 9 ? 3 : 4;
    static constexpr int kThreads = 768 / kRecords;
};
template <int NV>
__global__ void __launch_bounds__(PackShape<NV>::kThreads, PackShape<NV>::kBlocks) k_pack_bricks16(int32_t d0, int32_t d1, int32_t d2,
                                                          int32_t nbx, int32_t nby,
                                                          const double *__restrict__ uu,
                                                          const double *__restrict__ bb,
                                                          const double *__restrict__ jj,
                                                          uint4 *__restrict__ rec,
                                                          float *__restrict__ bscale)
{
    constexpr int NC16 = (NV == 9) ? 16 : 8, NS = (NV == 9) ? 20 : 12, NR = PackShape<NV>::kRecords;
    constexpr int NT = PackShape<NV>::kThreads, NU = 2 * NV;   /* threads; half components */
    __shared__ uint32_t keys[NV][NR * NT];                  /* high words */
    __shared__ uint32_t umin[NU], umax[NU], lmin[NV], lmax[NV];
    __shared__ float foff[NV], fsc[NV], srs[NV];
    const int64_t b = blockIdx.x;
    const int bx = (int)(b % nbx), by = (int)((b / nbx) % nby), bz = (int)(b / ((int64_t)nbx * nby));
    const int lane = threadIdx.x & 31;
    const int64_t nn = (int64_t)d0 * d1 * d2;
    const double *const src[3] = { uu, bb, jj };
    if (threadIdx.x < NV) {
        lmin[threadIdx.x] = 0xffffffffu;
        lmax[threadIdx.x] = 0u;
    }
    /* Node of record t, or -1 if no stencil reaches it (8 b < d, so within
     * reach a coordinate is the extent itself at most). */
    auto node = [&](int t) -> int64_t {
        const int gi = bx * 8 + t % 9, gj = by * 8 + (t / 9) % 9, gk = bz * 8 + t / 81;
        if (t >= 729 || gi > d0 || gj > d1 || gk > d2) return -1;
        const int i = gi == d0 ? 0 : gi, j = gj == d1 ? 0 : gj, k = gk == d2 ? 0 : gk;
        return i + (int64_t)d0 * (j + (int64_t)d1 * k);
    };
    double v[NR][NV];
    bool reach[NR];
    const int64_t first = node(0);
#pragma unroll
    for (int n = 0; n < NR; ++n) {
        const int t = threadIdx.x + NT * n;
        int64_t g = node(t);
        reach[n] = g >= 0;
        if (!reach[n]) g = first;             /* stands in, so the extremes need no mask */
#pragma unroll
        for (int c = 0; c < NV; ++c) v[n][c] = __ldg(src[c / 3] + g + (c % 3) * nn);
#pragma unroll
        for (int c = 0; c < NV; ++c) keys[c][t] = pt_key_hi(v[n][c]);
    }
    __syncthreads();
    /* a warp per half component: 12 keys per lane, then one warp reduction */
    for (int u = threadIdx.x >> 5; u < NU; u += NT / 32) {
        const uint32_t *k = &keys[u >> 1][(u & 1) * (NR * NT / 2) + lane];
        uint32_t mn = k[0], mx = k[0];
#pragma unroll
        for (int i = 32; i < NR * NT / 2; i += 32) {
            mn = min(mn, k[i]);
            mx = max(mx, k[i]);
        }
        mn = __reduce_min_sync(0xffffffffu, mn);
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) {
            umin[u] = mn;
            umax[u] = mx;
        }
    }
    __syncthreads();
    /* low words among the few values with an extreme high word */
#pragma unroll
    for (int c = 0; c < NV; ++c) {
        const uint32_t mn = min(umin[2 * c], umin[2 * c + 1]), mx = max(umax[2 * c], umax[2 * c + 1]);
#pragma unroll
        for (int n = 0; n < NR; ++n) {
            const uint32_t k = pt_key_hi(v[n][c]);
            if (k == mn) atomicMin(&lmin[c], pt_key_lo(v[n][c]));
            if (k == mx) atomicMax(&lmax[c], pt_key_lo(v[n][c]));
        }
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        const int c = threadIdx.x;
        double mn = pt_key_value(min(umin[2 * c], umin[2 * c + 1]), lmin[c]);
        double mx = pt_key_value(max(umax[2 * c], umax[2 * c + 1]), lmax[c]);
        if (mn != mn || mx != mx) {      /* NaN values do not take part in the extremes */
            mn = INFINITY;
            mx = -INFINITY;
            for (int t = 0; t < 729; ++t) {
                const int64_t g = node(t);
                const double x = g >= 0 ? src[c / 3][g + (c % 3) * nn] : NAN;
                mn = fmin(mn, x);
                mx = fmax(mx, x);
            }
        }
        const float off = (float)(0.5 * (mn + mx));
        float sc = (float)(0.5 * (mx - mn));
        if (!(sc > 0.0f)) sc = 1.0f;
        foff[c] = off;
        fsc[c] = sc;
        /* 0 turns the FP32 quotient off: 1/sc or v - off may leave its normal range */
        srs[c] = (sc > 1.0e-15f && sc < 1.0e15f) ? 1.0f / sc : 0.0f;
        bscale[b * NS + 2 * c] = off;
        bscale[b * NS + 2 * c + 1] = sc;
    } else if (threadIdx.x >= 2 * NV && threadIdx.x < NS) {
        bscale[b * NS + threadIdx.x] = 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NR; ++n) {
        const int t = threadIdx.x + NT * n;
        float x[NC16];
#pragma unroll
        for (int c = 0; c < NC16; ++c) x[c] = 0.0f;
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            /* v = vh + vl: its first 24 significant bits and the next 23 of the
             * rest, as floats (exponents 2^-63 .. 2^127, rebiased by one bit flip) */
            const uint32_t hi = (uint32_t)__double2hiint(v[n][c]), lo = (uint32_t)__double2loint(v[n][c]);
            const uint32_t sg = hi & 0x80000000u;
            const uint32_t f = ((__funnelshift_l(lo, hi, 3) & 0x7fffffffu) ^ 0x40000000u);
            const uint32_t e2 = (f & 0x7f800000u) - (23u << 23);
            const float vl = __uint_as_float(e2 | sg | ((lo >> 6) & 0x7fffffu)) - __uint_as_float(e2 | sg);
            const float vh = __uint_as_float(f | sg);
            const float d = (vh - foff[c]) + vl;
            x[c] = d * srs[c];
            const uint32_t xb = __float_as_uint(x[c]);
            const bool tie = (xb & 0xffffu) - 0x7ff8u <= 16u;
            const bool range = (hi & 0x7fffffffu) - 0x3c000000u < 0x47e00000u - 0x3c000000u;
            if ((tie | !range | (fabsf(d) < 4.8e-7f * fabsf(vh)) | (srs[c] == 0.0f)) && reach[n])
                x[c] = pt_pack_quotient(v[n][c], foff[c], fsc[c]);
            if (!reach[n]) x[c] = 0.0f;
        }
        if (t < 729) {
            uint32_t q[NC16 / 2];
#pragma unroll
            for (int w = 0; w < NC16 / 2; ++w) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(x[2 * w], x[2 * w + 1]);
                q[w] = *reinterpret_cast<const uint32_t *>(&h);
            }
            uint4 *o = rec + (b * 729 + t) * (NC16 / 8);
#pragma unroll
            for (int w = 0; w < NC16 / 8; ++w) o[w] = make_uint4(q[4 * w], q[4 * w + 1], q[4 * w + 2], q[4 * w + 3]);
        }
    }
}

static bool dims_ok(const int32_t dm[3])
{
    if (!dm) return false;
    for (int i = 0; i < 3; ++i)
        if (dm[i] < 1 || dm[i] > (1 << 16)) return false;
    const int64_t n = (int64_t)dm[0] * dm[1] * dm[2];
    return n * 10 < ((int64_t)1 << 40);
}

static int fields_create_impl(const int32_t dm[3], const double *uu, const double *bb,
                              const double *jj, int32_t precision, bool on_device,
                              cudaStream_t stream, pt_fields **out)
{
    if (!out) return set_err(PT_ERR_ARG, "pt_fields_create: out is NULL%s");
    *out = nullptr;
    if (!dims_ok(dm)) return set_err(PT_ERR_ARG, "pt_fields_create: bad dm%s");
    if (!uu || !bb) return set_err(PT_ERR_ARG, "pt_fields_create: uu/bb is NULL%s");
    if (precision != PT_PREC_FP64 && precision != PT_PREC_FP64_FMA && precision != PT_PREC_FP32 &&
        precision != PT_PREC_BF16)
        return set_err(PT_ERR_UNSUPPORTED, "pt_fields_create: precision not built%s");

    int rc = PT_OK;
    const size_t bytes3 = (size_t)dm[0] * dm[1] * dm[2] * 3 * sizeof(double);
    /* Host arrays that the packing kernels can read in place: no copies.  The BF16
     * kernel reads a node up to eight times (1.42 times on average, in runs of 72
     * bytes), which the link does not give back except on small grids.  In place /
     * staged, pageable arrays without J: FP64 64^3 0.25 / 0.40 ms, 100^3 0.44 / 0.62,
     * 256^3 4.4 / 5.5, 400^3 16.2 / 18.9; FP32 0.26 / 0.41, 0.51 / 0.62, 4.6 / 5.3, 16.7
     * / 18.4; BF16 0.34 / 0.41, 0.74 / 0.65, 9.1 / 5.5, 34.4 / 19.4.  Pinned arrays and
     * snapshots with J divide the same way. */
    const bool in_place = precision != PT_PREC_BF16 || (int64_t)dm[0] * dm[1] * dm[2] <= 64 * 64 * 64;
    if (!on_device && in_place)
        on_device = host_direct(uu, bytes3, false) && host_direct(bb, bytes3, false) &&
                    (!jj || host_direct(jj, bytes3, false));
    pt_fields *f = new pt_fields();
    double *d_uu = nullptr, *d_bb = nullptr, *d_jj = nullptr;
    const int64_t nn = (int64_t)dm[0] * dm[1] * dm[2];
    const size_t plane3 = bytes3;
    for (int i = 0; i < 3; ++i) f->dm[i] = dm[i];
    f->precision = precision;
    f->has_j = jj != nullptr;
    f->nc = f->has_j ? 10 : 6;
    f->nc32 = f->has_j ? 16 : 8;
    f->nc16 = f->has_j ? 16 : 8;
    for (int i = 0; i < 3; ++i) f->nb[i] = (dm[i] + 7) / 8;
    f->nodes = nn;
    PT_CU(cudaGetDevice(&f->device));
    PT_CU(cudaMalloc(&f->scratch, 256));
    PT_CU(cudaMemset(f->scratch, 0, 256));
    if (precision == PT_PREC_BF16) {
        const int64_t nbk = (int64_t)f->nb[0] * f->nb[1] * f->nb[2];
        const int ns = f->has_j ? 20 : 12;
        PT_CU(cudaMalloc(&f->rec16, (size_t)nbk * 729 * f->nc16 * 2));
        PT_CU(cudaMalloc(&f->bscale, (size_t)nbk * ns * sizeof(float)));
        f->bytes = nbk * 729 * f->nc16 * 2 + nbk * ns * 4 + 256;
    } else if (precision == PT_PREC_FP32) {
        const int64_t nbk = (int64_t)f->nb[0] * f->nb[1] * f->nb[2];
        const int64_t fl = nbk * 512 * (f->has_j ? 9 : 8);     /* floats of the store */
        PT_CU(cudaMalloc(&f->rec32, (size_t)fl * sizeof(float)));
        f->bytes = fl * (int64_t)sizeof(float) + 256;
    } else {
        PT_CU(cudaMalloc(&f->rec64, (size_t)nn * f->nc * sizeof(double)));
        f->bytes = (int64_t)nn * f->nc * sizeof(double) + 256;
    }
    if (on_device) {
        d_uu = const_cast<double *>(uu);
        d_bb = const_cast<double *>(bb);
        d_jj = const_cast<double *>(jj);
    } else {
        PT_CU(cudaMalloc(&d_uu, plane3));
        PT_CU(cudaMalloc(&d_bb, plane3));
        PT_CU(cudaMemcpyAsync(d_uu, uu, plane3, cudaMemcpyHostToDevice, stream));
        PT_CU(cudaMemcpyAsync(d_bb, bb, plane3, cudaMemcpyHostToDevice, stream));
        if (jj) {
            PT_CU(cudaMalloc(&d_jj, plane3));
            PT_CU(cudaMemcpyAsync(d_jj, jj, plane3, cudaMemcpyHostToDevice, stream));
        }
    }
    {
        int64_t blocks = (nn + 255) / 256;
        if (blocks > 65536) blocks = 65536;
        const int64_t nbk = (int64_t)f->nb[0] * f->nb[1] * f->nb[2];
        if (precision == PT_PREC_BF16 && f->has_j)
            k_pack_bricks16<9><<<(unsigned)nbk, PackShape<9>::kThreads, 0, stream>>>(dm[0], dm[1], dm[2], f->nb[0], f->nb[1],
                                                                  d_uu, d_bb, d_jj, f->rec16, f->bscale);
        else if (precision == PT_PREC_BF16)
            k_pack_bricks16<6><<<(unsigned)nbk, PackShape<6>::kThreads, 0, stream>>>(dm[0], dm[1], dm[2], f->nb[0], f->nb[1],
                                                                  d_uu, d_bb, d_jj, f->rec16, f->bscale);
        else if (precision == PT_PREC_FP32)
            k_pack_f32<<<(int)((nbk * 512 + 255) / 256 < 65536 ? (nbk * 512 + 255) / 256 : 65536), 256, 0,
                         stream>>>(dm[0], dm[1], dm[2], f->nb[0], f->nb[1], nbk * 512, d_uu, d_bb,
                                   d_jj, f->rec32);
        else
            k_pack_records64<<<(int)blocks, 256, 0, stream>>>(nn, d_uu, d_bb, d_jj, f->nc, f->rec64);
        PT_CU(cudaGetLastError());
    }
    PT_CU(cudaStreamSynchronize(stream));
done:
    if (!on_device) {
        cudaFree(d_uu);
        cudaFree(d_bb);
        cudaFree(d_jj);
    }
    if (rc != PT_OK) {
        cudaFree(f->rec64);
        cudaFree(f->rec32);
        cudaFree(f->rec16);
        cudaFree(f->bscale);
        cudaFree(f->scratch);
        delete f;
        return rc;
    }
    *out = f;
    return PT_OK;
}

extern "C" int pt_fields_create(const int32_t dm[3], const double *uu, const double *bb,
                                const double *jj, int32_t precision, pt_fields **out)
{
    return fields_create_impl(dm, uu, bb, jj, precision, false, (cudaStream_t)0, out);
}

extern "C" int pt_fields_create_device(const int32_t dm[3], const double *d_uu,
                                       const double *d_bb, const double *d_jj,
                                       int32_t precision, void *stream, pt_fields **out)
{
    return fields_create_impl(dm, d_uu, d_bb, d_jj, precision, true, (cudaStream_t)stream, out);
}

extern "C" int pt_fields_destroy(pt_fields *f)
{
    if (!f) return PT_OK;
    cudaFree(f->rec64);
    cudaFree(f->rec32);
    cudaFree(f->rec16);
    cudaFree(f->bscale);
    cudaFree(f->scratch);
    cudaFree(f->hand);
    cudaFree(f->ws);
    cudaFree(f->pack);
    cudaFreeHost(f->hst);
    delete f;
    return PT_OK;
}

extern "C" int64_t pt_fields_bytes(const pt_fields *f) { return f ? f->bytes : 0; }

