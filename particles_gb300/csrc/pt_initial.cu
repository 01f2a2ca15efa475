/*
 * pt_initial.cu -- seeded initial states and their moments on the device.
 *
 * The reference draws positions and momenta with the unseeded random_number
 * (particles.F90:291-296; random.F90:104-179) and prints the mean, standard
 * deviation, skewness and kurtosis of each state component
 * (particles.F90:303-312; random.F90:196-222).  Here every draw is a
 * SplitMix64 output (Steele, Lea & Flood, OOPSLA 2014) of a counter built
 * from (seed, particle index, draw number), the same generator as the host
 * module particles_gb300.initial, so a particle's initial state does not
 * depend on which device, rank or subsample produces it.
 *
 * Compiled with --fmad=false: every product and sum rounds separately in the
 * host generator's order, so positions, mu = 2u - 1 and the fixed-speed
 * momentum are bit-identical to the host; log, exp, sin and cos are CUDA's.
 */
#include <cuda_runtime.h>

#include <atomic>
#include <math.h>
#include <stdint.h>

#include "pt_common.cuh"
#include "pt_internal.h"

using namespace pt_internal;

namespace {

constexpr uint64_t kGolden = 0x9E3779B97F4A7C15ULL;
constexpr uint64_t kM1 = 0xBF58476D1CE4E5B9ULL;
constexpr uint64_t kM2 = 0x94D049BB133111EBULL;
constexpr int kMaxPolarDraws = 32;   /* (1 - pi/4)^32 ~ 2e-22 to run out */

__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t x)
{
    uint64_t z = x + kGolden;
    z = (z ^ (z >> 30)) * kM1;
    z = (z ^ (z >> 27)) * kM2;
    return z ^ (z >> 31);
}

/* The 53 random bits of particle idx, draw `stream`. */
__device__ __forceinline__ uint64_t bits53(uint64_t seed, uint64_t idx, uint64_t stream)
{
    const uint64_t key = splitmix64(seed * 0x100000001B3ULL + stream);
    return splitmix64(idx * kGolden + key) >> 11;
}

/* k 2^-s (k < 2^53: exact) put together from its bits.  The conversion, the
 * scaling and 2 U - 1 as FP64 instructions take slots of the FP64 pipe, which
 * bounds these draws (83 % busy, eight of the eleven of a polar pair); the
 * integer pipes have room.  1,000,003 Maxwellian particles 545 -> 381 us. */
__device__ __forceinline__ uint64_t scaled_bits(uint64_t k, int s)
{
    const int lz = __clzll((long long)k);
    const uint64_t b = (k << (lz - 11)) + ((uint64_t)(1085 - lz - s) << 52);
    return k ? b : 0;
}

/* U in [0, 1) of a draw */
__device__ __forceinline__ double uniform01(uint64_t seed, uint64_t idx, uint64_t stream)
{
    return __longlong_as_double((long long)scaled_bits(bits53(seed, idx, stream), 53));
}

/* 2 U - 1: (k - 2^52) 2^-52, exact */
__device__ __forceinline__ double uniform11(uint64_t seed, uint64_t idx, uint64_t stream)
{
    const int64_t j = (int64_t)bits53(seed, idx, stream) - ((int64_t)1 << 52);
    const uint64_t b = scaled_bits((uint64_t)(j < 0 ? -j : j), 52);
    return __longlong_as_double((long long)(b | ((uint64_t)j & 0x8000000000000000ULL)));
}

struct InitArgs {
    int32_t kind;
    int64_t np, m, index0;
    uint64_t seed;
    double lo[3], hi[3];
    double a, g0, g1;     /* speed, log gamma bounds, or vth */
};

__global__ void k_initial(const InitArgs A, double *__restrict__ state)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < A.np;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t idx = (uint64_t)(A.index0 + i);
        double s[6];
#pragma unroll
        for (int c = 0; c < 3; ++c) s[c] = pt_fadd(pt_fmul(A.hi[c] - A.lo[c], uniform01(A.seed, idx, c)), A.lo[c]);
        if (A.kind == PT_INIT_MAXWELLIAN) {
            /* The draws first, then the transform of the accepted one: a warp
             * leaves the loop after about three draws, and with the logarithm,
             * division and root inside it ran them that often for a few lanes
             * each (1,000,003 particles 1.12 ms). */
            for (int c = 0; c < 3; ++c) {
                double u = 0.0, q = 0.0;
                for (int d = 0; d < kMaxPolarDraws; ++d) {
                    u = uniform11(A.seed, idx, 16 + 64 * c + 2 * d);
                    const double v = uniform11(A.seed, idx, 17 + 64 * c + 2 * d);
                    q = pt_fadd(pt_fmul(u, u), pt_fmul(v, v));
                    /* 0 < q <= 1 on the bits (q >= +0) */
                    const long long b = __double_as_longlong(q);
                    if (b - 1 < 0x3ff0000000000000LL && b > 0) break;
                    q = 0.0;
                }
                s[3 + c] = (__double2hiint(q) != 0) ? u * sqrt(-2.0 * log(q) / q) * A.a : 0.0;
            }
        } else {
            const double mu = uniform11(A.seed, idx, 3);
            const double phi = (2.0 * M_PI) * uniform01(A.seed, idx, 4);
            const double st = sqrt(fmax(0.0, 1.0 - mu * mu));
            double umag;
            if (A.kind == PT_INIT_SPEED) {
                umag = A.a / sqrt(1.0 - A.a * A.a);
            } else {
                const double gam = exp(A.g0 + (A.g1 - A.g0) * uniform01(A.seed, idx, 5));
                umag = sqrt(gam * gam - 1.0);
            }
            double sp, cp;
            sincos(phi, &sp, &cp);
            s[3] = umag * st * cp;
            s[4] = umag * st * sp;
            s[5] = umag * mu;
        }
        double *row = state + (int64_t)8 * A.m * i;
#pragma unroll
        for (int c = 0; c < 6; ++c) row[c] = s[c];
    }
}

/* ---- moments -------------------------------------------------------------- */

constexpr int kMomBlocks = 304, kMomThreads = 256;
/* doubles of one call's scratch: per block two (sum, compensation) pairs, the
 * four moments, the arrival counter */
constexpr int kMomScratch = 4 * kMomBlocks + 4 + 1;

/* Neumaier accumulation of x into (s, c); magnitudes compared on their bits. */
__device__ __forceinline__ void neu_add(double &s, double &c, double x)
{
    const double t = pt_fadd(s, x);
    const bool ge = (__double_as_longlong(s) & 0x7fffffffffffffffLL) >=
                    (__double_as_longlong(x) & 0x7fffffffffffffffLL);
    const double a = ge ? s : x, b = ge ? x : s;
    c = pt_fadd(c, pt_fadd(pt_fsub(a, t), b));
    s = t;
}

/* One pass over the values.  PASS 0: sum of x; 1: of (x - mean)^2; 2: of t^3
 * and t^4 with t = (x - mean) / sd (x - mean where sd is 0).
 *
 * What bounds a pass is the FP64 pipe: 4 operations per Neumaier step, up to
 * 15 per value in pass 2 (the quotient through one reciprocal, pt_qdiv).  Fixed
 * partition: block b sums a contiguous chunk, thread j every blockDim-th
 * element of it, and a block combines its threads in a fixed tree; the block
 * that arrives last combines the blocks in the same way and finishes the
 * moments, so a moment takes one launch and its bits do not depend on the
 * order of arrival. */
template <int PASS>
__global__ void __launch_bounds__(kMomThreads) k_moments(int64_t n, const double *__restrict__ x,
                                                         int64_t stride, double *scratch)
{
    __shared__ double ss[2][kMomThreads], sc[2][kMomThreads];
    __shared__ bool last;
    double *const part = scratch, *const mom = scratch + 4 * kMomBlocks;
    unsigned long long *const arrived = reinterpret_cast<unsigned long long *>(mom + 4);
    constexpr int NS = PASS == 2 ? 2 : 1;
    double s[2] = { 0.0, 0.0 }, c[2] = { 0.0, 0.0 };
    const int tid = threadIdx.x;
    {
        const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
        const int64_t b0 = blockIdx.x * chunk;
        const int64_t b1 = (b0 + chunk < n) ? b0 + chunk : n;
        const double mean = PASS > 0 ? mom[0] : 0.0;
        const double sd = (PASS == 2 && mom[1] != 0.0) ? mom[1] : 1.0, ysd = 1.0 / sd;
#pragma unroll 4
        for (int64_t i = b0 + tid; i < b1; i += kMomThreads) {
            const double v = x[i * stride];
            if (PASS == 0) {
                neu_add(s[0], c[0], v);
            } else {
                double t = pt_fsub(v, mean);
                if (PASS == 1) {
                    neu_add(s[0], c[0], pt_fmul(t, t));
                } else {
                    t = pt_qdiv(t, sd, ysd);
                    const double t2 = pt_fmul(t, t);
                    neu_add(s[0], c[0], pt_fmul(t2, t));
                    neu_add(s[1], c[1], pt_fmul(t2, t2));
                }
            }
        }
    }
    auto tree = [&]() {
#pragma unroll
        for (int k = 0; k < NS; ++k) { ss[k][tid] = s[k]; sc[k][tid] = c[k]; }
        __syncthreads();
        for (int h = kMomThreads / 2; h > 0; h >>= 1) {
            if (tid < h * NS) {
                const int k = NS == 2 ? tid / h : 0, i = NS == 2 ? tid % h : tid;
                double a = ss[k][i], ac = sc[k][i] + sc[k][i + h];
                neu_add(a, ac, ss[k][i + h]);
                ss[k][i] = a;
                sc[k][i] = ac;
            }
            __syncthreads();
        }
    };
    tree();
    if (tid == 0) {
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            part[4 * blockIdx.x + 2 * k] = ss[k][0];
            part[4 * blockIdx.x + 2 * k + 1] = sc[k][0];
        }
        __threadfence();
        last = atomicAdd(arrived, 1ULL) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    /* the last block: thread j takes blocks j, j + 256, then the same tree */
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        s[k] = c[k] = 0.0;
        for (int b = tid; b < (int)gridDim.x; b += kMomThreads) {
            c[k] += __ldcg(part + 4 * b + 2 * k + 1);
            neu_add(s[k], c[k], __ldcg(part + 4 * b + 2 * k));
        }
    }
    __syncthreads();
    tree();
    if (tid == 0) {
        const double m0 = (ss[0][0] + sc[0][0]) / (double)n;
        if (PASS == 2) {
            mom[2] = m0;
            mom[3] = (ss[1][0] + sc[1][0]) / (double)n - 3.0;
        } else {
            mom[PASS] = PASS == 1 ? sqrt(m0) : m0;
        }
        *arrived = 0ULL;
    }
}

/* Scratch of pt_moments calls: the call returns after its stream is done, so
 * a slot serves one call at a time; more calls at once than slots allocate. */
constexpr int kMomSlots = 8;
__device__ double g_mom_scratch[kMomSlots][kMomScratch];
std::atomic<uint32_t> g_mom_taken{ 0 };

int mom_take()
{
    uint32_t t = g_mom_taken.load(std::memory_order_relaxed);
    for (;;) {
        int k = 0;
        while (k < kMomSlots && ((t >> k) & 1u)) ++k;
        if (k == kMomSlots) return -1;
        if (g_mom_taken.compare_exchange_weak(t, t | (1u << k), std::memory_order_acquire)) return k;
    }
}

}  // namespace

extern "C" int pt_initial_state(int32_t kind, int64_t np, int32_t m, uint64_t seed, int64_t index0,
                                const double p[8], double *d_state, void *stream)
{
    if (kind < PT_INIT_SPEED || kind > PT_INIT_MAXWELLIAN)
        return set_err(PT_ERR_ARG, "pt_initial_state: unknown kind%s", "");
    if (np < 0 || m < 1 || index0 < 0 || !p) return set_err(PT_ERR_ARG, "pt_initial_state: bad size or NULL p%s", "");
    if (np == 0) return PT_OK;
    if (!d_state) return set_err(PT_ERR_ARG, "pt_initial_state: NULL state%s", "");
    InitArgs A;
    A.kind = kind;
    A.np = np;
    A.m = m;
    A.index0 = index0;
    A.seed = seed;
    for (int c = 0; c < 3; ++c) {
        A.lo[c] = p[c];
        A.hi[c] = p[3 + c];
        if (!(A.hi[c] >= A.lo[c])) return set_err(PT_ERR_ARG, "pt_initial_state: empty domain%s", "");
    }
    A.a = p[6];
    A.g0 = A.g1 = 0.0;
    if (kind == PT_INIT_SPEED && !(p[6] >= 0.0 && p[6] < 1.0))
        return set_err(PT_ERR_ARG, "pt_initial_state: speed must be in [0, 1)%s", "");
    if (kind == PT_INIT_GAMMA) {
        if (!(p[6] >= 1.0 && p[7] >= p[6])) return set_err(PT_ERR_ARG, "pt_initial_state: need 1 <= gamma lo <= hi%s", "");
        A.g0 = log(p[6]);
        A.g1 = log(p[7]);
    }
    if (kind == PT_INIT_MAXWELLIAN && !(p[6] >= 0.0))
        return set_err(PT_ERR_ARG, "pt_initial_state: vth must be >= 0%s", "");
    int64_t grid = (np + 255) / 256;
    if (grid > 4096) grid = 4096;
    k_initial<<<(int)grid, 256, 0, (cudaStream_t)stream>>>(A, d_state);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_initial_state");
}

extern "C" int pt_moments(int64_t n, const double *d_x, int64_t stride, double out[4], void *stream)
{
    if (n < 1 || !d_x || stride < 1 || !out) return set_err(PT_ERR_ARG, "pt_moments: bad arguments%s", "");
    cudaStream_t s = (cudaStream_t)stream;
    const int slot = mom_take();
    double *buf = nullptr;
    cudaError_t e;
    if (slot >= 0) {
        e = cudaGetSymbolAddress(reinterpret_cast<void **>(&buf), g_mom_scratch);
        buf += (size_t)slot * kMomScratch;
    } else {
        e = cudaMalloc(&buf, kMomScratch * sizeof(double));
    }
    double *mom = buf + 4 * kMomBlocks;
    if (e == cudaSuccess) e = cudaMemsetAsync(mom, 0, 5 * sizeof(double), s);
    if (e == cudaSuccess) {
        const int64_t need = (n + kMomThreads - 1) / kMomThreads;
        const int grid = (int)(need < kMomBlocks ? need : kMomBlocks);
        k_moments<0><<<grid, kMomThreads, 0, s>>>(n, d_x, stride, buf);
        k_moments<1><<<grid, kMomThreads, 0, s>>>(n, d_x, stride, buf);
        k_moments<2><<<grid, kMomThreads, 0, s>>>(n, d_x, stride, buf);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, mom, 4 * sizeof(double), cudaMemcpyDeviceToHost, s);
    const cudaError_t w = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = w;
    if (slot >= 0) g_mom_taken.fetch_and(~(1u << slot), std::memory_order_release);
    else cudaFree(buf);
    return e == cudaSuccess ? PT_OK : cuda_err(e, "pt_moments");
}
