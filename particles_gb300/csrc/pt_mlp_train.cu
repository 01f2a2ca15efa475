/*
 * pt_mlp_train.cu -- training and packing of the learned step-size controller.
 *
 * The MLP 9 -> 64 -> 64 -> 1 (SiLU) is trained on accepted-step records that
 * the classical integrator itself writes (PT_REC_*): inputs are the nine
 * controller features, the target is a standardised log step.  Training runs
 * on the tensor cores (mma.sync, FP16 operands, FP32 accumulation; the
 * kernel below), mean-squared error, and Adam in FP32; the model's FP16
 * tensor-core inference (pt_mlp.cuh) uses the packed blob built by
 * pt_mlp_create.
 *
 * Flat parameter vector (FP32, 4865 values):
 *   W1[9][64] (input-major), b1[64], W2[64][64], b2[64], W3[64], b3.
 */
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <math.h>
#include <stdio.h>
#include <string.h>
#include <vector>

#include "pt_common.cuh"
#include "pt_mlp.cuh"

#define NIN PT_MLP_NIN
#define NH 64
#define OFF_W1 0
#define OFF_B1 (OFF_W1 + NIN * NH)
#define OFF_W2 (OFF_B1 + NH)
#define OFF_B2 (OFF_W2 + NH * NH)
#define OFF_W3 (OFF_B2 + NH)
#define OFF_B3 (OFF_W3 + NH)
#define NPARAM (OFF_B3 + 1)

void pt_set_last_error(const char *msg);

struct pt_mlp {
    unsigned char *blob;   /* device, PT_MLP_BLOB_BYTES */
};

namespace {

__device__ __forceinline__ float sig(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sig(z); }
__device__ __forceinline__ float dsilu(float z) { const float s = sig(z); return s * (1.0f + z * (1.0f - s)); }

#define GRID_LOOP(i, n) for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); \
                             i += (int64_t)gridDim.x * blockDim.x)

/* ---- training on the tensor cores (mma.sync m16n8k16, FP16 operands, FP32
 *      accumulation) --------------------------------------------------------
 *
 * k_train: one kernel per batch of n standardised rows (X n x 9, T n).  A block
 * of eight warps takes 128 rows at a time, 16 per warp:
 *   Z1 = X W1 + b1, H1 = silu(Z1), Z2 = H1 W2 + b2, H2 = silu(Z2),
 *   y = H2 W3 + b3, e = 2 (y - T) (the loss gradient times n), then
 *   dZ2 = e W3^T * silu'(Z2) and dZ1 = (dZ2 W2^T) * silu'(Z1).  A layer's
 *   FP32 accumulators convert in place into the next product's FP16 A
 *   fragments.  X, H1, H2, dZ1, dZ2 and e (FP16) stay in shared memory, from
 *   which the block forms the weight gradients as products over its rows, X^T dZ1
 *   (16 x 64), H1^T dZ2 (64 x 64) and H2^T e (64 x 8, column 0), in accumulators
 *   it keeps over all its rows; the bias gradients are column sums.  At the end
 *   each block adds its part, times 1/n, to the gradient (16-byte atomics).
 * Rows past n have x = 0 and e = 0, so every product they enter is zero.  e is
 * kept unscaled (O(1)) so that its FP16 copies stay normal; the 1/n of the
 * mean enters at the last addition.
 *
 * The bound at the batch sizes of the training (16,384 rows) is latency: one
 * pass of a warp through the three layers and back, so rows are spread 16 to a
 * warp over all SMs and nothing goes through global memory in between.
 *
 * Fragment layouts (PTX ISA, mma.m16n8k16 .f16): g = lane >> 2, q = lane & 3;
 *   A (16x16): a0a1 = A[g][2q..2q+1], a2a3 = A[g+8][2q..], a4a5 = A[g][2q+8..],
 *              a6a7 = A[g+8][2q+8..]
 *   B (16x8):  b0b1 = B[2q..2q+1][g], b2b3 = B[2q+8..2q+9][g]
 *   C (16x8):  c0c1 = C[g][2q..2q+1], c2c3 = C[g+8][2q..2q+1]
 * ldmatrix reads them from row-major tiles (.trans where the tile holds the
 * transposed operand); rows are padded by 16 bytes against bank conflicts.
 */
#define TR_ROWS 128                    /* rows per block and pass */
#define TR_THREADS 256
#define TR_LD 72                       /* halfs per row of a 64-column tile */
#define TR_LDX 24                      /* halfs per row of the 16-column input tile */

__device__ __forceinline__ uint32_t pk_h2(float lo, float hi)
{
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ float2 up_h2(uint32_t v)
{
    return __half22float2(*reinterpret_cast<const __half2 *>(&v));
}

/* 16 x 8 x 16 product with FP32 accumulation (same instruction as the
 * inference's pt_mma16816, kept local to the training kernel). */
__device__ __forceinline__ void mma_acc(float c[4], const uint32_t a[4], uint2 b)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

/* A fragment (16 x 16) of a row-major tile at (r0, c0). */
__device__ __forceinline__ void ld_a(const __half *t, int ld, int r0, int c0, int lane, uint32_t a[4])
{
    const __half *p = t + (r0 + (lane & 15)) * ld + c0 + ((lane >> 4) << 3);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(smem_u32(p)) : "memory");
}

/* A fragment of M^T at (m0, k0): the tile holds M[k][m]. */
__device__ __forceinline__ void ld_at(const __half *t, int ld, int k0, int m0, int lane, uint32_t a[4])
{
    const __half *p = t + (k0 + (lane & 7) + ((lane >> 4) << 3)) * ld + m0 + (((lane >> 3) & 1) << 3);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(smem_u32(p)) : "memory");
}

/* B fragment (16 x 8) at (k0, n0) of a tile N[k][n] ... */
__device__ __forceinline__ uint2 ld_b(const __half *t, int ld, int k0, int n0, int lane)
{
    const __half *p = t + (k0 + (lane & 15)) * ld + n0;
    uint2 b;
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                 : "=r"(b.x), "=r"(b.y) : "r"(smem_u32(p)) : "memory");
    return b;
}

/* ... and of the transposed tile: element (k, n) is N[n][k]. */
__device__ __forceinline__ uint2 ld_bt(const __half *t, int ld, int k0, int n0, int lane)
{
    const __half *p = t + (n0 + (lane & 7)) * ld + k0 + (((lane >> 3) & 1) << 3);
    uint2 b;
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
                 : "=r"(b.x), "=r"(b.y) : "r"(smem_u32(p)) : "memory");
    return b;
}

/* Dynamic shared memory: the FP16 tiles, then the parameters' FP32 rest; the
 * gradient parts take the tiles' place at the end. */
struct TrainSmem {
    __half X[TR_ROWS * TR_LDX], E[TR_ROWS * 8];
    __half H1[TR_ROWS * TR_LD], H2[TR_ROWS * TR_LD], D1[TR_ROWS * TR_LD], D2[TR_ROWS * TR_LD];
    __half W1[16 * TR_LD], W2[NH * TR_LD];
    float b1[NH], b2[NH], w3[NH];
    float bias[2][2 * NH], loss[TR_THREADS / 32], esum[TR_THREADS / 32];
};
static_assert(sizeof(float) * (NPARAM + 3) <= offsetof(TrainSmem, W1), "gradient parts fit the tiles");

__global__ void __launch_bounds__(TR_THREADS, 2) k_train(const float *__restrict__ p,
                                                      const float *__restrict__ X,
                                                      const float *__restrict__ T, int64_t n,
                                                      float inv_n, bool vec, float *__restrict__ grad,
                                                      float *__restrict__ loss)
{
    extern __shared__ __align__(16) unsigned char train_smem[];
    TrainSmem &S = *reinterpret_cast<TrainSmem *>(train_smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    for (int i = tid; i < 16 * NH; i += TR_THREADS)          /* W1, rows 9..15 zero */
        S.W1[(i >> 6) * TR_LD + (i & 63)] = __float2half_rn(i < NIN * NH ? p[OFF_W1 + i] : 0.0f);
    for (int i = tid; i < NH * NH; i += TR_THREADS)
        S.W2[(i >> 6) * TR_LD + (i & 63)] = __float2half_rn(p[OFF_W2 + i]);
    if (tid < NH) {
        S.b1[tid] = p[OFF_B1 + tid];
        S.b2[tid] = p[OFF_B2 + tid];
        S.w3[tid] = p[OFF_W3 + tid];
    }
    for (int i = tid; i < TR_ROWS * TR_LDX; i += TR_THREADS) S.X[i] = __float2half_rn(0.0f);
    for (int i = tid; i < TR_ROWS * 8; i += TR_THREADS) S.E[i] = __float2half_rn(0.0f);
    const float b3 = p[OFF_B3];
    __syncthreads();
    uint2 f3[4];                                             /* W3 (64 x 8, column 0) */
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
        const int k0 = 16 * kt + 2 * q;
        f3[kt] = g == 0 ? make_uint2(pk_h2(S.w3[k0], S.w3[k0 + 1]), pk_h2(S.w3[k0 + 8], S.w3[k0 + 9]))
                        : make_uint2(0u, 0u);
    }
    const int r0 = 16 * warp;                                /* the warp's rows of the tile */
    /* weight gradients: H1^T dZ2, m tile warp / 2, four n tiles; X^T dZ1, n tile
     * warp; H2^T e, m tile warp (warps 0-3); column sums of dZ1 | dZ2 */
    float c2[4][4] = {}, c1[4] = {}, c3[4] = {}, bsum = 0.0f, lsum = 0.0f, esum = 0.0f;
    for (int64_t base = (int64_t)blockIdx.x * TR_ROWS; base < n; base += (int64_t)gridDim.x * TR_ROWS) {
        for (int i = lane; i < 16 * NIN; i += 32) {
            const int64_t at = (base + r0) * NIN + i;
            S.X[(r0 + i / NIN) * TR_LDX + i % NIN] = __float2half_rn(at < n * NIN ? X[at] : 0.0f);
        }
        float tt[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t r = base + r0 + g + 8 * h;
            tt[h] = r < n ? T[r] : 0.0f;
        }
        __syncwarp();
        uint32_t a1[4], a2[4][4], a3[4][4], d1[8][2], d2[8][2];
        ld_a(S.X, TR_LDX, r0, 0, lane, a1);
        /* layer 1: H1 as the next A fragments, silu'(Z1) kept in FP16 */
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int col = 8 * nt + 2 * q;
            float c[4] = { S.b1[col], S.b1[col + 1], S.b1[col], S.b1[col + 1] };
            mma_acc(c, a1, ld_b(S.W1, TR_LD, 0, 8 * nt, lane));
            float h[4], d[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) { h[k] = silu(c[k]); d[k] = dsilu(c[k]); }
            const uint32_t h01 = pk_h2(h[0], h[1]), h23 = pk_h2(h[2], h[3]);
            a2[nt >> 1][(nt & 1) * 2] = h01;
            a2[nt >> 1][(nt & 1) * 2 + 1] = h23;
            d1[nt][0] = pk_h2(d[0], d[1]);
            d1[nt][1] = pk_h2(d[2], d[3]);
            *reinterpret_cast<uint32_t *>(S.H1 + (r0 + g) * TR_LD + col) = h01;
            *reinterpret_cast<uint32_t *>(S.H1 + (r0 + g + 8) * TR_LD + col) = h23;
        }
        /* layer 2: H2 as layer 3's A fragments, silu'(Z2) in FP16 */
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int col = 8 * nt + 2 * q;
            float c[4] = { S.b2[col], S.b2[col + 1], S.b2[col], S.b2[col + 1] };
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) mma_acc(c, a2[kt], ld_b(S.W2, TR_LD, 16 * kt, 8 * nt, lane));
            float h[4], d[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) { h[k] = silu(c[k]); d[k] = dsilu(c[k]); }
            const uint32_t h01 = pk_h2(h[0], h[1]), h23 = pk_h2(h[2], h[3]);
            a3[nt >> 1][(nt & 1) * 2] = h01;
            a3[nt >> 1][(nt & 1) * 2 + 1] = h23;
            d2[nt][0] = pk_h2(d[0], d[1]);
            d2[nt][1] = pk_h2(d[2], d[3]);
            *reinterpret_cast<uint32_t *>(S.H2 + (r0 + g) * TR_LD + col) = h01;
            *reinterpret_cast<uint32_t *>(S.H2 + (r0 + g + 8) * TR_LD + col) = h23;
        }
        /* layer 3: y in column 0 (lanes q == 0: rows g and g + 8) */
        float e[2], c[4] = { b3, 0.0f, b3, 0.0f };
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) mma_acc(c, a3[kt], f3[kt]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float res = (base + r0 + g + 8 * h < n) ? c[2 * h] - tt[h] : 0.0f;
            if (q == 0) lsum += res * res;
            /* e of rows g, g + 8 from the quad's q == 0 lane */
            e[h] = __shfl_sync(0xffffffffu, 2.0f * res, lane & ~3);
            if (q == 0) {
                S.E[(r0 + g + 8 * h) * 8] = __float2half_rn(e[h]);
                esum += e[h];
            }
        }
        /* dZ2 = e W3^T * silu'(Z2), as the A fragments of dZ2 W2^T */
        uint32_t az[4][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int col = 8 * nt + 2 * q;
            const float w0 = S.w3[col], w1 = S.w3[col + 1];
            const float2 dlo = up_h2(d2[nt][0]), dhi = up_h2(d2[nt][1]);
            const uint32_t z01 = pk_h2(e[0] * w0 * dlo.x, e[0] * w1 * dlo.y);
            const uint32_t z23 = pk_h2(e[1] * w0 * dhi.x, e[1] * w1 * dhi.y);
            az[nt >> 1][(nt & 1) * 2] = z01;
            az[nt >> 1][(nt & 1) * 2 + 1] = z23;
            *reinterpret_cast<uint32_t *>(S.D2 + (r0 + g) * TR_LD + col) = z01;
            *reinterpret_cast<uint32_t *>(S.D2 + (r0 + g + 8) * TR_LD + col) = z23;
        }
        /* dZ1 = (dZ2 W2^T) * silu'(Z1) */
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int col = 8 * nt + 2 * q;
            float z[4] = { 0.0f, 0.0f, 0.0f, 0.0f };
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) mma_acc(z, az[kt], ld_bt(S.W2, TR_LD, 16 * kt, 8 * nt, lane));
            const float2 dlo = up_h2(d1[nt][0]), dhi = up_h2(d1[nt][1]);
            *reinterpret_cast<uint32_t *>(S.D1 + (r0 + g) * TR_LD + col) = pk_h2(z[0] * dlo.x, z[1] * dlo.y);
            *reinterpret_cast<uint32_t *>(S.D1 + (r0 + g + 8) * TR_LD + col) = pk_h2(z[2] * dhi.x, z[3] * dhi.y);
        }
        __syncthreads();
        /* the tile's weight gradients */
        const int m0 = 16 * (warp >> 1), n0 = 32 * (warp & 1);
#pragma unroll
        for (int k0 = 0; k0 < TR_ROWS; k0 += 16) {
            uint32_t a[4];
            ld_at(S.H1, TR_LD, k0, m0, lane, a);
#pragma unroll
            for (int t = 0; t < 4; ++t) mma_acc(c2[t], a, ld_b(S.D2, TR_LD, k0, n0 + 8 * t, lane));
            ld_at(S.X, TR_LDX, k0, 0, lane, a);
            mma_acc(c1, a, ld_b(S.D1, TR_LD, k0, 8 * warp, lane));
            if (warp < 4) {
                ld_at(S.H2, TR_LD, k0, 16 * warp, lane, a);
                mma_acc(c3, a, ld_b(S.E, 8, k0, 0, lane));
            }
        }
        {   /* column tid & 127 of dZ1 | dZ2 over the lower or upper rows */
            const __half *d = ((tid & 64) ? S.D2 : S.D1) + (tid >> 7) * (TR_ROWS / 2) * TR_LD + (tid & 63);
#pragma unroll 16
            for (int r = 0; r < TR_ROWS / 2; ++r) bsum += __half2float(d[r * TR_LD]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        esum += __shfl_xor_sync(0xffffffffu, esum, o);
    }
    S.bias[tid >> 7][tid & 127] = bsum;
    if (lane == 0) {
        S.loss[warp] = lsum;
        S.esum[warp] = esum;
    }
    /* the block's gradient part in the parameters' order, over the tiles */
    float *const part = reinterpret_cast<float *>(train_smem);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int m = g + ((k & 2) ? 8 : 0), col = 2 * q + (k & 1);
#pragma unroll
        for (int t = 0; t < 4; ++t)
            part[OFF_W2 + (16 * (warp >> 1) + m) * NH + 32 * (warp & 1) + 8 * t + col] = c2[t][k];
        if (m < NIN) part[OFF_W1 + m * NH + 8 * warp + col] = c1[k];
        if (warp < 4 && col == 0) part[OFF_W3 + 16 * warp + m] = c3[k];
    }
    __syncthreads();
    if (tid < NH) {
        part[OFF_B1 + tid] = S.bias[0][tid] + S.bias[1][tid];
        part[OFF_B2 + tid] = S.bias[0][NH + tid] + S.bias[1][NH + tid];
    }
    if (tid == 0) {
        float es = 0.0f, ls = 0.0f;
        for (int w = 0; w < TR_THREADS / 32; ++w) {
            es += S.esum[w];
            ls += S.loss[w];
        }
        part[OFF_B3] = es;
        atomicAdd(loss, ls * inv_n);
    }
    __syncthreads();
    if (vec) {                                               /* grad on a 16-byte boundary */
        for (int i = tid; i < NPARAM / 4; i += TR_THREADS) {
            const float4 v = reinterpret_cast<const float4 *>(part)[i];
            atomicAdd(reinterpret_cast<float4 *>(grad) + i,
                      make_float4(v.x * inv_n, v.y * inv_n, v.z * inv_n, v.w * inv_n));
        }
        for (int i = NPARAM / 4 * 4 + tid; i < NPARAM; i += TR_THREADS) atomicAdd(grad + i, part[i] * inv_n);
    } else {
        for (int i = tid; i < NPARAM; i += TR_THREADS) atomicAdd(grad + i, part[i] * inv_n);
    }
}

__global__ void k_zero_grad(float *grad, float *loss)
{
    GRID_LOOP(i, NPARAM + 1) *(i < NPARAM ? grad + i : loss) = 0.0f;
}

__global__ void k_adam(float *p, const float *g, float *m, float *v, float lr, float b1, float b2,
                       float eps, float c1, float c2)
{
    GRID_LOOP(e, NPARAM) {
        const float gi = g[e];
        const float mi = b1 * m[e] + (1.0f - b1) * gi;
        const float vi = b2 * v[e] + (1.0f - b2) * gi * gi;
        m[e] = mi;
        v[e] = vi;
        p[e] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

/* The integrator's warp inference on rows of features (tests and tools). */
__global__ void k_infer(const unsigned char *blob, const float *X, int64_t n, float *out)
{
    __shared__ __align__(16) unsigned char sm[PT_MLP_BLOB_BYTES];
    const PtMlpSmem M = pt_mlp_load(blob, sm);
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    for (int64_t w = w0; w * 32 < n; w += warps) {
        const int64_t row = w * 32 + lane;
        float x[NIN];
#pragma unroll
        for (int i = 0; i < NIN; ++i) x[i] = (row < n) ? X[row * NIN + i] : 0.0f;
        const float y = pt_mlp_warp(M, x, row < n);
        if (row < n) out[row] = y;
    }
}

int grid_for(int64_t n)
{
    int64_t g = (n + 255) / 256;
    if (g > 8192) g = 8192;
    return g < 1 ? 1 : (int)g;
}

uint32_t h2bits(float lo, float hi)
{
    const __half a = __float2half_rn(lo), b = __float2half_rn(hi);
    uint16_t ua, ub;
    memcpy(&ua, &a, 2);
    memcpy(&ub, &b, 2);
    return (uint32_t)ua | ((uint32_t)ub << 16);
}

}  // namespace

extern "C" int32_t pt_mlp_nparam(void) { return NPARAM; }

extern "C" int pt_mlp_loss_grad(const float *d_params, const float *d_X, const float *d_T,
                                int64_t n, float *d_grad, float *d_loss, void *stream)
{
    if (!d_params || !d_X || !d_T || !d_grad || !d_loss || n <= 0) {
        pt_set_last_error("pt_mlp_loss_grad: bad argument");
        return PT_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    static std::atomic<uint64_t> configured{ 0 };            /* devices whose attribute is set */
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && !(configured.load(std::memory_order_relaxed) >> (dev & 63) & 1u)) {
        e = cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem));
        if (e == cudaSuccess && dev < 64) configured.fetch_or(1ULL << dev, std::memory_order_relaxed);
    }
    if (e == cudaSuccess) {
        k_zero_grad<<<(NPARAM + 256) / 256, 256, 0, s>>>(d_grad, d_loss);
        /* two blocks fit an SM; blocks beyond that would only add partial gradients */
        const int64_t tiles = (n + TR_ROWS - 1) / TR_ROWS;
        const int blocks = (int)(tiles < 304 ? tiles : 304);
        k_train<<<blocks, TR_THREADS, sizeof(TrainSmem), s>>>(
            d_params, d_X, d_T, n, 1.0f / (float)n, (reinterpret_cast<uintptr_t>(d_grad) & 15u) == 0,
            d_grad, d_loss);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) { pt_set_last_error(cudaGetErrorString(e)); return PT_ERR_CUDA; }
    return PT_OK;
}

extern "C" int pt_mlp_adam(float *d_params, const float *d_grad, float *d_m, float *d_v,
                           int64_t step, float lr, float beta1, float beta2, float eps,
                           void *stream)
{
    if (!d_params || !d_grad || !d_m || !d_v || step < 1) {
        pt_set_last_error("pt_mlp_adam: bad argument");
        return PT_ERR_ARG;
    }
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    k_adam<<<grid_for(NPARAM), 256, 0, (cudaStream_t)stream>>>(d_params, d_grad, d_m, d_v, lr,
                                                                beta1, beta2, eps, c1, c2);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { pt_set_last_error(cudaGetErrorString(e)); return PT_ERR_CUDA; }
    return PT_OK;
}

extern "C" int pt_mlp_create(const float *params, const float norm[2 * PT_MLP_NIN + 2],
                             float safety, pt_mlp **out)
{
    if (!params || !norm || !out || !(safety > 0.0f)) {
        pt_set_last_error("pt_mlp_create: bad argument");
        return PT_ERR_ARG;
    }
    *out = nullptr;
    const float *W1 = params + OFF_W1, *b1 = params + OFF_B1, *W2 = params + OFF_W2;
    const float *b2 = params + OFF_B2, *W3 = params + OFF_W3, b3 = params[OFF_B3];
    const float *mu = norm, *sd = norm + NIN, ymu = norm[2 * NIN], ysd = norm[2 * NIN + 1];
    std::vector<uint32_t> frag(2 * PT_MLP_NFRAG, 0u);
    for (int nt = 0; nt < 8; ++nt)
        for (int lane = 0; lane < 32; ++lane) {
            const int g = lane >> 2, q = lane & 3, nn = 8 * nt + g;
            frag[2 * (PT_MLP_FRAG_W1 + nt * 32 + lane)] =
                h2bits(0.5f * W1[(2 * q) * NH + nn], 0.5f * W1[(2 * q + 1) * NH + nn]);
            /* rows 2q + 8, 2q + 9 of the K = 16 tile: feature 8 (q == 0), else 0 */
            if (q == 0) frag[2 * (PT_MLP_FRAG_W1 + nt * 32 + lane) + 1] =
                h2bits(0.5f * W1[8 * NH + nn], 0.0f);
        }
    for (int kt = 0; kt < 4; ++kt)
        for (int nt = 0; nt < 8; ++nt)
            for (int lane = 0; lane < 32; ++lane) {
                const int g = lane >> 2, q = lane & 3, nn = 8 * nt + g, k0 = 16 * kt + 2 * q;
                const int f = PT_MLP_FRAG_W2 + (kt * 8 + nt) * 32 + lane;
                frag[2 * f] = h2bits(0.5f * W2[k0 * NH + nn], 0.5f * W2[(k0 + 1) * NH + nn]);
                frag[2 * f + 1] = h2bits(0.5f * W2[(k0 + 8) * NH + nn], 0.5f * W2[(k0 + 9) * NH + nn]);
            }
    for (int kt = 0; kt < 4; ++kt)
        for (int lane = 0; lane < 32; ++lane) {
            const int g = lane >> 2, q = lane & 3, k0 = 16 * kt + 2 * q;
            const int f = PT_MLP_FRAG_W3 + kt * 32 + lane;
            if (g == 0) {
                frag[2 * f] = h2bits(W3[k0] * ysd, W3[k0 + 1] * ysd);
                frag[2 * f + 1] = h2bits(W3[k0 + 8] * ysd, W3[k0 + 9] * ysd);
            }
        }
    std::vector<float> tail(PT_MLP_BLOB_FLOATS, 0.0f);
    /* layers 1 and 2 carry a factor 1/2 (exact in FP16/FP32): the inference
     * takes their accumulators as h = z / 2, and silu(z) = h + h tanh(h) */
    for (int j = 0; j < 64; ++j) { tail[j] = 0.5f * b1[j]; tail[64 + j] = 0.5f * b2[j]; }
    tail[128] = b3 * ysd + ymu + logf(safety);
    for (int i = 0; i < NIN; ++i) {
        tail[132 + i] = mu[i];
        tail[132 + PT_MLP_NORM_PAD + i] = (sd[i] > 0.0f) ? 1.0f / sd[i] : 1.0f;
    }
    std::vector<unsigned char> blob(PT_MLP_BLOB_BYTES);
    memcpy(blob.data(), frag.data(), PT_MLP_NFRAG * 8);
    memcpy(blob.data() + PT_MLP_NFRAG * 8, tail.data(), PT_MLP_BLOB_FLOATS * 4);
    pt_mlp *m = new pt_mlp();
    cudaError_t e = cudaMalloc(&m->blob, PT_MLP_BLOB_BYTES);
    if (e == cudaSuccess) e = cudaMemcpy(m->blob, blob.data(), PT_MLP_BLOB_BYTES, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(m->blob);
        delete m;
        pt_set_last_error(cudaGetErrorString(e));
        return PT_ERR_CUDA;
    }
    *out = m;
    return PT_OK;
}

extern "C" int pt_mlp_destroy(pt_mlp *m)
{
    if (!m) return PT_OK;
    cudaFree(m->blob);
    delete m;
    return PT_OK;
}

extern "C" int pt_mlp_infer(const pt_mlp *m, const float *d_X, int64_t n, float *d_out, void *stream)
{
    if (!m || !d_X || !d_out || n < 0) {
        pt_set_last_error("pt_mlp_infer: bad argument");
        return PT_ERR_ARG;
    }
    if (n == 0) return PT_OK;
    int64_t blocks = (n + 127) / 128;
    if (blocks > 4096) blocks = 4096;
    k_infer<<<(int)blocks, 128, 0, (cudaStream_t)stream>>>(m->blob, d_X, n, d_out);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { pt_set_last_error(cudaGetErrorString(e)); return PT_ERR_CUDA; }
    return PT_OK;
}

/* Device blob of a model, for the integrator's launch parameters. */
const unsigned char *pt_mlp_blob(const pt_mlp *m) { return m ? m->blob : nullptr; }
