/*
 * fsph_mlp.cu -- BF16 tensor-core kernels of the warm-start network
 * (inference, training gradients, Adam) and the fsph_mlp_* C ABI.
 *
 * Tensor-core use: mma.sync.m16n8k16 BF16 x BF16 -> FP32.  One warp owns
 * 16 particles (the M dimension); layer outputs stay in registers and the
 * FP32 accumulator fragment of one layer is repacked in place as the BF16
 * A fragment of the next (the m16n8k16 C and A layouts line up tile pairs).
 * Training stages each 64-sample chunk's activations and deltas in shared
 * memory, transposed ([feature][sample]), so that the weight-gradient
 * products (K = samples) are tensor-core MMAs as well; every block writes a
 * partial gradient and a fixed-order reduction sums them (deterministic).
 */
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "../../include/fsph.h"
#include "fsph_kernels.cuh"
#include "fsph_mlp.cuh"

namespace fsph {

static_assert(kBlob == FSPH_MLP_BLOB_SIZE, "blob size in fsph.h");

__device__ __forceinline__ void mma16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

/* two floats -> bf16x2, the first in the low half (the lower column) */
__device__ __forceinline__ unsigned pack2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned *>(&v);
}
__device__ __forceinline__ unsigned ld32(const __nv_bfloat16 *p) { return *reinterpret_cast<const unsigned *>(p); }

/* --------------------------------------------------------------------- */
__global__ void k_mlp_pack(const float *__restrict__ b, MlpDev *__restrict__ d) {
    const __nv_bfloat16 z = __float2bfloat16(0.0f);
    for (int e = threadIdx.x; e < kHid * kS1; e += blockDim.x) {
        int n = e / kS1, k = e % kS1;
        d->w1t[e] = k < kIn ? __float2bfloat16(b[kBW1 + k * kHid + n]) : z;
    }
    for (int e = threadIdx.x; e < kHid * kS2; e += blockDim.x) {
        int n = e / kS2, k = e % kS2;
        d->w2t[e] = k < kHid ? __float2bfloat16(b[kBW2 + k * kHid + n]) : z;
        d->w2[e] = k < kHid ? __float2bfloat16(b[kBW2 + n * kHid + k]) : z;
    }
    for (int e = threadIdx.x; e < 8 * kS2; e += blockDim.x) {
        int n = e / kS2, k = e % kS2;
        d->w3t[e] = (n < kOut && k < kHid) ? __float2bfloat16(b[kBW3 + k * kOut + n]) : z;
    }
    for (int e = threadIdx.x; e < kHid * kS3; e += blockDim.x) {
        int n = e / kS3, k = e % kS3;
        d->w3[e] = k < kOut ? __float2bfloat16(b[kBW3 + n * kOut + k]) : z;
    }
    for (int e = threadIdx.x; e < kHid; e += blockDim.x) {
        d->b1[e] = b[kBB1 + e];
        d->b2[e] = b[kBB2 + e];
    }
    for (int e = threadIdx.x; e < 8; e += blockDim.x) d->b3[e] = e < kOut ? b[kBB3 + e] : 0.0f;
    for (int e = threadIdx.x; e < kIn; e += blockDim.x) {
        d->mu[e] = b[kBMu + e];
        float s = b[kBSig + e];
        d->isig[e] = s > 1e-20f ? 1.0f / s : 0.0f;
    }
    if (threadIdx.x == 0) d->out_scale = b[kBScale];
}

/* 16 bytes a load and, at 128 threads, all of a thread's in flight: word by word
 * the copy was a chain of loads at the head of every launch.  sm is 16-byte
 * aligned; the struct's size, which saved states record, is not a multiple of 16. */
__device__ __forceinline__ void copy_model(MlpDev &sm, const MlpDev *__restrict__ gm) {
    constexpr int kVec = (int)(sizeof(MlpDev) / 16), kWords = (int)(sizeof(MlpDev) / 4);
    const uint4 *src = reinterpret_cast<const uint4 *>(gm);
    uint4 *dst = reinterpret_cast<uint4 *>(&sm);
#pragma unroll 14
    for (int k = threadIdx.x; k < kVec; k += blockDim.x) dst[k] = __ldg(src + k);
    if (4 * kVec + (int)threadIdx.x < kWords)
        reinterpret_cast<unsigned *>(&sm)[4 * kVec + threadIdx.x] =
            reinterpret_cast<const unsigned *>(gm)[4 * kVec + threadIdx.x];
}

/* Forward pass of one warp's 16 rows starting at base.  Leaves the ReLU'd
 * hidden layers (h1, h2) and the output fragment o (rows g / g+8, columns
 * 2c, 2c+1; columns >= 3 are padding).  Rows >= n read zero features. */
struct Fwd {
    float h1[8][4], h2[8][4], o[4];
};

/* The inputs of one thread, rows g and g+8 (past the last row: zero), per
 * 16-column k tile kt: columns 16kt+2c..+1 and 16kt+2c+8..+9. */
template <int KT>
__device__ __forceinline__ void mlp_load(const float *__restrict__ x, int n, int base, int g, int c, float (&v)[KT][8]) {
    const int r0 = base + g, r1 = base + g + 8;
#pragma unroll
    for (int kt = 0; kt < KT; ++kt)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int col = 16 * kt + 2 * c + (q & 1) + 8 * (q >> 1);
            v[kt][q] = r0 < n ? __ldg(x + (size_t)r0 * kIn + col) : 0.0f;
            v[kt][4 + q] = r1 < n ? __ldg(x + (size_t)r1 * kIn + col) : 0.0f;
        }
}
/* ... normalised, as operands */
template <int KT>
__device__ __forceinline__ void mlp_inputs(const MlpDev &sm, const float (&v)[KT][8], int n, int base, int g, int c,
                                           unsigned (&ax)[KT][4]) {
    const int r0 = base + g, r1 = base + g + 8;
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
        float xn[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int col = 16 * kt + 2 * c + (q & 1) + 8 * (q >> 1);
            xn[q] = r0 < n ? (v[kt][q] - sm.mu[col]) * sm.isig[col] : 0.0f;         /* row g   */
            xn[4 + q] = r1 < n ? (v[kt][4 + q] - sm.mu[col]) * sm.isig[col] : 0.0f; /* row g+8 */
        }
        ax[kt][0] = pack2(xn[0], xn[1]);
        ax[kt][1] = pack2(xn[4], xn[5]);
        ax[kt][2] = pack2(xn[2], xn[3]);
        ax[kt][3] = pack2(xn[6], xn[7]);
    }
}

/* KT: the 16-wide input tiles read (inputs past them contribute nothing:
 * a network that gives them no weight runs with KT = 1) */
template <int KT = kIn / 16>
__device__ __forceinline__ void mlp_forward(const MlpDev &sm, const float *__restrict__ x, int n, int base, int g,
                                            int c, Fwd &F) {
    unsigned ax[KT][4];
    {
        float v[KT][8];
        mlp_load<KT>(x, n, base, g, c, v);
        mlp_inputs<KT>(sm, v, n, base, g, c, ax);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float b0v = sm.b1[8 * j + 2 * c], b1v = sm.b1[8 * j + 2 * c + 1];
        F.h1[j][0] = b0v; F.h1[j][1] = b1v; F.h1[j][2] = b0v; F.h1[j][3] = b1v;
#pragma unroll
        for (int kt = 0; kt < KT; ++kt) {
            const __nv_bfloat16 *w = sm.w1t + (8 * j + g) * kS1 + 16 * kt + 2 * c;
            mma16816(F.h1[j], ax[kt], ld32(w), ld32(w + 8));
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) F.h1[j][e] = fmaxf(F.h1[j][e], 0.0f);
    }
    unsigned a[4][4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        a[s][0] = pack2(F.h1[2 * s][0], F.h1[2 * s][1]);
        a[s][1] = pack2(F.h1[2 * s][2], F.h1[2 * s][3]);
        a[s][2] = pack2(F.h1[2 * s + 1][0], F.h1[2 * s + 1][1]);
        a[s][3] = pack2(F.h1[2 * s + 1][2], F.h1[2 * s + 1][3]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float b0v = sm.b2[8 * j + 2 * c], b1v = sm.b2[8 * j + 2 * c + 1];
        F.h2[j][0] = b0v; F.h2[j][1] = b1v; F.h2[j][2] = b0v; F.h2[j][3] = b1v;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const __nv_bfloat16 *w = sm.w2t + (8 * j + g) * kS2 + 16 * s + 2 * c;
            mma16816(F.h2[j], a[s], ld32(w), ld32(w + 8));
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) F.h2[j][e] = fmaxf(F.h2[j][e], 0.0f);
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        a[s][0] = pack2(F.h2[2 * s][0], F.h2[2 * s][1]);
        a[s][1] = pack2(F.h2[2 * s][2], F.h2[2 * s][3]);
        a[s][2] = pack2(F.h2[2 * s + 1][0], F.h2[2 * s + 1][1]);
        a[s][3] = pack2(F.h2[2 * s + 1][2], F.h2[2 * s + 1][3]);
    }
    F.o[0] = sm.b3[2 * c]; F.o[1] = sm.b3[2 * c + 1]; F.o[2] = F.o[0]; F.o[3] = F.o[1];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const __nv_bfloat16 *w = sm.w3t + g * kS2 + 16 * s + 2 * c;
        mma16816(F.o, a[s], ld32(w), ld32(w + 8));
    }
}

/* y = net(x) * out_scale * scale into float4 rows (inference in the step) or
 * plain rows of 3 (y3). */
template <int KT>
__global__ void __launch_bounds__(128) k_mlp_infer(const MlpDev *__restrict__ gm, const float *__restrict__ x, int n,
                                                   float4 *__restrict__ y, float *__restrict__ y3, float scale,
                                                   const unsigned int *__restrict__ valid) {
    __shared__ __align__(16) MlpDev sm;
    copy_model(sm, gm);
    __syncthreads();
    const bool ok = valid == nullptr || *valid != 0u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const float k = sm.out_scale * scale;
    const int ntiles = (n + 15) / 16;
    for (int tile = blockIdx.x * 4 + warp; tile < ntiles; tile += gridDim.x * 4) {
        const int base = tile * 16, r0 = base + g, r1 = base + g + 8;
        if (!ok) {
            if (c == 0 && y) {
                if (r0 < n) y[r0] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r1 < n) y[r1] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            continue;
        }
        Fwd F;
        mlp_forward<KT>(sm, x, n, base, g, c, F);
        const float y2a = __shfl_down_sync(0xffffffffu, F.o[0], 1);
        const float y2b = __shfl_down_sync(0xffffffffu, F.o[2], 1);
        if (c == 0) {
            if (y) {
                if (r0 < n) y[r0] = make_float4(F.o[0] * k, F.o[1] * k, y2a * k, 0.0f);
                if (r1 < n) y[r1] = make_float4(F.o[2] * k, F.o[3] * k, y2b * k, 0.0f);
            } else {
                if (r0 < n) { y3[3 * (size_t)r0] = F.o[0] * k; y3[3 * (size_t)r0 + 1] = F.o[1] * k; y3[3 * (size_t)r0 + 2] = y2a * k; }
                if (r1 < n) { y3[3 * (size_t)r1] = F.o[2] * k; y3[3 * (size_t)r1 + 1] = F.o[3] * k; y3[3 * (size_t)r1 + 2] = y2b * k; }
            }
        }
    }
}

/* --------------------------------------------------------------------- */
/* training                                                              */
/* --------------------------------------------------------------------- */
constexpr int kChunk = 64;            /* samples per block iteration (4 warps x 16) */
constexpr int kSS = kChunk + 8;       /* padded stride of the [feature][sample] staging */
constexpr size_t kGradSmem = sizeof(MlpDev) + (size_t)(kIn + 4 * kHid + 8) * kSS * sizeof(__nv_bfloat16) + 64;

int mlp_grad_blocks(int n) {
    int chunks = (n + kChunk - 1) / kChunk;
    return chunks < 304 ? (chunks > 0 ? chunks : 1) : 304;
}

__device__ __forceinline__ unsigned smem_at(const __nv_bfloat16 *p) { return (unsigned)__cvta_generic_to_shared(p); }
/* four 8 x 8 matrices, lane 8m + r gives row r of matrix m */
__device__ __forceinline__ void load_m4(unsigned (&v)[4], const __nv_bfloat16 *row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(smem_at(row))
                 : "memory");
}
/* two, from the rows of lanes 0-15 */
__device__ __forceinline__ void load_m2(unsigned &v0, unsigned &v1, const __nv_bfloat16 *row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];"
                 : "=r"(v0), "=r"(v1)
                 : "r"(smem_at(row))
                 : "memory");
}
/* the same, to memory and transposed */
__device__ __forceinline__ void store_t4(__nv_bfloat16 *row, const unsigned (&v)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(smem_at(row)),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
                 : "memory");
}
__device__ __forceinline__ void store_t2(__nv_bfloat16 *row, unsigned v0, unsigned v1) {
    asm volatile("stmatrix.sync.aligned.m8n8.x2.trans.shared.b16 [%0], {%1, %2};" ::"r"(smem_at(row)), "r"(v0), "r"(v1)
                 : "memory");
}
/* acc += a (16 x 64) times eight columns whose 64 weights each lie in a row; row:
 * this lane's for k = 0 .. 31 */
__device__ __forceinline__ void mma_row64(float (&acc)[4], const unsigned (&a)[4][4], const __nv_bfloat16 *row) {
#pragma unroll
    for (int s = 0; s < 4; s += 2) {
        unsigned v[4];
        load_m4(v, row + 16 * s);
        mma16816(acc, a[s], v[0], v[1]);
        mma16816(acc, a[s + 1], v[2], v[3]);
    }
}
/* tiles 2s and 2s + 1 as the next product's operand, and the bits of what passes */
__device__ __forceinline__ void relu_pack(float (&h)[2][4], int s, unsigned (&a)[4], unsigned &on) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            h[u][e] = fmaxf(h[u][e], 0.0f);
            if (h[u][e] > 0.0f) on |= 1u << (4 * (2 * s + u) + e);
        }
        a[2 * u] = pack2(h[u][0], h[u][1]);
        a[2 * u + 1] = pack2(h[u][2], h[u][3]);
    }
}
__device__ __forceinline__ void mask_pack(float (&d)[2][4], int s, unsigned on, unsigned (&a)[4]) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int e = 0; e < 4; ++e) d[u][e] = (on >> (4 * (2 * s + u) + e) & 1u) ? d[u][e] : 0.f;
        a[2 * u] = pack2(d[u][0], d[u][1]);
        a[2 * u + 1] = pack2(d[u][2], d[u][3]);
    }
}

/* What bounds it is latency: 8 warps per SM (216 registers, which hold the sums of
 * the weight gradients), each a chain of small products, 15 % of the issue slots
 * used.  So the loads from memory leave early (the model 16 bytes at a time, the
 * next chunk's inputs before this one's weight products, the targets before the
 * layers), and operands move as 8 x 8 matrices.  65,536 rows: 27.6 -> 23.0 us; with
 * three blocks per SM (168 registers, 456 partial gradients to add) the call took
 * 54 us instead of 49. */
__global__ void __launch_bounds__(128, 2) k_mlp_grad(const MlpDev *__restrict__ gm, const float *__restrict__ x,
                                                  const float *__restrict__ t, int n, float *__restrict__ part,
                                                  float *__restrict__ loss_part) {
    extern __shared__ __align__(16) unsigned char dsm[];
    MlpDev &sm = *reinterpret_cast<MlpDev *>(dsm);
    __nv_bfloat16 *sx = reinterpret_cast<__nv_bfloat16 *>(dsm + ((sizeof(MlpDev) + 15) & ~(size_t)15));
    __nv_bfloat16 *sh1 = sx + kIn * kSS;
    __nv_bfloat16 *sh2 = sh1 + kHid * kSS;
    __nv_bfloat16 *sd1 = sh2 + kHid * kSS;
    __nv_bfloat16 *sd2 = sd1 + kHid * kSS;
    __nv_bfloat16 *sdy = sd2 + kHid * kSS;
    __shared__ float s_loss[4];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, c = lane & 3;
    float xv[kIn / 16][8]; /* the next chunk's inputs, on the way during the products of this one */
    mlp_load<kIn / 16>(x, n, (int)blockIdx.x * kChunk + w * 16, g, c, xv);
    copy_model(sm, gm);
    __syncthreads();
    const int row8 = lane & 7, mat = lane >> 3; /* the row of the 8 x 8 matrix that this lane addresses */
    const int st_at = (8 * (mat >> 1) + row8) * kSS + 16 * w + 8 * (mat & 1); /* features down, this warp's samples */
    const int a_at = (8 * (mat & 1) + row8) * kSS + 8 * (mat >> 1); /* a left operand's four matrices */
    const int b_at = (8 * (mat >> 1) + row8) * kSS + 8 * (mat & 1); /* two right operands' */
    const float inv_scale = sm.out_scale != 0.0f ? 1.0f / sm.out_scale : 0.0f;
    const float gscale = 2.0f / (float)n;
    float acc2[8][4], acc3[4], acc1[kIn / 16][2][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc2[j][0] = acc2[j][1] = acc2[j][2] = acc2[j][3] = 0.f;
    acc3[0] = acc3[1] = acc3[2] = acc3[3] = 0.f;
#pragma unroll
    for (int mt = 0; mt < kIn / 16; ++mt)
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) acc1[mt][jj][0] = acc1[mt][jj][1] = acc1[mt][jj][2] = acc1[mt][jj][3] = 0.f;
    /* the bias gradients are sums over the samples of the deltas that the weight
     * products read anyway: products with a matrix of ones (all 16 rows alike),
     * warp w for columns 16w .. 16w + 15 (they had been summed by 64 threads over
     * the 64 staged samples while the other threads waited).  With the reduction
     * below, a gradient over 65,536 rows went from 92 to 44 us, and to 41 with the loads of this kernel moved ahead. */
    float accb1[2][4], accb2[2][4], accb3[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
        accb1[jj][0] = accb1[jj][1] = accb1[jj][2] = accb1[jj][3] = 0.f;
        accb2[jj][0] = accb2[jj][1] = accb2[jj][2] = accb2[jj][3] = 0.f;
    }
    const unsigned one2 = pack2(1.0f, 1.0f);
    const unsigned ones[4] = {one2, one2, one2, one2};
    float loss = 0.f;
    const int nchunks = (n + kChunk - 1) / kChunk;
    for (int ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
        const int base = ch * kChunk + w * 16;
        const int r0 = base + g, r1 = base + g + 8;
        /* forward; x~, h1 and h2 go to the staging transposed as they are made */
        unsigned ax[kIn / 16][4], a[4][4];
        mlp_inputs<kIn / 16>(sm, xv, n, base, g, c, ax);
        /* the targets are needed after three layers */
        const bool in0 = 2 * c < kOut, in1 = 2 * c + 1 < kOut;
        const float t00 = (r0 < n && in0) ? __ldg(t + 3 * (size_t)r0 + 2 * c) * inv_scale : 0.f;
        const float t01 = (r0 < n && in1) ? __ldg(t + 3 * (size_t)r0 + 2 * c + 1) * inv_scale : 0.f;
        const float t10 = (r1 < n && in0) ? __ldg(t + 3 * (size_t)r1 + 2 * c) * inv_scale : 0.f;
        const float t11 = (r1 < n && in1) ? __ldg(t + 3 * (size_t)r1 + 2 * c + 1) * inv_scale : 0.f;
#pragma unroll
        for (int kt = 0; kt < kIn / 16; ++kt) store_t4(sx + 16 * kt * kSS + st_at, ax[kt]);
        unsigned on1 = 0u, on2 = 0u; /* bit 4j + e: element e of tile j is positive */
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            float h[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int j = 2 * s + u;
                const float b0v = sm.b1[8 * j + 2 * c], b1v = sm.b1[8 * j + 2 * c + 1];
                h[u][0] = b0v; h[u][1] = b1v; h[u][2] = b0v; h[u][3] = b1v;
                unsigned wv[4];
                load_m4(wv, sm.w1t + 8 * j * kS1 + row8 * kS1 + 8 * mat);
                mma16816(h[u], ax[0], wv[0], wv[1]);
                mma16816(h[u], ax[1], wv[2], wv[3]);
            }
            relu_pack(h, s, a[s], on1);
            store_t4(sh1 + 16 * s * kSS + st_at, a[s]);
        }
        {
            unsigned a2[4][4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                float h[2][4];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int j = 2 * s + u;
                    const float b0v = sm.b2[8 * j + 2 * c], b1v = sm.b2[8 * j + 2 * c + 1];
                    h[u][0] = b0v; h[u][1] = b1v; h[u][2] = b0v; h[u][3] = b1v;
                    mma_row64(h[u], a, sm.w2t + (8 * j + row8) * kS2 + 8 * mat);
                }
                relu_pack(h, s, a2[s], on2);
                store_t4(sh2 + 16 * s * kSS + st_at, a2[s]);
            }
#pragma unroll
            for (int s = 0; s < 4; ++s)
#pragma unroll
                for (int e = 0; e < 4; ++e) a[s][e] = a2[s][e];
        }
        float o[4] = {sm.b3[2 * c], sm.b3[2 * c + 1], sm.b3[2 * c], sm.b3[2 * c + 1]};
        mma_row64(o, a, sm.w3t + row8 * kS2 + 8 * mat);
        /* dL/dy = 2 (y - t / out_scale) / n for the 3 real outputs of real rows */
        unsigned ady[4] = {0u, 0u, 0u, 0u}; /* padded to K = 16 */
        {
            const float e00 = (r0 < n && in0) ? o[0] - t00 : 0.f;
            const float e01 = (r0 < n && in1) ? o[1] - t01 : 0.f;
            const float e10 = (r1 < n && in0) ? o[2] - t10 : 0.f;
            const float e11 = (r1 < n && in1) ? o[3] - t11 : 0.f;
            loss += e00 * e00 + e01 * e01 + e10 * e10 + e11 * e11;
            ady[0] = pack2(gscale * e00, gscale * e01);
            ady[1] = pack2(gscale * e10, gscale * e11);
            store_t2(sdy + row8 * kSS + w * 16 + 8 * (mat & 1), ady[0], ady[1]);
        }
        /* dH2 = (dY W3^T) * relu'(H2) */
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            unsigned wv[4];
            load_m4(wv, sm.w3 + (16 * s + 8 * (mat >> 1) + row8) * kS3 + 8 * (mat & 1));
            float d[2][4] = {};
            mma16816(d[0], ady, wv[0], wv[1]);
            mma16816(d[1], ady, wv[2], wv[3]);
            mask_pack(d, s, on2, a[s]);
            store_t4(sd2 + 16 * s * kSS + st_at, a[s]);
        }
        /* dH1 = (dH2 W2^T) * relu'(H1) */
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            float d[2][4] = {};
#pragma unroll
            for (int u = 0; u < 2; ++u) mma_row64(d[u], a, sm.w2 + (8 * (2 * s + u) + row8) * kS2 + 8 * mat);
            unsigned v[4];
            mask_pack(d, s, on1, v);
            store_t4(sd1 + 16 * s * kSS + st_at, v);
        }
        mlp_load<kIn / 16>(x, n, (ch + (int)gridDim.x < nchunks ? ch + (int)gridDim.x : ch) * kChunk + w * 16, g, c, xv);
        __syncthreads();
        /* weight gradients of the chunk: K = the 64 samples, 4 k-steps.
         * warp w owns dW2 rows 16w..16w+15, dW3 rows 16w.., dW1 columns 16w.. */
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            unsigned ah[4], bv[4];
            load_m4(ah, sh1 + 16 * w * kSS + a_at + 16 * ks);
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                load_m4(bv, sd2 + 8 * j * kSS + b_at + 16 * ks);
                mma16816(acc2[j], ah, bv[0], bv[1]);
                mma16816(acc2[j + 1], ah, bv[2], bv[3]);
            }
            load_m4(ah, sh2 + 16 * w * kSS + a_at + 16 * ks);
            load_m2(bv[0], bv[1], sdy + row8 * kSS + 8 * (mat & 1) + 16 * ks);
            mma16816(acc3, ah, bv[0], bv[1]);
            mma16816(accb3, ones, bv[0], bv[1]);
            load_m4(bv, sd2 + 16 * w * kSS + b_at + 16 * ks);
            mma16816(accb2[0], ones, bv[0], bv[1]);
            mma16816(accb2[1], ones, bv[2], bv[3]);
            load_m4(bv, sd1 + 16 * w * kSS + b_at + 16 * ks);
            mma16816(accb1[0], ones, bv[0], bv[1]);
            mma16816(accb1[1], ones, bv[2], bv[3]);
#pragma unroll
            for (int mt = 0; mt < kIn / 16; ++mt) {
                load_m4(ah, sx + 16 * mt * kSS + a_at + 16 * ks);
                mma16816(acc1[mt][0], ah, bv[0], bv[1]);
                mma16816(acc1[mt][1], ah, bv[2], bv[3]);
            }
        }
        __syncthreads();
    }
    /* this block's partial gradient, blob layout */
    float *P = part + (size_t)blockIdx.x * kBlob;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int m0 = 16 * w + g, n0 = 8 * j + 2 * c;
        P[kBW2 + m0 * kHid + n0] = acc2[j][0];
        P[kBW2 + m0 * kHid + n0 + 1] = acc2[j][1];
        P[kBW2 + (m0 + 8) * kHid + n0] = acc2[j][2];
        P[kBW2 + (m0 + 8) * kHid + n0 + 1] = acc2[j][3];
    }
    {
        const int m0 = 16 * w + g, n0 = 2 * c;
        if (n0 < kOut) { P[kBW3 + m0 * kOut + n0] = acc3[0]; P[kBW3 + (m0 + 8) * kOut + n0] = acc3[2]; }
        if (n0 + 1 < kOut) { P[kBW3 + m0 * kOut + n0 + 1] = acc3[1]; P[kBW3 + (m0 + 8) * kOut + n0 + 1] = acc3[3]; }
    }
#pragma unroll
    for (int mt = 0; mt < kIn / 16; ++mt)
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
            const int n0 = 8 * (2 * w + jj) + 2 * c, m0 = 16 * mt + g;
            P[kBW1 + m0 * kHid + n0] = acc1[mt][jj][0];
            P[kBW1 + m0 * kHid + n0 + 1] = acc1[mt][jj][1];
            P[kBW1 + (m0 + 8) * kHid + n0] = acc1[mt][jj][2];
            P[kBW1 + (m0 + 8) * kHid + n0 + 1] = acc1[mt][jj][3];
        }
    if (g == 0) {
#pragma unroll
        for (int jj = 0; jj < 2; ++jj)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                P[kBB1 + 8 * (2 * w + jj) + 2 * c + e] = accb1[jj][e];
                P[kBB2 + 8 * (2 * w + jj) + 2 * c + e] = accb2[jj][e];
            }
        if (w == 0)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (2 * c + e < kOut) P[kBB3 + 2 * c + e] = accb3[e];
    }
    if (tid < kBW1) P[tid] = 0.0f;
    if (tid == 0) P[kBScale] = 0.0f;
    loss = warp_sum(loss);
    if (lane == 0) s_loss[w] = loss;
    __syncthreads();
    if (tid == 0) loss_part[blockIdx.x] = s_loss[0] + s_loss[1] + s_loss[2] + s_loss[3];
}

/* Fixed-order sums of the blocks' partials.  A block takes 32 entries, one a
 * lane, and each of its 16 warps every 16th partial (19 independent loads, rows
 * of 128 bytes); the warps' sums are then added in order.  One thread an entry,
 * 304 loads in series on 26 blocks, took 38 us, the loss's 304 by one thread
 * among them.  grad and loss may lie in pinned host memory. */
constexpr int kRedWarps = 16;
__global__ void __launch_bounds__(32 * kRedWarps) k_mlp_reduce(const float *__restrict__ part,
                                                               const float *__restrict__ loss_part, int nblocks, int n,
                                                               float *__restrict__ grad, float *__restrict__ loss) {
    __shared__ float s_sum[kRedWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + lane;
    float sum = 0.f;
    if (e < kBlob) {
#pragma unroll 4
        for (int b = warp; b < nblocks; b += kRedWarps) sum += part[(size_t)b * kBlob + e];
    }
    s_sum[warp][lane] = sum;
    __syncthreads();
    if (warp == 0 && e < kBlob) {
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < kRedWarps; ++k) t += s_sum[k][lane];
        grad[e] = t;
    }
    if (blockIdx.x == gridDim.x - 1 && warp == 1 && loss) {
        double t = 0.0;
        for (int b = lane; b < nblocks; b += 32) t += loss_part[b];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) *loss = (float)(t / (double)(n > 0 ? n : 1));
    }
}

__global__ void k_mlp_adam(float *__restrict__ w, float *__restrict__ m1, float *__restrict__ m2,
                           const float *__restrict__ grad, float lr, float b1, float b2, float eps, float c1,
                           float c2) {
    int e = kTrainFirst + blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= kTrainLast) return;
    float gr = grad[e];
    float a = b1 * m1[e] + (1.0f - b1) * gr;
    float v = b2 * m2[e] + (1.0f - b2) * gr * gr;
    m1[e] = a;
    m2[e] = v;
    w[e] -= lr * (a / c1) / (sqrtf(v / c2) + eps);
}

/* --------------------------------------------------------------------- */
void launch_mlp_pack(const float *blob, MlpDev *dev, cudaStream_t s) { k_mlp_pack<<<1, 256, 0, s>>>(blob, dev); }

static unsigned int infer_blocks(int n) {
    unsigned int tiles = (unsigned int)((n + 15) / 16);
    unsigned int b = (tiles + 3) / 4;
    return b < 1216u ? (b > 0 ? b : 1u) : 1216u;
}

void launch_mlp_infer(const MlpDev *m, const float *x, int n, float4 *y, float scale, const unsigned int *valid,
                      cudaStream_t s, bool local_only) {
    auto k = local_only ? k_mlp_infer<1> : k_mlp_infer<kIn / 16>;
    k<<<infer_blocks(n), 128, 0, s>>>(m, x, n, y, nullptr, scale, valid);
}
void launch_mlp_forward3(const MlpDev *m, const float *x, int n, float *y, cudaStream_t s) {
    k_mlp_infer<kIn / 16><<<infer_blocks(n), 128, 0, s>>>(m, x, n, nullptr, y, 1.0f, nullptr);
}
void launch_mlp_grad(const MlpDev *m, const float *x, const float *t, int n, float *part, float *loss_part,
                     cudaStream_t s) {
    static PerDevice limit;
    raise_shared_limit(limit, (const void *)k_mlp_grad, kGradSmem); /* without it the launch fails */
    k_mlp_grad<<<mlp_grad_blocks(n), 128, kGradSmem, s>>>(m, x, t, n, part, loss_part);
}
void launch_mlp_reduce(const float *part, const float *loss_part, int nblocks, int n, float *grad, float *loss,
                       cudaStream_t s) {
    k_mlp_reduce<<<(kBlob + 31) / 32, 32 * kRedWarps, 0, s>>>(part, loss_part, nblocks, n, grad, loss);
}
void launch_mlp_adam(float *blob, float *m1, float *m2, const float *grad, float lr, float b1, float b2, float eps,
                     int step, cudaStream_t s) {
    float c1 = 1.0f - std::pow(b1, (float)step), c2 = 1.0f - std::pow(b2, (float)step);
    int cnt = kTrainLast - kTrainFirst;
    k_mlp_adam<<<(cnt + 255) / 256, 256, 0, s>>>(blob, m1, m2, grad, lr, b1, b2, eps, c1, c2);
}

}  // namespace fsph

/* ======================================================================== */
/* fsph_mlp C ABI                                                           */
/* ======================================================================== */
using namespace fsph;

struct fsph_mlp {
    MlpDev *dev = nullptr;
    float *blob = nullptr, *m1 = nullptr, *m2 = nullptr, *grad = nullptr;
    float *part = nullptr, *loss_part = nullptr;
    int part_blocks = 0;
    int step = 0;
    float *out = nullptr; /* pinned host memory: a gradient call's results, kBlob entries and the loss */
    unsigned int *tc_err = nullptr; /* set by the tcgen05 forward when a wait ran out */
    cudaStream_t stream = nullptr;
    std::string err;
};

namespace {
int mlp_fail(fsph_mlp *m, cudaError_t e, const char *what) {
    if (m) m->err = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? FSPH_OOM : FSPH_CUDA_ERROR;
}
#define MLP_CUDA(m, call)                                     \
    do {                                                      \
        cudaError_t e_ = (call);                              \
        if (e_ != cudaSuccess) return mlp_fail(m, e_, #call); \
    } while (0)

int ensure_part(fsph_mlp *m, int n) {
    int nb = mlp_grad_blocks(n);
    if (nb <= m->part_blocks) return FSPH_OK;
    cudaFree(m->part);
    cudaFree(m->loss_part);
    m->part = nullptr;
    m->loss_part = nullptr;
    MLP_CUDA(m, cudaMalloc((void **)&m->part, (size_t)nb * kBlob * sizeof(float)));
    MLP_CUDA(m, cudaMalloc((void **)&m->loss_part, (size_t)nb * sizeof(float)));
    m->part_blocks = nb;
    return FSPH_OK;
}
}  // namespace

extern "C" {

int fsph_mlp_create(fsph_mlp **out) {
    if (!out) return FSPH_INVALID_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return FSPH_NO_DEVICE;
    }
    fsph_mlp *m = new (std::nothrow) fsph_mlp();
    if (!m) return FSPH_OOM;
    auto bail = [&](int st) { fsph_mlp_destroy(m); return st; };
    if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) return bail(FSPH_CUDA_ERROR);
    if (cudaMalloc((void **)&m->dev, sizeof(MlpDev)) != cudaSuccess) return bail(FSPH_OOM);
    for (float **p : {&m->blob, &m->m1, &m->m2, &m->grad})
        if (cudaMalloc((void **)p, kBlob * sizeof(float)) != cudaSuccess) return bail(FSPH_OOM);
    if (cudaMalloc((void **)&m->tc_err, sizeof(unsigned int)) != cudaSuccess) return bail(FSPH_OOM);
    if (cudaMallocHost((void **)&m->out, (kBlob + 1) * sizeof(float)) != cudaSuccess) return bail(FSPH_OOM);
    cudaMemsetAsync(m->tc_err, 0, sizeof(unsigned int), m->stream);
    cudaMemsetAsync(m->blob, 0, kBlob * sizeof(float), m->stream);
    cudaMemsetAsync(m->m1, 0, kBlob * sizeof(float), m->stream);
    cudaMemsetAsync(m->m2, 0, kBlob * sizeof(float), m->stream);
    launch_mlp_pack(m->blob, m->dev, m->stream);
    if (cudaStreamSynchronize(m->stream) != cudaSuccess) return bail(FSPH_CUDA_ERROR);
    *out = m;
    return FSPH_OK;
}

int fsph_mlp_destroy(fsph_mlp *m) {
    if (!m) return FSPH_INVALID_ARG;
    if (m->stream) cudaStreamSynchronize(m->stream);
    cudaFree(m->dev);
    cudaFree(m->blob); cudaFree(m->m1); cudaFree(m->m2); cudaFree(m->grad);
    cudaFree(m->part); cudaFree(m->loss_part); cudaFree(m->tc_err);
    if (m->out) cudaFreeHost(m->out);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return FSPH_OK;
}

int fsph_mlp_set_blob(fsph_mlp *m, const float *blob) {
    if (!m || !blob) return FSPH_INVALID_ARG;
    MLP_CUDA(m, cudaMemcpyAsync(m->blob, blob, kBlob * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    MLP_CUDA(m, cudaMemsetAsync(m->m1, 0, kBlob * sizeof(float), m->stream));
    MLP_CUDA(m, cudaMemsetAsync(m->m2, 0, kBlob * sizeof(float), m->stream));
    m->step = 0;
    launch_mlp_pack(m->blob, m->dev, m->stream);
    MLP_CUDA(m, cudaStreamSynchronize(m->stream));
    return FSPH_OK;
}

int fsph_mlp_get_blob(fsph_mlp *m, float *blob) {
    if (!m || !blob) return FSPH_INVALID_ARG;
    MLP_CUDA(m, cudaMemcpyAsync(blob, m->blob, kBlob * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MLP_CUDA(m, cudaStreamSynchronize(m->stream));
    return FSPH_OK;
}

int fsph_mlp_forward(fsph_mlp *m, const float *x, int n, float *y, void *stream) {
    if (!m || n < 0 || (n > 0 && (!x || !y))) return FSPH_INVALID_ARG;
    if (n == 0) return FSPH_OK;
    cudaStream_t s = stream ? (cudaStream_t)stream : m->stream;
    launch_mlp_forward3(m->dev, x, n, y, s);
    MLP_CUDA(m, cudaGetLastError());
    if (!stream) MLP_CUDA(m, cudaStreamSynchronize(s));
    return FSPH_OK;
}

int fsph_mlp_forward_tcgen05(fsph_mlp *m, const float *x, int n, float *y) {
    if (!m || n < 0 || (n > 0 && (!x || !y))) return FSPH_INVALID_ARG;
    if (n == 0) return FSPH_OK;
    cudaStream_t s = m->stream;
    MLP_CUDA(m, cudaMemsetAsync(m->tc_err, 0, sizeof(unsigned int), s));
    launch_mlp_forward3_tc(m->dev, x, n, y, m->tc_err, s);
    MLP_CUDA(m, cudaGetLastError());
    unsigned int e = 0;
    MLP_CUDA(m, cudaMemcpyAsync(&e, m->tc_err, sizeof(e), cudaMemcpyDeviceToHost, s));
    MLP_CUDA(m, cudaStreamSynchronize(s));
    if (e) {
        m->err = "tcgen05 forward: a wait on an MMA ran out";
        return FSPH_TIMEOUT;
    }
    return FSPH_OK;
}

int fsph_mlp_gradient(fsph_mlp *m, const float *x, const float *t, int n, float *grad, float *loss) {
    if (!m || n <= 0 || !x || !t || !grad) return FSPH_INVALID_ARG;
    int st = ensure_part(m, n);
    if (st != FSPH_OK) return st;
    int nb = mlp_grad_blocks(n);
    launch_mlp_grad(m->dev, x, t, n, m->part, m->loss_part, m->stream);
    launch_mlp_reduce(m->part, m->loss_part, nb, n, m->out, m->out + kBlob, m->stream);
    MLP_CUDA(m, cudaGetLastError());
    MLP_CUDA(m, cudaStreamSynchronize(m->stream));
    std::memcpy(grad, m->out, kBlob * sizeof(float));
    if (loss) *loss = m->out[kBlob];
    return FSPH_OK;
}

int fsph_mlp_train(fsph_mlp *m, const float *x, const float *t, int n, int batch, int epochs, float lr,
                   float *loss_per_epoch) {
    if (!m || !x || !t || n <= 0 || batch <= 0 || epochs <= 0 || !(lr > 0.0f)) return FSPH_INVALID_ARG;
    if (batch > n) batch = n;
    int st = ensure_part(m, batch);
    if (st != FSPH_OK) return st;
    const int nbatches = n / batch;
    std::vector<float> losses((size_t)nbatches);
    float *dloss = nullptr;
    MLP_CUDA(m, cudaMalloc((void **)&dloss, (size_t)nbatches * sizeof(float)));
    for (int ep = 0; ep < epochs; ++ep) {
        for (int b = 0; b < nbatches; ++b) {
            const float *xb = x + (size_t)b * batch * kIn;
            const float *tb = t + (size_t)b * batch * 3;
            const int nb = mlp_grad_blocks(batch);
            launch_mlp_grad(m->dev, xb, tb, batch, m->part, m->loss_part, m->stream);
            launch_mlp_reduce(m->part, m->loss_part, nb, batch, m->grad, dloss + b, m->stream);
            m->step += 1;
            launch_mlp_adam(m->blob, m->m1, m->m2, m->grad, lr, 0.9f, 0.999f, 1e-8f, m->step, m->stream);
            launch_mlp_pack(m->blob, m->dev, m->stream);
        }
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(losses.data(), dloss, (size_t)nbatches * sizeof(float), cudaMemcpyDeviceToHost,
                                m->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
        if (e != cudaSuccess) {
            cudaFree(dloss);
            return mlp_fail(m, e, "training epoch");
        }
        if (loss_per_epoch) {
            double s = 0.0;
            for (float l : losses) s += l;
            loss_per_epoch[ep] = (float)(s / (double)(nbatches > 0 ? nbatches : 1));
        }
    }
    cudaFree(dloss);
    return FSPH_OK;
}

const char *fsph_mlp_last_error(const fsph_mlp *m) { return m ? m->err.c_str() : "null network"; }

}  // extern "C"
