// rt_mlp.cu -- the MLP radiance cache: encoding, fused forward on the tensor
// cores, backward, Adam.
//
// No counterpart in the reference (its sample has no path tracer to cache).
//
// Network (padded layout, FP32 master parameters and a BF16 copy):
//   layer 0: 96 (81 used) -> 64, ReLU
//   layers 1-4: 64 -> 64, ReLU
//   layer 5: 64 -> 8 (3 used), linear
// Inference (queries): tcgen05 MMAs with TMEM accumulators, see
// k_cache_query_tc.
// Training forward: one warp owns 16 rows of a 128-row tile; each layer is
// m16n8k16 BF16 MMAs with FP32 accumulation; the FP32 accumulator fragment of
// one layer is exactly the A-operand fragment layout of the next (after bias,
// ReLU and BF16 packing), so activations never leave registers between
// layers.  Weights sit in shared memory with padded row strides.
// Backward: the same MMAs propagate delta through W (B fragments of W read
// transposed from its forward layout with ldmatrix.trans); the weight
// gradients delta^T A are MMAs too (both operands loaded transposed with
// ldmatrix.trans), added to global FP32 gradients once per weight and tile;
// Adam updates the FP32 master copy and refreshes the BF16 one.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/rtcore_cache.h"
#include "rt_internal.h"

namespace rtc {
namespace {

constexpr int kLayers = 6;
constexpr int kParams = 23368;  // sum of out*in + out

__host__ __device__ constexpr int in_dim(int l) { return l == 0 ? 96 : 64; }
__host__ __device__ constexpr int out_dim(int l) { return l == 5 ? 8 : 64; }
__host__ __device__ constexpr int w_off(int l) {
    int o = 0;
    for (int k = 0; k < l; ++k) o += out_dim(k) * in_dim(k) + out_dim(k);
    return o;
}
__host__ __device__ constexpr int b_off(int l) { return w_off(l) + out_dim(l) * in_dim(l); }
static_assert(w_off(kLayers) == kParams, "parameter count");

// shared-memory strides (elements): +8 bf16 keeps fragment loads conflict free
__host__ __device__ constexpr int w_stride(int l) { return in_dim(l) + 8; }
constexpr int kBiasFloats = 64 * 5 + 8;
constexpr int kInStride = 104;
constexpr int kActStride = 72;

// State buffer layout (bytes)
struct CacheState {
    float params[kParams];
    float grads[kParams];
    float m[kParams];
    float v[kParams];
    __nv_bfloat16 wbf[kParams];
    uint32_t step;
    float lo[3], hi[3];
    float lr, beta1, beta2, eps;
    float loss;
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&h);
}

__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// c[j] = bias + A (16 x 16*KS) * V^T where V is row-major [8*NT][16*KS] in
// shared memory (stride vs).  bias may be null.
template <int KS, int NT>
__device__ __forceinline__ void warp_dense(const uint32_t (&a)[KS][4], const __nv_bfloat16 *V, int vs,
                                           const float *bias, float (&c)[NT][4], int lane) {
    const int g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        const float b0 = bias ? bias[8 * j + 2 * q] : 0.0f, b1 = bias ? bias[8 * j + 2 * q + 1] : 0.0f;
        c[j][0] = b0; c[j][1] = b1; c[j][2] = b0; c[j][3] = b1;
    }
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const __nv_bfloat16 *row = V + (8 * j + g) * vs + 16 * ks + 2 * q;
            const uint32_t b0 = *reinterpret_cast<const uint32_t *>(row);
            const uint32_t b1 = *reinterpret_cast<const uint32_t *>(row + 8);
            mma_bf16(c[j], a[ks], b0, b1);
        }
    }
}

// ReLU + BF16 pack of an accumulator (16 x 64) into the next layer's A
// fragments.
__device__ __forceinline__ void relu_to_a(const float (&c)[8][4], uint32_t (&a)[4][4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        a[q][0] = pack_bf16(fmaxf(c[2 * q][0], 0.0f), fmaxf(c[2 * q][1], 0.0f));
        a[q][1] = pack_bf16(fmaxf(c[2 * q][2], 0.0f), fmaxf(c[2 * q][3], 0.0f));
        a[q][2] = pack_bf16(fmaxf(c[2 * q + 1][0], 0.0f), fmaxf(c[2 * q + 1][1], 0.0f));
        a[q][3] = pack_bf16(fmaxf(c[2 * q + 1][2], 0.0f), fmaxf(c[2 * q + 1][3], 0.0f));
    }
}

// A fragments of a 16-row slab from a row-major BF16 shared-memory matrix.
template <int KS>
__device__ __forceinline__ void load_a(const __nv_bfloat16 *M, int ms, int r0, int lane, uint32_t (&a)[KS][4]) {
    const int g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
        const __nv_bfloat16 *p0 = M + (r0 + g) * ms + 16 * ks + 2 * q;
        const __nv_bfloat16 *p1 = p0 + 8 * ms;
        a[ks][0] = *reinterpret_cast<const uint32_t *>(p0);
        a[ks][1] = *reinterpret_cast<const uint32_t *>(p1);
        a[ks][2] = *reinterpret_cast<const uint32_t *>(p0 + 8);
        a[ks][3] = *reinterpret_cast<const uint32_t *>(p1 + 8);
    }
}

// Input encoding of one row into 96 BF16 values.
__device__ void encode_row(const rt_cache_input &in, const CacheState *S, __nv_bfloat16 *out) {
    float f[96];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float ext = S->hi[a] - S->lo[a];
        const float pn = ext > 0.0f ? (in.pos[a] - S->lo[a]) / ext : 0.0f;
        // octave k = sin/cos(2^k pi x): one sincospif, then the double-angle
        // recurrence (the error doubles per octave: ~2^11 ulp after 11
        // octaves, far below the BF16 rounding of the features)
        float s, c;
        sincospif(pn, &s, &c);
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            f[24 * a + 2 * k] = s;
            f[24 * a + 2 * k + 1] = c;
            const float s2 = 2.0f * s * c, c2 = (c - s) * (c + s);
            s = s2;
            c = c2;
        }
    }
    for (int a = 0; a < 3; ++a) {
        f[72 + a] = in.dir[a];
        f[75 + a] = in.normal[a];
        f[78 + a] = in.albedo[a];
    }
    for (int k = 81; k < 96; ++k) f[k] = 0.0f;
    for (int k = 0; k < 96; k += 2)
        *reinterpret_cast<uint32_t *>(out + k) = pack_bf16(f[k], f[k + 1]);
}

// ---------------------------------------------------------------------------
// Training: forward + backward over 128-row tiles, gradients into S->grads
// ---------------------------------------------------------------------------
//
// Eight warps, 16 rows each.  Forward as in the inference form, keeping each
// layer's BF16 post-activations.  Backward, layer L = 5 .. 0: the weight and
// bias gradients dW_L = delta_L^T A_{L-1}, db_L = sum delta_L over the tile's
// 128 rows, on the tensor cores (m16n8k16, BF16 operands loaded transposed
// from shared memory with ldmatrix.trans, FP32 accumulation, one atomic add
// per weight and tile), then delta_{L-1} = (delta_L W_L) * relu'(A_{L-1})
// with W_L read transposed by ldmatrix.trans from its forward layout.

constexpr int kTrainRows = 128;
constexpr int kTrainThreads = 256;
__host__ __device__ constexpr int tw_rows(int l) { return l == 5 ? 16 : 64; }  // weight rows kept in shared memory
__host__ __device__ constexpr int tw_off(int l) {
    int o = 0;
    for (int k = 0; k < l; ++k) o += tw_rows(k) * w_stride(k);
    return o;
}
constexpr int kTwElems = tw_off(kLayers);                    // 26240 BF16
constexpr int kDStride = 72;                                 // BF16 delta rows
constexpr size_t kTrainSmem = (size_t)kTwElems * 2 + (size_t)kBiasFloats * 4 + (size_t)kTrainRows * kInStride * 2 +
                              (size_t)5 * kTrainRows * kActStride * 2 + (size_t)kTrainRows * kDStride * 2;
static_assert(kTrainSmem <= 227u * 1024u, "shared memory of the training kernel");

__device__ __forceinline__ void ldsm_x4_t(const void *p, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm_x2_t(const void *p, uint32_t &r0, uint32_t &r1) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                 : "=r"(r0), "=r"(r1)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// Weights (BF16, padded rows; the 8-output layer padded to 16 zero rows) and
// FP32 biases into shared memory, 16 bytes at a time.  Every thread issues
// all of its loads before it stores any (the chunks are independent), so the
// copy costs about one memory round trip instead of one per layer and step:
// 5.5 us of a 16,384-sample batch when each layer's loads waited on the
// previous layer's stores.
constexpr int kTrainWChunks = 64 * 12 + 4 * 64 * 8 + 16 * 8;  // 2,944 sixteen-byte chunks
constexpr int kTrainWPerThread = (kTrainWChunks + kTrainThreads - 1) / kTrainThreads;
__device__ __forceinline__ void train_chunk(int e, int &l, int &o, int &c) {
    if (e < 768) { l = 0; o = e / 12; c = e % 12; }
    else if (e < 2816) { l = 1 + (e - 768) / 512; o = ((e - 768) % 512) / 8; c = (e - 768) % 8; }
    else { l = 5; o = (e - 2816) / 8; c = (e - 2816) % 8; }
}
__device__ void load_weights_train(const CacheState *S, __nv_bfloat16 *sW, float *sB) {
    uint4 r[kTrainWPerThread];
#pragma unroll
    for (int k = 0; k < kTrainWPerThread; ++k) {
        const int e = threadIdx.x + k * kTrainThreads;
        r[k] = make_uint4(0u, 0u, 0u, 0u);
        if (e < kTrainWChunks) {
            int l, o, c;
            train_chunk(e, l, o, c);
            if (o < out_dim(l)) r[k] = reinterpret_cast<const uint4 *>(S->wbf + w_off(l))[o * (in_dim(l) / 8) + c];
        }
    }
    float b[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int e = threadIdx.x + k * kTrainThreads, l = e < 320 ? e / 64 : 5, o = e < 320 ? e % 64 : e - 320;
        b[k] = (e < kBiasFloats && o < out_dim(l)) ? S->params[b_off(l) + o] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < kTrainWPerThread; ++k) {
        const int e = threadIdx.x + k * kTrainThreads;
        if (e >= kTrainWChunks) continue;
        int l, o, c;
        train_chunk(e, l, o, c);
        *reinterpret_cast<uint4 *>(sW + tw_off(l) + o * w_stride(l) + 8 * c) = r[k];
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int e = threadIdx.x + k * kTrainThreads;
        if (e < kBiasFloats) sB[e] = b[k];  // layer l's bias at 64 l, the output layer's at 320
    }
}

// c[j] = A (16 x 16*KS, registers) * W (row-major [16*KS][*], shared memory,
// read transposed): the backward product delta * W over NT n-tiles of 8.
template <int KS, int NT>
__device__ __forceinline__ void warp_dense_wt(const uint32_t (&a)[KS][4], const __nv_bfloat16 *W, int ws,
                                              float (&c)[NT][4], int lane) {
    static_assert(NT % 2 == 0, "n-tiles in pairs");
    const int row = lane & 7, mat = lane >> 3;
#pragma unroll
    for (int j = 0; j < NT; ++j) c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
#pragma unroll
        for (int jp = 0; jp < NT / 2; ++jp) {
            // matrices: (k 0-7, n 0-7), (k 8-15, n 0-7), (k 0-7, n 8-15), (k 8-15, n 8-15)
            const __nv_bfloat16 *p = W + (16 * ks + 8 * (mat & 1) + row) * ws + 16 * jp + 8 * (mat >> 1);
            uint32_t b0, b1, b2, b3;
            ldsm_x4_t(p, b0, b1, b2, b3);
            mma_bf16(c[2 * jp], a[ks], b0, b1);
            mma_bf16(c[2 * jp + 1], a[ks], b2, b3);
        }
    }
}

// dW[o][i] += sum_r delta[r][o] * A[r][i] over the tile's ROWS rows for the
// outputs [o0, o0 + 16) and NT n-tiles of inputs from i0, on the tensor
// cores; rows o >= OUT (padding) are dropped.
template <int IN, int OUT, int NT, int ROWS>
__device__ __forceinline__ void warp_grad_w(const __nv_bfloat16 *sD, const __nv_bfloat16 *sA, int as, int o0, int i0,
                                            float *gW, float *gb, int lane) {
    const int row = lane & 7, mat = lane >> 3, g = lane >> 2, q = lane & 3;
    float c[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.0f;
#pragma unroll 2
    for (int ks = 0; ks < ROWS / 16; ++ks) {
        const int r = 16 * ks;
        // A = delta^T (m = output, k = row): matrices (rows r..r+7 | r+8..r+15) x (o0.. | o0+8..)
        uint32_t a[4];
        ldsm_x4_t(sD + (r + 8 * (mat >> 1) + row) * kDStride + o0 + 8 * (mat & 1), a[0], a[1], a[2], a[3]);
        if constexpr (NT == 1) {
            uint32_t b0, b1;
            ldsm_x2_t(sA + (r + 8 * (mat & 1) + row) * as + i0, b0, b1);
            mma_bf16(c[0], a, b0, b1);
        } else {
#pragma unroll
            for (int jp = 0; jp < NT / 2; ++jp) {
                // B = A (k = row, n = input): matrices (r.., i) (r+8.., i) (r.., i+8) (r+8.., i+8)
                uint32_t b0, b1, b2, b3;
                ldsm_x4_t(sA + (r + 8 * (mat & 1) + row) * as + i0 + 16 * jp + 8 * (mat >> 1), b0, b1, b2, b3);
                mma_bf16(c[2 * jp], a, b0, b1);
                mma_bf16(c[2 * jp + 1], a, b2, b3);
            }
        }
    }
    // input IN is the tile's column of ones: its sums are the bias gradient;
    // columns past it are discarded
#pragma unroll
    // (each lane holds two adjacent inputs of a row: one 8-byte vector add)
    for (int j = 0; j < NT; ++j) {
        const int i = i0 + 8 * j + 2 * q;  // even; IN is even
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int o = o0 + g + 8 * h;
            const float x = c[j][2 * h], y = c[j][2 * h + 1];
            if (o >= OUT || (x == 0.0f && y == 0.0f)) continue;
            if (i < IN)
                asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(gW + o * IN + i), "f"(x), "f"(y) : "memory");
            else if (i == IN && x != 0.0f)
                atomicAdd(gb + o, x);
        }
    }
}

// The weight and bias gradients of layer L, split over the eight warps.  The
// input tiles carry a column of ones right after their last input (column 96
// of the encoded inputs, 64 of the activations, in the row padding), so the
// warps whose input range reaches it take one more n-tile and the MMAs leave
// the bias gradient sum_r delta[r][o] there: no separate row loop (it held two
// warps for ~2 us per layer while the block waited at its barrier).
template <int ROWS>
__device__ __forceinline__ void grads_of_layer(int L, const __nv_bfloat16 *sD, const __nv_bfloat16 *ain, int as,
                                               float *grads, int warp, int lane) {
    if (L == 0) {
        if (warp >> 2)
            warp_grad_w<96, 64, 8, ROWS>(sD, ain, as, 16 * (warp & 3), 48, grads + w_off(0), grads + b_off(0), lane);
        else
            warp_grad_w<96, 64, 6, ROWS>(sD, ain, as, 16 * (warp & 3), 0, grads + w_off(0), grads + b_off(0), lane);
    } else if (L == 5) {
        if (warp == 7)
            warp_grad_w<64, 8, 2, ROWS>(sD, ain, as, 0, 56, grads + w_off(5), grads + b_off(5), lane);
        else
            warp_grad_w<64, 8, 1, ROWS>(sD, ain, as, 0, 8 * warp, grads + w_off(5), grads + b_off(5), lane);
    } else {
        if (warp >> 2)
            warp_grad_w<64, 64, 6, ROWS>(sD, ain, as, 16 * (warp & 3), 32, grads + w_off(L), grads + b_off(L), lane);
        else
            warp_grad_w<64, 64, 4, ROWS>(sD, ain, as, 16 * (warp & 3), 0, grads + w_off(L), grads + b_off(L), lane);
    }
}

// bump_step: this launch is followed by an Adam step (k_cache_adam), whose
// step count it advances first (block 0), so no launch of its own is needed.
__global__ void __launch_bounds__(kTrainThreads, 1) k_cache_fwd_bwd(CacheState *S, const rt_cache_input *in,
                                                                    const float4 *targets, uint32_t n,
                                                                    float inv_count, const uint32_t *n_dev,
                                                                    uint32_t row0, uint32_t bump_step) {
    pdl_wait();
    pdl_launch();
    if (bump_step && blockIdx.x == 0 && threadIdx.x == 0) S->step += 1u;
    if (n_dev) {
        // rows [row0, row0 + n) of a set whose size is produced on the device
        const uint32_t total = *n_dev;
        n = total > row0 ? min(n, total - row0) : 0u;
        if (n == 0) return;
        in += row0;
        targets += row0;
        inv_count = 1.0f / (3.0f * (float)n);
    }
    extern __shared__ __align__(16) uint8_t smem[];
    __nv_bfloat16 *sW = reinterpret_cast<__nv_bfloat16 *>(smem);
    float *sB = reinterpret_cast<float *>(sW + kTwElems);
    __nv_bfloat16 *sIn = reinterpret_cast<__nv_bfloat16 *>(sB + kBiasFloats);
    __nv_bfloat16 *sAct = sIn + kTrainRows * kInStride;
    __nv_bfloat16 *sD = sAct + 5 * kTrainRows * kActStride;
    load_weights_train(S, sW, sB);
    {
        // the ones columns of the bias gradients (row padding, never written otherwise)
        const uint4 ones = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
        for (int e = threadIdx.x; e < 6 * kTrainRows; e += kTrainThreads) {
            const int t = e / kTrainRows, r = e % kTrainRows;
            if (t == 0) *reinterpret_cast<uint4 *>(sIn + r * kInStride + 96) = ones;
            else *reinterpret_cast<uint4 *>(sAct + (t - 1) * kTrainRows * kActStride + r * kActStride + 64) = ones;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int r0 = warp * 16;
    const uint32_t tiles = (n + kTrainRows - 1) / kTrainRows;
    float loss = 0.0f;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        __syncthreads();
        if (threadIdx.x < kTrainRows) {
            const uint32_t row = tile * kTrainRows + threadIdx.x;
            __nv_bfloat16 *dst = sIn + threadIdx.x * kInStride;
            if (row < n) encode_row(in[row], S, dst);
            else
                for (int k = 0; k < 96; k += 2) *reinterpret_cast<uint32_t *>(dst + k) = 0u;
        }
        __syncthreads();
        // ---- forward, keeping post-activations for the backward pass
        uint32_t a0[6][4];
        load_a<6>(sIn, kInStride, r0, lane, a0);
        float c[8][4];
        warp_dense<6, 8>(a0, sW + tw_off(0), w_stride(0), sB, c, lane);
        uint32_t a[4][4];
        relu_to_a(c, a);
#pragma unroll 1
        for (int l = 1; l <= 5; ++l) {
            // store layer l-1 output (the input of layer l) as BF16
            __nv_bfloat16 *act = sAct + (l - 1) * kTrainRows * kActStride;
#pragma unroll
            for (int qq = 0; qq < 4; ++qq) {
                *reinterpret_cast<uint32_t *>(act + (r0 + g) * kActStride + 16 * qq + 2 * q) = a[qq][0];
                *reinterpret_cast<uint32_t *>(act + (r0 + g + 8) * kActStride + 16 * qq + 2 * q) = a[qq][1];
                *reinterpret_cast<uint32_t *>(act + (r0 + g) * kActStride + 16 * qq + 8 + 2 * q) = a[qq][2];
                *reinterpret_cast<uint32_t *>(act + (r0 + g + 8) * kActStride + 16 * qq + 8 + 2 * q) = a[qq][3];
            }
            if (l <= 4) {
                warp_dense<4, 8>(a, sW + tw_off(l), w_stride(l), sB + 64 * l, c, lane);
                relu_to_a(c, a);
            }
        }
        float y[1][4];
        warp_dense<4, 1>(a, sW + tw_off(5), w_stride(5), sB + 320, y, lane);
        // ---- loss gradient at the outputs (cols 0..2 of each row); delta_5
        // as BF16 (cols 0..15, 3..15 zero)
        float dy[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int rr = r0 + g + (e >= 2 ? 8 : 0), col = 2 * q + (e & 1);
            const uint32_t row = tile * kTrainRows + rr;
            dy[e] = 0.0f;
            if (col < 3 && row < n) {
                const float4 tg = targets[row];
                const float yt = col == 0 ? tg.x : (col == 1 ? tg.y : tg.z);
                const float diff = y[0][e] - yt, den = y[0][e] * y[0][e] + 0.01f;
                dy[e] = 2.0f * diff / den * inv_count;
                loss += diff * diff / den;
            }
        }
        uint32_t ad[4][4];
        ad[0][0] = pack_bf16(dy[0], dy[1]);
        ad[0][1] = pack_bf16(dy[2], dy[3]);
        ad[0][2] = 0u;
        ad[0][3] = 0u;
        *reinterpret_cast<uint32_t *>(sD + (r0 + g) * kDStride + 2 * q) = ad[0][0];
        *reinterpret_cast<uint32_t *>(sD + (r0 + g + 8) * kDStride + 2 * q) = ad[0][1];
        *reinterpret_cast<uint32_t *>(sD + (r0 + g) * kDStride + 8 + 2 * q) = 0u;
        *reinterpret_cast<uint32_t *>(sD + (r0 + g + 8) * kDStride + 8 + 2 * q) = 0u;
        // ---- backward, layers 5 .. 0
#pragma unroll 1
        for (int L = 5; L >= 0; --L) {
            __syncthreads();  // delta_L and every activation complete
            const __nv_bfloat16 *ain = L == 0 ? sIn : sAct + (L - 1) * kTrainRows * kActStride;
            const int as = L == 0 ? kInStride : kActStride;
            grads_of_layer<kTrainRows>(L, sD, ain, as, S->grads, warp, lane);
            if (L == 0) break;
            // delta_{L-1} = (delta_L W_L) * relu'(act_{L-1})
            float dc[8][4];
            if (L == 5) {
                uint32_t a1[1][4] = {{ad[0][0], ad[0][1], ad[0][2], ad[0][3]}};
                warp_dense_wt<1, 8>(a1, sW + tw_off(5), w_stride(5), dc, lane);
            } else {
                warp_dense_wt<4, 8>(ad, sW + tw_off(L), w_stride(L), dc, lane);
            }
            const __nv_bfloat16 *act = sAct + (L - 1) * kTrainRows * kActStride;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const __nv_bfloat162 m0 =
                    *reinterpret_cast<const __nv_bfloat162 *>(act + (r0 + g) * kActStride + 8 * j + 2 * q);
                const __nv_bfloat162 m1 =
                    *reinterpret_cast<const __nv_bfloat162 *>(act + (r0 + g + 8) * kActStride + 8 * j + 2 * q);
                if (!(__bfloat162float(m0.x) > 0.0f)) dc[j][0] = 0.0f;
                if (!(__bfloat162float(m0.y) > 0.0f)) dc[j][1] = 0.0f;
                if (!(__bfloat162float(m1.x) > 0.0f)) dc[j][2] = 0.0f;
                if (!(__bfloat162float(m1.y) > 0.0f)) dc[j][3] = 0.0f;
            }
#pragma unroll
            for (int qq = 0; qq < 4; ++qq) {
                ad[qq][0] = pack_bf16(dc[2 * qq][0], dc[2 * qq][1]);
                ad[qq][1] = pack_bf16(dc[2 * qq][2], dc[2 * qq][3]);
                ad[qq][2] = pack_bf16(dc[2 * qq + 1][0], dc[2 * qq + 1][1]);
                ad[qq][3] = pack_bf16(dc[2 * qq + 1][2], dc[2 * qq + 1][3]);
            }
            __syncthreads();  // every warp is done reading delta_L
#pragma unroll
            for (int qq = 0; qq < 4; ++qq) {
                *reinterpret_cast<uint32_t *>(sD + (r0 + g) * kDStride + 16 * qq + 2 * q) = ad[qq][0];
                *reinterpret_cast<uint32_t *>(sD + (r0 + g + 8) * kDStride + 16 * qq + 2 * q) = ad[qq][1];
                *reinterpret_cast<uint32_t *>(sD + (r0 + g) * kDStride + 16 * qq + 8 + 2 * q) = ad[qq][2];
                *reinterpret_cast<uint32_t *>(sD + (r0 + g + 8) * kDStride + 16 * qq + 8 + 2 * q) = ad[qq][3];
            }
        }
    }
    // block loss -> state (mean over samples and channels)
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) atomicAdd(&S->loss, loss * inv_count);
}

// ---------------------------------------------------------------------------
// Small batches: tiles of 32 or 64 rows
// ---------------------------------------------------------------------------
//
// A batch is one chain of layer steps per tile, and a batch of 4,096 rows is 32
// tiles of 128: most SMs idle, and each warp runs 32 MMAs per layer step and as
// many for its weight gradients.  With smaller tiles a layer step is split over
// the eight warps by rows and columns (16 x 16 outputs each with 32 rows, 16 x
// 32 with 64), the activations passing through shared memory, so the chain is
// shorter and more SMs work; the price is a tile's 23,368 gradient reductions,
// which more tiles do more often.  The deltas alternate between two buffers, so
// a backward step has one barrier.  Every output sums in the order of the
// 128-row kernel.
//
// 65,536 samples, us at tiles of 128 / 64 / 32 rows: batches of 1,024 1,208 /
// 952 / 810; 4,096 310 / 245 / 276 (45 of them the reductions); 8,192 161 / 140
// / 154; 16,384 89 / 122 / 145.  (The sums of four blocks added up in a cluster
// first: 1,042 and 280 at 1,024 and 4,096 with 32 rows.)

constexpr size_t small_smem(int rows) {
    return (size_t)kTwElems * 2 + (size_t)kBiasFloats * 4 + (size_t)rows * kInStride * 2 +
           (size_t)5 * rows * kActStride * 2 + (size_t)2 * rows * kDStride * 2;
}
static_assert(small_smem(64) <= 227u * 1024u, "shared memory of the small-batch kernel");

// encode_row's features of a tile's rows, four or eight lanes per row: lanes 0-2
// an axis each, lane 3 the rest.
template <int ROWS>
__device__ __forceinline__ void encode_small(const rt_cache_input *in, uint32_t row0, uint32_t n, const CacheState *S,
                                             __nv_bfloat16 *sIn) {
    constexpr uint32_t kLanes = kTrainThreads / ROWS;
    const uint32_t r = threadIdx.x / kLanes, part = threadIdx.x % kLanes, row = row0 + r;
    if (part > 3u) return;
    uint32_t *dst = reinterpret_cast<uint32_t *>(sIn + r * kInStride + 24u * part);
    if (row >= n) {
#pragma unroll
        for (int k = 0; k < 12; ++k) dst[k] = 0u;
        return;
    }
    if (part < 3u) {
        const float lo = S->lo[part], ext = S->hi[part] - lo;
        const float pn = ext > 0.0f ? (in[row].pos[part] - lo) / ext : 0.0f;
        float s, c;
        sincospif(pn, &s, &c);
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            dst[k] = pack_bf16(s, c);
            const float s2 = 2.0f * s * c, c2 = (c - s) * (c + s);
            s = s2;
            c = c2;
        }
    } else {
        const rt_cache_input x = in[row];
        dst[0] = pack_bf16(x.dir[0], x.dir[1]);
        dst[1] = pack_bf16(x.dir[2], x.normal[0]);
        dst[2] = pack_bf16(x.normal[1], x.normal[2]);
        dst[3] = pack_bf16(x.albedo[0], x.albedo[1]);
        dst[4] = pack_bf16(x.albedo[2], 0.0f);
#pragma unroll
        for (int k = 5; k < 12; ++k) dst[k] = 0u;
    }
}

// after_adam: the launch before is this training call's own Adam step, so the
// inputs were there before it and are encoded while it still runs.
template <int ROWS>
__global__ void __launch_bounds__(kTrainThreads, 1) k_cache_fwd_bwd_small(CacheState *S, const rt_cache_input *in,
                                                                          const float4 *targets, uint32_t n,
                                                                          float inv_count, const uint32_t *n_dev,
                                                                          uint32_t row0, uint32_t bump_step,
                                                                          uint32_t after_adam) {
    constexpr int kSmallSlabs = ROWS / 16;  // 16-row slabs; also a warp's 8-column tiles
    constexpr int kSmallNt = kSmallSlabs;
    extern __shared__ __align__(16) uint8_t smem[];
    __nv_bfloat16 *sW = reinterpret_cast<__nv_bfloat16 *>(smem);
    float *sB = reinterpret_cast<float *>(sW + kTwElems);
    __nv_bfloat16 *sIn = reinterpret_cast<__nv_bfloat16 *>(sB + kBiasFloats);
    __nv_bfloat16 *sAct = sIn + ROWS * kInStride;
    __nv_bfloat16 *sDelta = sAct + 5 * ROWS * kActStride;
    {
        // the ones columns of the bias gradients (row padding, never written otherwise)
        const uint4 ones = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
        for (int e = threadIdx.x; e < 6 * ROWS; e += kTrainThreads) {
            const int t = e / ROWS, r = e % ROWS;
            if (t == 0) *reinterpret_cast<uint4 *>(sIn + r * kInStride + 96) = ones;
            else *reinterpret_cast<uint4 *>(sAct + (t - 1) * ROWS * kActStride + r * kActStride + 64) = ones;
        }
    }
    if (!after_adam) pdl_wait();
    if (n_dev) {
        // rows [row0, row0 + n) of a set whose size is produced on the device
        const uint32_t total = *n_dev;
        n = total > row0 ? min(n, total - row0) : 0u;
        in += row0;
        targets += row0;
        inv_count = 1.0f / (3.0f * (float)n);
    }
    const uint32_t tiles = (n + ROWS - 1) / ROWS;
    if (blockIdx.x < tiles) encode_small<ROWS>(in, blockIdx.x * ROWS, n, S, sIn);
    if (after_adam) pdl_wait();
    pdl_launch();
    if (bump_step && blockIdx.x == 0 && threadIdx.x == 0) S->step += 1u;
    if (blockIdx.x >= tiles) return;
    load_weights_train(S, sW, sB);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int r0 = 16 * (warp % kSmallSlabs), col0 = 8 * kSmallNt * (warp / kSmallSlabs);  // this warp's rows and columns
    float loss = 0.0f;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        if (tile != blockIdx.x) {
            __syncthreads();
            encode_small<ROWS>(in, tile * ROWS, n, S, sIn);
        }
        __syncthreads();
        // ---- forward, keeping post-activations for the backward pass
        auto store2 = [&](__nv_bfloat16 *m, int stride, const float (&c)[kSmallNt][4], bool relu) {
#pragma unroll
            for (int j = 0; j < kSmallNt; ++j) {
                const float x0 = relu ? fmaxf(c[j][0], 0.0f) : c[j][0], x1 = relu ? fmaxf(c[j][1], 0.0f) : c[j][1];
                const float x2 = relu ? fmaxf(c[j][2], 0.0f) : c[j][2], x3 = relu ? fmaxf(c[j][3], 0.0f) : c[j][3];
                *reinterpret_cast<uint32_t *>(m + (r0 + g) * stride + col0 + 8 * j + 2 * q) = pack_bf16(x0, x1);
                *reinterpret_cast<uint32_t *>(m + (r0 + g + 8) * stride + col0 + 8 * j + 2 * q) = pack_bf16(x2, x3);
            }
        };
        {
            uint32_t a0[6][4];
            load_a<6>(sIn, kInStride, r0, lane, a0);
            float c[kSmallNt][4];
            warp_dense<6, kSmallNt>(a0, sW + tw_off(0) + col0 * w_stride(0), w_stride(0), sB + col0, c, lane);
            store2(sAct, kActStride, c, true);
        }
#pragma unroll 1
        for (int l = 1; l <= 4; ++l) {
            __syncthreads();
            uint32_t a[4][4];
            load_a<4>(sAct + (l - 1) * ROWS * kActStride, kActStride, r0, lane, a);
            float c[kSmallNt][4];
            warp_dense<4, kSmallNt>(a, sW + tw_off(l) + col0 * w_stride(l), w_stride(l), sB + 64 * l + col0, c, lane);
            store2(sAct + l * ROWS * kActStride, kActStride, c, true);
        }
        __syncthreads();
        if (warp < kSmallSlabs) {
            uint32_t a[4][4];
            load_a<4>(sAct + 4 * ROWS * kActStride, kActStride, r0, lane, a);
            float y[1][4];
            warp_dense<4, 1>(a, sW + tw_off(5), w_stride(5), sB + 320, y, lane);
            // ---- loss gradient at the outputs (cols 0..2 of each row);
            // delta_5 as BF16 (cols 0..15, 3..15 zero)
            float dy[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int rr = r0 + g + (e >= 2 ? 8 : 0), col = 2 * q + (e & 1);
                const uint32_t row = tile * ROWS + rr;
                dy[e] = 0.0f;
                if (col < 3 && row < n) {
                    const float4 tg = targets[row];
                    const float yt = col == 0 ? tg.x : (col == 1 ? tg.y : tg.z);
                    const float diff = y[0][e] - yt, den = y[0][e] * y[0][e] + 0.01f;
                    dy[e] = 2.0f * diff / den * inv_count;
                    loss += diff * diff / den;
                }
            }
            *reinterpret_cast<uint32_t *>(sDelta + (r0 + g) * kDStride + 2 * q) = pack_bf16(dy[0], dy[1]);
            *reinterpret_cast<uint32_t *>(sDelta + (r0 + g + 8) * kDStride + 2 * q) = pack_bf16(dy[2], dy[3]);
            *reinterpret_cast<uint32_t *>(sDelta + (r0 + g) * kDStride + 8 + 2 * q) = 0u;
            *reinterpret_cast<uint32_t *>(sDelta + (r0 + g + 8) * kDStride + 8 + 2 * q) = 0u;
        }
        // ---- backward, layers 5 .. 0
#pragma unroll 1
        for (int L = 5; L >= 0; --L) {
            __syncthreads();  // delta_L complete; the other buffer is free
            const __nv_bfloat16 *dcur = sDelta + ((L + 1) & 1) * ROWS * kDStride;
            __nv_bfloat16 *dnext = sDelta + (L & 1) * ROWS * kDStride;
            const __nv_bfloat16 *ain = L == 0 ? sIn : sAct + (L - 1) * ROWS * kActStride;
            const int as = L == 0 ? kInStride : kActStride;
            if (L > 0) {
                // delta_{L-1} = (delta_L W_L) * relu'(act_{L-1}), first: the next step waits for it
                float dc[kSmallNt][4];
                if (L == 5) {
                    uint32_t a1[1][4];
                    load_a<1>(dcur, kDStride, r0, lane, a1);
                    warp_dense_wt<1, kSmallNt>(a1, sW + tw_off(5) + col0, w_stride(5), dc, lane);
                } else {
                    uint32_t ad[4][4];
                    load_a<4>(dcur, kDStride, r0, lane, ad);
                    warp_dense_wt<4, kSmallNt>(ad, sW + tw_off(L) + col0, w_stride(L), dc, lane);
                }
#pragma unroll
                for (int j = 0; j < kSmallNt; ++j) {
                    const __nv_bfloat162 m0 =
                        *reinterpret_cast<const __nv_bfloat162 *>(ain + (r0 + g) * kActStride + col0 + 8 * j + 2 * q);
                    const __nv_bfloat162 m1 = *reinterpret_cast<const __nv_bfloat162 *>(
                        ain + (r0 + g + 8) * kActStride + col0 + 8 * j + 2 * q);
                    if (!(__bfloat162float(m0.x) > 0.0f)) dc[j][0] = 0.0f;
                    if (!(__bfloat162float(m0.y) > 0.0f)) dc[j][1] = 0.0f;
                    if (!(__bfloat162float(m1.x) > 0.0f)) dc[j][2] = 0.0f;
                    if (!(__bfloat162float(m1.y) > 0.0f)) dc[j][3] = 0.0f;
                }
                store2(dnext, kDStride, dc, false);
            }
            grads_of_layer<ROWS>(L, dcur, ain, as, S->grads, warp, lane);
        }
    }
    // block loss -> state (mean over samples and channels)
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0 && warp < kSmallSlabs) atomicAdd(&S->loss, loss * inv_count);
}

// ---------------------------------------------------------------------------
// Inference on the 5th-generation tensor cores (tcgen05 + TMEM)
// ---------------------------------------------------------------------------
//
// One CTA per SM with five independent groups of 4 warps = 128 threads, one
// query row per thread, 128-row tiles; the groups share one copy of the weights
// in shared memory, and the tensor core works on one group's layer while the
// others encode or run their epilogues.
//
// Weights and encoded inputs live in shared memory in the canonical K-major
// layout without swizzle: 8-row x 16-byte core matrices; element (r, k) of a
// tile with K columns sits at (r/8)*16K + (k/8)*128 + (r%8)*16 + (k%8)*2 bytes,
// so one MMA step of K = 16 is described by LBO = 128 (next core matrix along
// K) and SBO = 16K (next 8-row group).  A group's thread 0 issues
// tcgen05.mma.kind::f16 with M = 128, N = 64 (N = 16 for the output layer),
// K = 16 per instruction, BF16 x BF16 -> FP32 accumulators in TMEM (row r =
// TMEM lane r), and commits to the group's mbarrier, on which the group waits.
//
// A layer starts with one MMA that sets the accumulators to the bias: a tile of
// ones times the bias split in three BF16 parts, whose sum is the FP32 bias
// exactly (a tiny one scaled up against a column of 2^-64), so the layer's MMAs
// add onto the bias.  The epilogue of every thread
// reads its row's 64 accumulators with tcgen05.ld (each warp its own 32-lane
// quarter), applies ReLU and packs BF16 in one cvt.rn.relu.bf16x2.f32 per pair,
// and writes the row back to TMEM as the next layer's A operand (two BF16 per
// 32-bit column): the activations never pass through shared memory.  Every
// mbarrier wait is bounded: on expiry the kernel records RT_ERR_TIMEOUT, waits
// once more (bounded) for its MMAs, frees its TMEM and returns.
//
// 2,073,600 queries: 141 us, tensor pipe busy 62 % of the cycles at 36 % of its
// rate (an MMA of N = 64 fills about half of it), the rest the encoding and the
// epilogues.  248 us with four groups, the
// biases stored to TMEM for every row and layer and the activations written to
// shared memory in the MMA's layout.

constexpr int kTcRows = 128;
constexpr int kTcGroups = 5;                      // independent 128-row tile groups per CTA
constexpr int kTcThreads = 128 * kTcGroups;
constexpr uint32_t kTcTmemCols = 512;             // a power of two; 96 per group are used
constexpr uint32_t kTcGroupCols = 96;             // 64 accumulators, 32 columns of BF16 pairs
constexpr uint32_t kTcACol = 64;
// tile byte sizes / offsets
__host__ __device__ constexpr uint32_t tc_tile_bytes(int rows, int k) { return (uint32_t)(rows / 8) * 16u * k; }
__host__ __device__ constexpr uint32_t tc_w_off(int l) {
    uint32_t o = 0;
    for (int i = 0; i < l; ++i) o += tc_tile_bytes(i == 5 ? 16 : 64, in_dim(i));
    return o;
}
constexpr uint32_t kTcWBytes = tc_w_off(6);                        // 47104: all weights, shared by the groups
constexpr uint32_t kTcBias = kTcWBytes;                            // per layer, the bias as a K = 16 operand
__host__ __device__ constexpr uint32_t tc_bias_off(int l) { return kTcBias + (uint32_t)l * tc_tile_bytes(64, 16); }
constexpr uint32_t kTcOnes = tc_bias_off(5) + tc_tile_bytes(16, 16);  // 128 x 16 ones
constexpr uint32_t kTcBar = kTcOnes + tc_tile_bytes(kTcRows, 16);  // one mbarrier per group + the TMEM address
constexpr uint32_t kTcGroupBase = (kTcBar + 8u * kTcGroups + 8u + 127u) & ~127u;
constexpr uint32_t kTcGroupBytes = tc_tile_bytes(kTcRows, 96);     // per group: the K = 96 input tile
constexpr uint32_t kTcSmem = kTcGroupBase + kTcGroups * kTcGroupBytes;
static_assert(kTcSmem <= 227u * 1024u, "shared memory of the inference kernel");
static_assert(kTcSmem < (1u << 18), "descriptor addresses do not wrap");
static_assert(kTcGroups * kTcGroupCols <= kTcTmemCols, "TMEM of the inference kernel");
constexpr int kTcSpinLimit = 1 << 20;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint32_t tc_off(int r, int k, int kdim) {
    return (uint32_t)(r >> 3) * 16u * (uint32_t)kdim + (uint32_t)(k >> 3) * 128u + (uint32_t)(r & 7) * 16u +
           (uint32_t)(k & 7) * 2u;
}
// Shared-memory matrix descriptor: start >> 4, LBO >> 4, SBO >> 4,
// descriptor version 1 (bits 46-47), no swizzle (bits 61-63 = 0).
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3fffu) | ((uint64_t)((lbo >> 4) & 0x3fffu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3fffu) << 32) | (1ull << 46);
}
// Instruction descriptor of kind::f16: FP32 accumulate (bits 4-5 = 1), BF16
// A and B (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bits 17-22,
// M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t tc_idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    for (int it = 0; it < kTcSpinLimit; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// A from TMEM (two BF16 per column), B from shared memory.
__device__ __forceinline__ void tc_mma_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(db), "r"(idesc));
}
// 32 consecutive columns of this thread's TMEM lane
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tc_ld4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}
// Waits for the thread's TMEM loads; the registers pass through, so that no use
// of them moves above the wait.
__device__ __forceinline__ void tc_wait_ld(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}
__device__ __forceinline__ void tc_wait_ld(uint32_t (&r)[4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]) : : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// max(lo, 0) and max(hi, 0) rounded to BF16 and packed (lo in the low half):
// one cvt.rn.relu.bf16x2.f32
__device__ __forceinline__ uint32_t relu_pack_bf16(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void group_sync(int group) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(kTcRows) : "memory");
}

// Two-wide FP32 arithmetic (each half rounded as the scalar instruction).
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    uint64_t x, y, d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
    return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    uint64_t x, y, d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
    return r;
}

// encode_row's 96 features of one row into the K = 96 input tile: the same
// operations, axes 0 and 1 two at a time, each eight features stored as they
// are ready.
__device__ __forceinline__ void encode_to_tile(const rt_cache_input &in, const float (&lo)[3], const float (&ext)[3],
                                               uint8_t *tile, int r) {
    float s[3], c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float pn = ext[a] > 0.0f ? (in.pos[a] - lo[a]) / ext[a] : 0.0f;
        sincospif(pn, &s[a], &c[a]);
    }
    auto put = [&](int kc, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
        *reinterpret_cast<uint4 *>(tile + tc_off(r, 8 * kc, 96)) = make_uint4(x, y, z, w);
    };
    {
        float2 sv = make_float2(s[0], s[1]), cv = make_float2(c[0], c[1]);
#pragma unroll
        for (int kc = 0; kc < 3; ++kc) {
            uint32_t p0[4], p1[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                p0[k] = pack_bf16(sv.x, cv.x);
                p1[k] = pack_bf16(sv.y, cv.y);
                const float2 s2 = mul2(mul2(make_float2(2.0f, 2.0f), sv), cv);
                const float2 c2 = mul2(add2(cv, make_float2(-sv.x, -sv.y)), add2(cv, sv));
                sv = s2;
                cv = c2;
            }
            put(kc, p0[0], p0[1], p0[2], p0[3]);
            put(3 + kc, p1[0], p1[1], p1[2], p1[3]);
        }
    }
    float s1 = s[2], c1 = c[2];
#pragma unroll
    for (int kc = 0; kc < 3; ++kc) {
        uint32_t p[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            p[k] = pack_bf16(s1, c1);
            const float s2 = 2.0f * s1 * c1, c2 = (c1 - s1) * (c1 + s1);
            s1 = s2;
            c1 = c2;
        }
        put(6 + kc, p[0], p[1], p[2], p[3]);
    }
    put(9, pack_bf16(in.dir[0], in.dir[1]), pack_bf16(in.dir[2], in.normal[0]), pack_bf16(in.normal[1], in.normal[2]),
        pack_bf16(in.albedo[0], in.albedo[1]));
    put(10, pack_bf16(in.albedo[2], 0.0f), 0u, 0u, 0u);
    put(11, 0u, 0u, 0u, 0u);
}

__global__ void __launch_bounds__(kTcThreads, 1) k_cache_query_tc(const CacheState *S, const rt_cache_input *in,
                                                                  float4 *out, uint32_t n, const uint32_t *n_dev,
                                                                  uint32_t *err) {
    if (n_dev) n = min(n, *n_dev);
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t *sW = smem;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kTcBar);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + kTcBar + 8u * kTcGroups);
    // per group: set by a thread whose barrier wait ran out, before the
    // group's barrier, read by all the group's threads after it (so the whole
    // group leaves its loop together)
    __shared__ int s_gfail[kTcGroups];
    const int tid = threadIdx.x, warp = tid >> 5;
    const int group = tid / kTcRows, gtid = tid % kTcRows;
    uint8_t *tile_a = smem + kTcGroupBase + (uint32_t)group * kTcGroupBytes;

    // ---- weights (canonical K-major, eight inputs of an output per 16-byte
    // chunk), the split biases and the ones, once
    constexpr int kChunks = 64 * 12 + 4 * 64 * 8 + 16 * 8;
    for (int e = tid; e < kChunks; e += kTcThreads) {
        int l, o, c;
        train_chunk(e, l, o, c);
        uint4 w = make_uint4(0u, 0u, 0u, 0u);
        if (o < out_dim(l)) w = __ldg(reinterpret_cast<const uint4 *>(S->wbf + w_off(l)) + o * (in_dim(l) / 8) + c);
        *reinterpret_cast<uint4 *>(sW + tc_w_off(l) + tc_off(o, 8 * c, in_dim(l))) = w;
    }
    for (int e = tid; e < 336; e += kTcThreads) {
        const int l = e < 320 ? e / 64 : 5, o = e < 320 ? e % 64 : e - 320;
        const float b = o < out_dim(l) ? S->params[b_off(l) + o] : 0.0f;
        // hi + mid + lo == b: 8 significant bits each of its 24 (rounded to zero
        // where hi would round to infinity); of an infinity or NaN hi alone.  A
        // small bias goes in times 2^64, against the 2^-64 in columns 3-5 of the
        // ones: its lower parts would be below BF16's range.
        const bool finite = fabsf(b) < kInf, small = fabsf(b) < 0x1p-60f;
        const float v = small ? b * 0x1p64f : b;
        float hi = __bfloat162float(__float2bfloat16(v));
        const bool high = finite && !(fabsf(hi) < kInf);
        if (high) hi = __bfloat162float(__float2bfloat16_rz(v));
        const float r1 = finite ? v - hi : 0.0f;
        const float mid = __bfloat162float(high ? __float2bfloat16_rz(r1) : __float2bfloat16(r1)), r2 = r1 - mid;
        uint8_t *dst = smem + tc_bias_off(l) + tc_off(o, 0, 16);
        *reinterpret_cast<uint4 *>(dst) = small ? make_uint4(0u, pack_bf16(0.0f, hi), pack_bf16(mid, r2), 0u)
                                                : make_uint4(pack_bf16(hi, mid), pack_bf16(r2, 0.0f), 0u, 0u);
        *reinterpret_cast<uint4 *>(dst + 128) = make_uint4(0u, 0u, 0u, 0u);
    }
    for (int e = tid; e < kTcRows * 2; e += kTcThreads) {
        constexpr uint32_t one = 0x3f80u, tiny = 0x1f80u;  // 1 and 2^-64; 8 rows' first eight columns, then the others
        const bool first = ((e >> 3) & 1) == 0;
        *reinterpret_cast<uint4 *>(smem + kTcOnes + 16 * e) =
            first ? make_uint4(one | one << 16, one | tiny << 16, tiny | tiny << 16, 0u) : make_uint4(0u, 0u, 0u, 0u);
    }
    if (tid < kTcGroups) s_gfail[tid] = 0;
    if (tid == 0) {
        for (int g = 0; g < kTcGroups; ++g)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bars + g)) : "memory");
        // make the initialised barriers visible to the tensor core's arrivals
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTcTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // this group's accumulator columns; warp w of the group reads TMEM lanes
    // [32 (w % 4), 32 (w % 4) + 32)
    const uint32_t tmem = *tmem_slot + kTcGroupCols * (uint32_t)group;
    const uint32_t bar_a = smem_u32(bars + group);
    const uint32_t w_base = smem_u32(sW);
    // operand descriptors (the address field counts 16 bytes; a step of K = 16
    // is 256): ones, biases, input tile, weights of layer 0 and from layer 1 on
    const uint64_t d_ones = tc_desc(w_base + kTcOnes, 128u, 256u), d_bias = tc_desc(w_base + kTcBias, 128u, 256u);
    const uint64_t d_in = tc_desc(smem_u32(tile_a), 128u, 16u * 96u), d_w0 = tc_desc(w_base, 128u, 16u * 96u);
    const uint64_t d_w1 = tc_desc(w_base + tc_w_off(1), 128u, 16u * 64u);
    uint32_t phase = 0;
    volatile int *gfail = s_gfail + group;
    const uint32_t tiles = (n + kTcRows - 1) / kTcRows;
    const uint32_t lane_base = (uint32_t)(32 * (warp & 3)) << 16;
    float lo[3], ext[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = S->lo[a];
        ext[a] = S->hi[a] - S->lo[a];
    }

    // The groups run independently (own tiles, buffers, barrier, phase); tiles
    // go to the SMs before they go to the groups of one.
    // this thread's input row of the group's next tile, loaded one tile ahead
    const uint32_t tile_stride = gridDim.x * kTcGroups;
    uint32_t tile = blockIdx.x + gridDim.x * (uint32_t)group;
    rt_cache_input cur = {};
    if (tile < tiles && tile * kTcRows + (uint32_t)gtid < n) cur = in[tile * kTcRows + (uint32_t)gtid];
    for (; tile < tiles; tile += tile_stride) {
        // ---- encode this thread's row into the K = 96 input tile (a row past
        // the end encodes whatever the thread holds: its output is dropped)
        const uint32_t row = tile * kTcRows + (uint32_t)gtid;
        encode_to_tile(cur, lo, ext, tile_a, gtid);
        {
            const uint32_t nrow = (tile + tile_stride) * kTcRows + (uint32_t)gtid;
            if (tile + tile_stride < tiles && nrow < n) cur = in[nrow];  // in flight during the layers
        }
        fence_async_smem();
        tc_fence_before();
        group_sync(group);
        tc_fence_after();
        if (*gfail) break;  // read after the barrier: the same for the whole group
        bool failed = false;
#pragma unroll 1
        for (int l = 0; l < kLayers; ++l) {
            if (gtid == 0) {
                const uint32_t idesc = l == 5 ? tc_idesc(kTcRows, 16) : tc_idesc(kTcRows, 64);
                // accumulators = bias
                tc_mma(tmem, d_ones, d_bias + (uint32_t)l * (tc_tile_bytes(64, 16) >> 4), idesc, 0u);
                if (l == 0) {
#pragma unroll
                    for (uint32_t ks = 0; ks < 6u; ++ks) tc_mma(tmem, d_in + 16u * ks, d_w0 + 16u * ks, idesc, 1u);
                } else {
                    const uint64_t db = d_w1 + (uint32_t)(l - 1) * (tc_tile_bytes(64, 64) >> 4);
#pragma unroll
                    for (uint32_t ks = 0; ks < 4u; ++ks) tc_mma_ta(tmem, tmem + kTcACol + 8u * ks, db + 16u * ks, idesc);
                }
                tc_commit(bar_a);
            }
            if (!mbar_wait_bounded(bar_a, phase)) {
                report_error(err, RT_ERR_TIMEOUT, 0x90000000u | (uint32_t)l);
                mbar_wait_bounded(bar_a, phase);  // once more: no MMA may outlive the TMEM
                *gfail = 1;
            }
            phase ^= 1u;
            __syncwarp();
            tc_fence_after();
            if (l < 5) {
                // hidden layer: ReLU -> BF16 row, the next layer's A
                uint32_t v0[32], v1[32], p[32];
                tc_ld32(tmem + lane_base, v0);
                tc_ld32(tmem + lane_base + 32u, v1);
                tc_wait_ld(v0);
                tc_wait_ld(v1);
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    p[k] = relu_pack_bf16(__uint_as_float(v0[2 * k]), __uint_as_float(v0[2 * k + 1]));
                    p[16 + k] = relu_pack_bf16(__uint_as_float(v1[2 * k]), __uint_as_float(v1[2 * k + 1]));
                }
                tc_st32(tmem + lane_base + kTcACol, p);
                tc_wait_st();
            } else {
                uint32_t v[4];
                tc_ld4(tmem + lane_base, v);
                tc_wait_ld(v);
                if (row < n)
                    out[row] = make_float4(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]), 0.0f);
            }
            if (l < 5) {
                tc_fence_before();
                group_sync(group);
                tc_fence_after();
                failed = *gfail != 0;
                if (failed) break;
            }
        }
        if (failed) break;
        // the next tile's encoding may overwrite the input tile (layer 0 has
        // read it), and the barrier after it orders this tile's last TMEM
        // reads before the next MMAs
    }
    // ---- teardown: every MMA has been waited for (a group that gave up
    // waited once more); free the TMEM
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*tmem_slot), "r"(kTcTmemCols)
                     : "memory");
}

// One Adam step on every parameter; S->step already counts it (advanced by
// the k_cache_fwd_bwd launch before).  Thread 0 also hands the batch's mean
// loss to loss_out and clears it for the next batch.
__global__ void k_cache_adam(CacheState *S, float *loss_out) {
    pdl_launch();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    // written by earlier Adam steps only, which were complete when the launch
    // before this one (forward and backward) let this one start
    float m0 = 0.0f, v0 = 0.0f, p0 = 0.0f;
    if (i < kParams) {
        m0 = __ldcg(S->m + i);
        v0 = __ldcg(S->v + i);
        p0 = __ldcg(S->params + i);
    }
    pdl_wait();
    if (i == 0) {
        if (loss_out) *loss_out = S->loss;
        S->loss = 0.0f;
    }
    if (i >= kParams) return;
    const uint32_t t = S->step;
    const float g = S->grads[i];
    const float m = S->beta1 * m0 + (1.0f - S->beta1) * g;
    const float v = S->beta2 * v0 + (1.0f - S->beta2) * g * g;
    S->m[i] = m;
    S->v[i] = v;
    const float mh = m / (1.0f - powf(S->beta1, (float)t));
    const float vh = v / (1.0f - powf(S->beta2, (float)t));
    const float p = p0 - S->lr * mh / (sqrtf(vh) + S->eps);
    S->params[i] = p;
    S->wbf[i] = __float2bfloat16(p);
    S->grads[i] = 0.0f;
}

__global__ void k_cache_refresh_bf16(CacheState *S) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kParams) S->wbf[i] = __float2bfloat16(S->params[i]);
}

int set_smem(rt_context *ctx) {
    RT_CUDA_CTX(ctx, cudaFuncSetAttribute(k_cache_query_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem));
    RT_CUDA_CTX(ctx, cudaFuncSetAttribute(k_cache_fwd_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem));
    RT_CUDA_CTX(ctx, cudaFuncSetAttribute(k_cache_fwd_bwd_small<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)small_smem(32)));
    RT_CUDA_CTX(ctx, cudaFuncSetAttribute(k_cache_fwd_bwd_small<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)small_smem(64)));
    return RT_OK;
}

// One batch of at most n rows (n_dev: rows [row0, row0 + n) of *n_dev).
int launch_fwd_bwd(rt_context *ctx, cudaStream_t st, CacheState *S, const rt_cache_input *in, const float *tg,
                   uint32_t n, const uint32_t *n_dev, uint32_t row0, uint32_t bump_step, uint32_t after_adam) {
    if (n == 0) return RT_OK;
    const float inv = n_dev ? 0.0f : 1.0f / (3.0f * (float)n);
    const float4 *t4 = reinterpret_cast<const float4 *>(tg);
    const uint32_t sms = (uint32_t)ctx->sm_count;
    // the shortest chain while its reductions are few, one wave of 64-row tiles
    // while there is one (measured above the kernel)
    const uint32_t tiles32 = (n + 31u) / 32u, tiles64 = (n + 63u) / 64u;
    if (tiles32 <= 64u) {
        RT_CUDA_CTX(ctx, launch_pdl(k_cache_fwd_bwd_small<32>, tiles32, kTrainThreads, small_smem(32), st, S, in, t4, n,
                                    inv, n_dev, row0, bump_step, after_adam));
    } else if (tiles64 <= sms) {
        RT_CUDA_CTX(ctx, launch_pdl(k_cache_fwd_bwd_small<64>, tiles64, kTrainThreads, small_smem(64), st, S, in, t4, n,
                                    inv, n_dev, row0, bump_step, after_adam));
    } else {
        const uint32_t tiles = (n + kTrainRows - 1) / kTrainRows;
        RT_CUDA_CTX(ctx, launch_pdl(k_cache_fwd_bwd, tiles < sms ? tiles : sms, kTrainThreads, kTrainSmem, st, S, in,
                                    t4, n, inv, n_dev, row0, bump_step));
    }
    return RT_OK;
}

// He-uniform initial weights of the padded layout, host side (PCG32).
std::vector<float> initial_params(uint32_t seed) {
    std::vector<float> p(kParams, 0.0f);
    uint64_t state = 0, inc = ((uint64_t)seed << 1u) | 1u;
    auto next = [&]() {
        uint64_t old = state;
        state = old * 6364136223846793005ull + inc;
        uint32_t xs = (uint32_t)(((old >> 18u) ^ old) >> 27u), rot = (uint32_t)(old >> 59u);
        return (xs >> rot) | (xs << ((32u - rot) & 31u));
    };
    next();
    state += 0x853c49e6748fea9bull;
    next();
    const int used_in[kLayers] = {RT_CACHE_INPUTS, 64, 64, 64, 64, 64};
    const int used_out[kLayers] = {64, 64, 64, 64, 64, RT_CACHE_OUTPUTS};
    for (int l = 0; l < kLayers; ++l) {
        const float s = std::sqrt(6.0f / (float)used_in[l]);
        for (int o = 0; o < used_out[l]; ++o)
            for (int i = 0; i < used_in[l]; ++i) {
                float u = (float)(next() >> 8) * (1.0f / 16777216.0f);
                p[w_off(l) + o * in_dim(l) + i] = (2.0f * u - 1.0f) * s;
            }
    }
    return p;
}

}  // namespace
}  // namespace rtc

using namespace rtc;

extern "C" rt_status rt_cache_bytes(uint64_t *bytes) {
    if (!bytes) return RT_ERR_INVALID_ARG;
    *bytes = align_up(sizeof(CacheState), 256);
    return RT_OK;
}

extern "C" uint32_t rt_cache_param_count(void) { return (uint32_t)kParams; }

extern "C" rt_status rt_cache_init(rt_context *ctx, rt_stream stream, void *cache, const rt_cache_config *cfg) {
    if (!ctx || !cache || !cfg) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_init: null argument");
    if (reinterpret_cast<uintptr_t>(cache) & 255u) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_init: cache must be 256-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int rc = set_smem(ctx);
    if (rc) return rc;
    std::vector<uint8_t> h(sizeof(CacheState), 0);
    CacheState *hs = reinterpret_cast<CacheState *>(h.data());
    std::vector<float> p = initial_params(cfg->seed);
    std::memcpy(hs->params, p.data(), sizeof(float) * kParams);
    for (int i = 0; i < kParams; ++i) {
        __nv_bfloat16 b = __float2bfloat16(p[i]);
        hs->wbf[i] = b;
    }
    for (int a = 0; a < 3; ++a) { hs->lo[a] = cfg->scene_lo[a]; hs->hi[a] = cfg->scene_hi[a]; }
    hs->lr = cfg->lr;
    hs->beta1 = cfg->beta1;
    hs->beta2 = cfg->beta2;
    hs->eps = cfg->eps;
    RT_CUDA_CTX(ctx, cudaMemcpyAsync(cache, h.data(), h.size(), cudaMemcpyHostToDevice, st));
    RT_CUDA_CTX(ctx, cudaStreamSynchronize(st));
    return RT_OK;
}

extern "C" rt_status rt_cache_query(rt_context *ctx, rt_stream stream, const void *cache, const rt_cache_input *in,
                                    float *out, uint32_t n) {
    if (!ctx || !cache || (n && (!in || !out))) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_query: null argument");
    if (reinterpret_cast<uintptr_t>(cache) & 255u) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_query: cache must be 256-byte aligned");
    if (n == 0) return RT_OK;
    int rc = set_smem(ctx);
    if (rc) return rc;
    const uint32_t tiles = (n + kTcRows - 1) / kTcRows;
    uint32_t grid = (uint32_t)ctx->sm_count;
    if (grid > tiles) grid = tiles;
    k_cache_query_tc<<<grid, kTcThreads, kTcSmem, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const CacheState *>(cache), in, reinterpret_cast<float4 *>(out), n, nullptr, ctx->d_err);
    RT_CUDA_CTX(ctx, cudaGetLastError());
    return RT_OK;
}

extern "C" rt_status rt_cache_train(rt_context *ctx, rt_stream stream, void *cache, const rt_cache_input *in,
                                    const float *targets, uint32_t n, uint32_t batch, float *loss_out) {
    if (!ctx || !cache || (n && (!in || !targets))) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_train: null argument");
    if (reinterpret_cast<uintptr_t>(cache) & 255u) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_train: cache must be 256-byte aligned");
    if (batch == 0 || batch % 64u) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_train: batch must be a positive multiple of 64");
    int rc = set_smem(ctx);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    CacheState *S = static_cast<CacheState *>(cache);
    for (uint32_t b = 0; b < n; b += batch) {
        const uint32_t m = (n - b) < batch ? (n - b) : batch;
        rc = launch_fwd_bwd(ctx, st, S, in + b, targets + 4u * (size_t)b, m, nullptr, 0u, 1u, b ? 1u : 0u);
        if (rc) return rc;
        RT_CUDA_CTX(ctx, launch_pdl(k_cache_adam, (kParams + 255) / 256, 256, 0, st, S, loss_out));
    }
    return RT_OK;
}

extern "C" rt_status rt_cache_gradient(rt_context *ctx, rt_stream stream, void *cache, const rt_cache_input *in,
                                       const float *targets, uint32_t n, float *grad_out) {
    if (!ctx || !cache || !grad_out || (n && (!in || !targets)))
        return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_gradient: null argument");
    if (reinterpret_cast<uintptr_t>(cache) & 255u) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_gradient: cache must be 256-byte aligned");
    int rc = set_smem(ctx);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    CacheState *S = static_cast<CacheState *>(cache);
    RT_CUDA_CTX(ctx, cudaMemsetAsync(S->grads, 0, sizeof(float) * kParams, st));
    rc = launch_fwd_bwd(ctx, st, S, in, targets, n, nullptr, 0u, 0u, 0u);
    if (rc) return rc;
    RT_CUDA_CTX(ctx, cudaMemcpyAsync(grad_out, S->grads, sizeof(float) * kParams, cudaMemcpyDeviceToDevice, st));
    RT_CUDA_CTX(ctx, cudaMemsetAsync(S->grads, 0, sizeof(float) * kParams, st));
    RT_CUDA_CTX(ctx, cudaMemsetAsync(&S->loss, 0, sizeof(float), st));
    return RT_OK;
}

extern "C" rt_status rt_cache_get_params(rt_context *ctx, rt_stream stream, const void *cache, float *params) {
    if (!ctx || !cache || !params) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_get_params: null argument");
    const CacheState *S = static_cast<const CacheState *>(cache);
    RT_CUDA_CTX(ctx, cudaMemcpyAsync(params, S->params, sizeof(float) * kParams, cudaMemcpyDeviceToDevice,
                                     static_cast<cudaStream_t>(stream)));
    return RT_OK;
}

extern "C" rt_status rt_cache_set_params(rt_context *ctx, rt_stream stream, void *cache, const float *params) {
    if (!ctx || !cache || !params) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_set_params: null argument");
    if (reinterpret_cast<uintptr_t>(cache) & 255u) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_set_params: cache must be 256-byte aligned");
    CacheState *S = static_cast<CacheState *>(cache);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RT_CUDA_CTX(ctx, cudaMemcpyAsync(S->params, params, sizeof(float) * kParams, cudaMemcpyDeviceToDevice, st));
    k_cache_refresh_bf16<<<(kParams + 255) / 256, 256, 0, st>>>(S);
    RT_CUDA_CTX(ctx, cudaGetLastError());
    return RT_OK;
}

// ---------------------------------------------------------------------------
// Checkpoints
// ---------------------------------------------------------------------------

namespace {

struct CheckpointHeader {
    char magic[4];         // "RTMC"
    uint32_t version;      // 1
    uint32_t params;       // kParams
    uint32_t reserved0;
    uint64_t state_bytes;  // sizeof(CacheState)
    uint64_t checksum;     // FNV-1a 64 of the state bytes
    uint8_t reserved[32];
};
static_assert(sizeof(CheckpointHeader) == 64, "checkpoint header");

uint64_t fnv1a64(const uint8_t *p, size_t n) {
    uint64_t h = 0xcbf29ce484222325ull;
    for (size_t i = 0; i < n; ++i) {
        h ^= p[i];
        h *= 0x100000001b3ull;
    }
    return h;
}

}  // namespace

extern "C" rt_status rt_cache_save(rt_context *ctx, rt_stream stream, const void *cache, const char *path) {
    if (!ctx || !cache || !path) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_save: null argument");
    std::vector<uint8_t> state(sizeof(CacheState));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RT_CUDA_CTX(ctx, cudaMemcpyAsync(state.data(), cache, state.size(), cudaMemcpyDeviceToHost, st));
    RT_CUDA_CTX(ctx, cudaStreamSynchronize(st));
    CheckpointHeader h;
    std::memset(&h, 0, sizeof(h));
    std::memcpy(h.magic, "RTMC", 4);
    h.version = 1u;
    h.params = (uint32_t)kParams;
    h.state_bytes = state.size();
    h.checksum = fnv1a64(state.data(), state.size());
    const std::string tmp = std::string(path) + ".tmp";
    FILE *f = std::fopen(tmp.c_str(), "wb");
    if (!f) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_save: cannot open the file for writing");
    bool ok = std::fwrite(&h, sizeof(h), 1, f) == 1 && std::fwrite(state.data(), 1, state.size(), f) == state.size();
    ok = (std::fclose(f) == 0) && ok;
    if (!ok || std::rename(tmp.c_str(), path) != 0) {
        std::remove(tmp.c_str());
        return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_save: write failed");
    }
    return RT_OK;
}

extern "C" rt_status rt_cache_load(rt_context *ctx, rt_stream stream, void *cache, const char *path) {
    if (!ctx || !cache || !path) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_load: null argument");
    FILE *f = std::fopen(path, "rb");
    if (!f) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_load: cannot open the file");
    CheckpointHeader h;
    std::vector<uint8_t> state(sizeof(CacheState));
    const bool got = std::fread(&h, sizeof(h), 1, f) == 1 &&
                     std::memcmp(h.magic, "RTMC", 4) == 0 && h.version == 1u && h.params == (uint32_t)kParams &&
                     h.state_bytes == state.size() && std::fread(state.data(), 1, state.size(), f) == state.size();
    const bool at_end = got && std::fgetc(f) == EOF;
    std::fclose(f);
    if (!got || !at_end)
        return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_load: not a cache checkpoint of this network");
    if (fnv1a64(state.data(), state.size()) != h.checksum)
        return set_error(ctx, RT_ERR_INVALID_ARG, "rt_cache_load: checksum mismatch");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RT_CUDA_CTX(ctx, cudaMemcpyAsync(cache, state.data(), state.size(), cudaMemcpyHostToDevice, st));
    RT_CUDA_CTX(ctx, cudaStreamSynchronize(st));
    return RT_OK;
}

// ---------------------------------------------------------------------------
// Device-count launchers for the path tracer's learned form (no host reads,
// no allocation): the number of query / training rows is produced on the
// device by the shading kernels.
// ---------------------------------------------------------------------------
namespace rtc {

int cache_query_dev(rt_context *ctx, cudaStream_t st, const void *cache, const rt_cache_input *in, float *out,
                    const uint32_t *n_dev, uint32_t max_n) {
    if (max_n == 0) return RT_OK;
    int rc = set_smem(ctx);
    if (rc) return rc;
    const uint32_t tiles = (max_n + kTcRows - 1) / kTcRows;
    uint32_t grid = (uint32_t)ctx->sm_count;
    if (grid > tiles) grid = tiles;
    k_cache_query_tc<<<grid, kTcThreads, kTcSmem, st>>>(static_cast<const CacheState *>(cache), in,
                                                 reinterpret_cast<float4 *>(out), max_n, n_dev, ctx->d_err);
    RT_CUDA_CTX(ctx, cudaGetLastError());
    return RT_OK;
}

// Adam steps over the first *n_dev samples in batches of `batch` (at most
// max_n samples in total).
int cache_train_dev(rt_context *ctx, cudaStream_t st, void *cache, const rt_cache_input *in, const float *targets,
                    const uint32_t *n_dev, uint32_t max_n, uint32_t batch) {
    if (max_n == 0 || batch == 0) return RT_OK;
    int rc = set_smem(ctx);
    if (rc) return rc;
    CacheState *S = static_cast<CacheState *>(cache);
    for (uint32_t b = 0; b < max_n; b += batch) {
        const uint32_t m = (max_n - b) < batch ? (max_n - b) : batch;
        rc = launch_fwd_bwd(ctx, st, S, in, targets, m, n_dev, b, 1u, b ? 1u : 0u);
        if (rc) return rc;
        RT_CUDA_CTX(ctx, launch_pdl(k_cache_adam, (kParams + 255) / 256, 256, 0, st, S,
                                    static_cast<float *>(nullptr)));
    }
    return RT_OK;
}

}  // namespace rtc
