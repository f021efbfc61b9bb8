// Learned coarse-grid closure: a small MLP (96 -> 128 -> 128 -> 128 -> 48, GELU on the hidden
// layers) with BF16 weights and activations and FP32 accumulation, with its own inference,
// training-forward, backward, gradient-reduction and Adam kernels, plus the closure's feature
// extraction from a coarse state and the application of its correction to an RK stage.
//
// Matrix products run on the tensor cores with mma.sync.m16n8k16 (bf16 x bf16 -> f32).  The forward
// and the backpropagation kernels give a CTA 32 samples and split a layer's output columns over its 8
// warps: activations pass from layer to layer through shared memory (ldmatrix), where the next layer's
// weights arrive by cp.async meanwhile, from the two layouts kept by the optimizer ([out][in] forward,
// [in][out] backward).  The weight gradients H^T dZ are one kernel over output tiles (mlp_grad_kernel).
// At minibatches of this size all three are bound by the latency of their chains (layers, summation
// blocks), not by a rate.  Minibatch of 8192: forward 14 us (28.9 with one warp per 16 samples carrying the
// whole network in its registers), backward 51 us (110 with the gradients of every 64 samples written as
// a partial and reduced); of 576: 9 and 17 us (28 and 97).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>

#include "vlasov1d2v.h"

void vl_internal_set_error(const char *msg);

namespace {

constexpr int IN = 96, HID = 128, OUT = 48;
constexpr int NL = 4;                          // layers
constexpr int WARPS = 8, ROWS = 32;            // warps and samples per CTA (forward, backpropagation)
constexpr int BLOCK = 64;                      // samples per summation block of the gradients
__host__ __device__ constexpr int layer_in(int l) { return l == 0 ? IN : HID; }
__host__ __device__ constexpr int layer_out(int l) { return l == NL - 1 ? OUT : HID; }

struct MlpWeights {
    const __nv_bfloat16 *wf[NL];   // [out][in]
    const __nv_bfloat16 *wb[NL];   // [in][out]
    const float *bias[NL];         // [out]
};

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// GELU(x) = x Phi(x) and its derivative Phi(x) + x phi(x) (erf form)
__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float x) {
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * __expf(-0.5f * x * x);
    return cdf + x * pdf;
}

// shared-memory row stride (bf16) of a K-wide activation tile: an odd number of 16-byte units, so the
// eight rows of an ldmatrix fall in distinct banks
__host__ __device__ constexpr int act_stride(int K) { return K + 8; }

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const __nv_bfloat16 *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const __nv_bfloat16 *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

__device__ __forceinline__ void cp16(void *dst, const void *src, bool in = true) {   // (zeros when !in)
    const int bytes = in ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes)
                 : "memory");
}

// a layer's weights [N][K] (bf16) to shared memory, rows of act_stride(K)
template <int K, int N>
__device__ __forceinline__ void stage_weights(__nv_bfloat16 *sW, const __nv_bfloat16 *__restrict__ w) {
    if ((reinterpret_cast<uintptr_t>(w) & 15) == 0) {
        for (int q = threadIdx.x; q < N * K / 8; q += 32 * WARPS) {
            const int n = q / (K / 8), c = 8 * (q - n * (K / 8));
            cp16(sW + n * act_stride(K) + c, w + n * K + c);
        }
    } else {   // not on a 16-byte boundary: pairs
        for (int q = threadIdx.x; q < N * K / 2; q += 32 * WARPS) {
            const int n = q / (K / 2), c = 2 * (q - n * (K / 2));
            *reinterpret_cast<uint32_t *>(sW + n * act_stride(K) + c) =
                __ldg(reinterpret_cast<const uint32_t *>(w + n * K + c));
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int LEFT>
__device__ __forceinline__ void weights_ready() {   // all but the last LEFT staged layers, and the activations
    asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
    __syncthreads();
}

// acc[row tile][column tile][4] = A (the CTA's ROWS x K activations) . the warp's weight columns
template <int K, int NT>
__device__ __forceinline__ void layer_mma(const __nv_bfloat16 *sA, const __nv_bfloat16 *sW, int n0, int lane,
                                          float (&acc)[ROWS / 16][NT][4]) {
    const __nv_bfloat16 *pw = sW + (8 * n0 + (lane & 7)) * act_stride(K) + (lane >> 3) * 8;
    uint32_t b[NT][4];   // two k tiles of each column tile
    const __nv_bfloat16 *p = sA + ((lane & 7) + ((lane >> 3) & 1) * 8) * act_stride(K) + (lane >> 4) * 8;
#pragma unroll
    for (int mm = 0; mm < ROWS / 16; ++mm)
#pragma unroll
        for (int nn = 0; nn < NT; ++nn) acc[mm][nn][0] = acc[mm][nn][1] = acc[mm][nn][2] = acc[mm][nn][3] = 0.0f;
#pragma unroll
    for (int kk = 0; kk < K / 16; ++kk) {
        if (kk % 2 == 0) {   // (the last k tile of an odd count: its own columns again as the second half)
#pragma unroll
            for (int nn = 0; nn < NT; ++nn) {
                if (kk + 1 < K / 16)
                    ldsm_x4(b[nn], pw + 8 * nn * act_stride(K) + 16 * kk);
                else
                    ldsm_x4(b[nn], pw + 8 * nn * act_stride(K) + 16 * kk - (lane >> 4) * 16);
            }
        }
#pragma unroll
        for (int mm = 0; mm < ROWS / 16; ++mm) {
            uint32_t a[4];
            ldsm_x4(a, p + mm * 16 * act_stride(K) + 16 * kk);
#pragma unroll
            for (int nn = 0; nn < NT; ++nn) mma_bf16(acc[mm][nn], a, b[nn][2 * (kk & 1)], b[nn][2 * (kk & 1) + 1]);
        }
    }
}

// dynamic shared memory of the two kernels: two activation tiles, two layers' weights (bf16 elements)
constexpr int SMEM_A = ROWS * act_stride(HID), SMEM_W = HID * act_stride(HID);
constexpr int MLP_SMEM = (2 * SMEM_A + 2 * SMEM_W) * (int)sizeof(__nv_bfloat16);

// ---------------------------------------------------------------------------------------------
// forward: Y = MLP(X); with H0 also H_l (bf16 layer inputs) and Z_l (FP32 hidden pre-activations) for
// the backward pass.  One CTA per ROWS samples.
// ---------------------------------------------------------------------------------------------
// one hidden layer: bias, pre-activation out, GELU, bf16 activation to the next tile (and out)
template <int K>
__device__ __forceinline__ void forward_hidden(const __nv_bfloat16 *sA, const __nv_bfloat16 *sW,
                                               const float *__restrict__ bias, int n0, int row0, int nrows, int lane,
                                               float *__restrict__ Z, __nv_bfloat16 *__restrict__ H,
                                               __nv_bfloat16 *sNext) {
    const int g = lane >> 2, t = lane & 3;
    float acc[ROWS / 16][2][4];
    layer_mma<K, 2>(sA, sW, n0, lane, acc);
#pragma unroll
    for (int nn = 0; nn < 2; ++nn) {
        const int c = 8 * (n0 + nn) + 2 * t;
        const float b0 = __ldg(bias + c), b1 = __ldg(bias + c + 1);
#pragma unroll
        for (int mm = 0; mm < ROWS / 16; ++mm)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = 16 * mm + 8 * h + g, row = row0 + r;
                const float z0 = acc[mm][nn][2 * h] + b0, z1 = acc[mm][nn][2 * h + 1] + b1;
                const uint32_t hv = pack_bf16(gelu(z0), gelu(z1));
                *reinterpret_cast<uint32_t *>(sNext + r * act_stride(HID) + c) = hv;
                if (Z != nullptr && row < nrows) {
                    *reinterpret_cast<float2 *>(Z + (size_t)row * HID + c) = make_float2(z0, z1);
                    *reinterpret_cast<uint32_t *>(H + (size_t)row * HID + c) = hv;
                }
            }
    }
}

__global__ void __launch_bounds__(32 * WARPS) mlp_forward_kernel(const float *__restrict__ X, int nrows,
                                                                  MlpWeights w, float *__restrict__ Y,
                                                                  __nv_bfloat16 *__restrict__ H0,
                                                                  __nv_bfloat16 *__restrict__ Hh,
                                                                  float *__restrict__ Z) {
    extern __shared__ __align__(16) __nv_bfloat16 mlp_smem[];
    __nv_bfloat16 *sA[2] = {mlp_smem, mlp_smem + SMEM_A}, *sW[2] = {mlp_smem + 2 * SMEM_A, mlp_smem + 2 * SMEM_A + SMEM_W};
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int row0 = blockIdx.x * ROWS;
    stage_weights<IN, HID>(sW[0], w.wf[0]);
    stage_weights<HID, HID>(sW[1], w.wf[1]);
    for (int q = tid; q < ROWS * IN / 2; q += 32 * WARPS) {   // input, rounded to bf16
        const int r = q / (IN / 2), c = 2 * (q - r * (IN / 2)), row = row0 + r;
        uint32_t v = 0u;
        if (row < nrows) {
            const float2 x = *reinterpret_cast<const float2 *>(X + (size_t)row * IN + c);
            v = pack_bf16(x.x, x.y);
            if (H0) *reinterpret_cast<uint32_t *>(H0 + (size_t)row * IN + c) = v;
        }
        *reinterpret_cast<uint32_t *>(&sA[0][r * act_stride(IN) + c]) = v;
    }
    const size_t hs = (size_t)nrows * HID;
    weights_ready<1>();
    forward_hidden<IN>(sA[0], sW[0], w.bias[0], 2 * wp, row0, nrows, lane, Z, Hh, sA[1]);
    weights_ready<0>();
    stage_weights<HID, HID>(sW[0], w.wf[2]);
    forward_hidden<HID>(sA[1], sW[1], w.bias[1], 2 * wp, row0, nrows, lane, Z ? Z + hs : nullptr, Hh + hs, sA[0]);
    weights_ready<0>();
    stage_weights<HID, OUT>(sW[1], w.wf[NL - 1]);
    forward_hidden<HID>(sA[0], sW[0], w.bias[2], 2 * wp, row0, nrows, lane, Z ? Z + 2 * hs : nullptr, Hh + 2 * hs, sA[1]);
    weights_ready<0>();
    if (wp < OUT / 8) {
        float acc[ROWS / 16][1][4];
        layer_mma<HID, 1>(sA[1], sW[1], wp, lane, acc);
        const int c = 8 * wp + 2 * t;
        const float y0 = __ldg(w.bias[NL - 1] + c), y1 = __ldg(w.bias[NL - 1] + c + 1);
#pragma unroll
        for (int mm = 0; mm < ROWS / 16; ++mm)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = row0 + 16 * mm + 8 * h + g;
                if (row < nrows)
                    *reinterpret_cast<float2 *>(Y + (size_t)row * OUT + c) =
                        make_float2(acc[mm][0][2 * h] + y0, acc[mm][0][2 * h + 1] + y1);
            }
    }
}

// ---------------------------------------------------------------------------------------------
// backward of the mean-squared loss over the first nout outputs:
//   L = sum_rows sum_{c < nout} (Y - T)^2 / (nrows nout)
// mlp_backprop_kernel: dZ of every layer (dH = dZ W^T, dZ = dH * GELU'(Z)), bf16, zero rows up to a
// multiple of BLOCK samples.  mlp_grad_kernel: gW_l = H_l^T dZ_l and gb_l = sum of dZ_l.
// ---------------------------------------------------------------------------------------------
constexpr int GW_ELEMS = IN * HID + 2 * HID * HID + HID * OUT;   // weight elements
constexpr int GB_ELEMS = 3 * HID + OUT;                          // bias elements
__host__ __device__ constexpr int w_off(int l) { return l == 0 ? 0 : IN * HID + (l - 1) * HID * HID; }
__host__ __device__ constexpr int b_off(int l) { return l * HID; }

// dZ buffers, back to back: three hidden layers [rows][HID], then the output layer [rows][OUT]
__host__ __device__ constexpr size_t dz_off(int l, size_t rows) { return (size_t)l * rows * HID; }

// dZ of a hidden layer from the next layer's dZ (sD, K wide): W^T given as wb [HID][K]
template <int K>
__device__ __forceinline__ void backprop_hidden(const __nv_bfloat16 *sD, const __nv_bfloat16 *sW,
                                                const float *__restrict__ Z, bool z8, int n0, int row0, int nrows,
                                                int lane, __nv_bfloat16 *__restrict__ dZ, __nv_bfloat16 *sNext) {
    const int g = lane >> 2, t = lane & 3;
    float acc[ROWS / 16][2][4];
    layer_mma<K, 2>(sD, sW, n0, lane, acc);
#pragma unroll
    for (int nn = 0; nn < 2; ++nn) {
        const int c = 8 * (n0 + nn) + 2 * t;
#pragma unroll
        for (int mm = 0; mm < ROWS / 16; ++mm)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = 16 * mm + 8 * h + g, row = row0 + r;
                float d0 = 0.f, d1 = 0.f;
                if (row < nrows) {
                    const float *pz = Z + (size_t)row * HID + c;
                    const float2 z = z8 ? *reinterpret_cast<const float2 *>(pz) : make_float2(pz[0], pz[1]);
                    d0 = acc[mm][nn][2 * h] * gelu_d(z.x);
                    d1 = acc[mm][nn][2 * h + 1] * gelu_d(z.y);
                }
                const uint32_t v = pack_bf16(d0, d1);
                *reinterpret_cast<uint32_t *>(dZ + (size_t)row * HID + c) = v;
                *reinterpret_cast<uint32_t *>(sNext + r * act_stride(HID) + c) = v;
            }
    }
}

__global__ void __launch_bounds__(32 * WARPS) mlp_backprop_kernel(const float *__restrict__ Y,
                                                                   const float *__restrict__ T, int nrows, int nout,
                                                                   MlpWeights w, const float *__restrict__ Z,
                                                                   __nv_bfloat16 *__restrict__ dZ, int rows) {
    extern __shared__ __align__(16) __nv_bfloat16 mlp_smem[];
    __nv_bfloat16 *sD[2] = {mlp_smem, mlp_smem + SMEM_A}, *sW[2] = {mlp_smem + 2 * SMEM_A, mlp_smem + 2 * SMEM_A + SMEM_W};
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int row0 = blockIdx.x * ROWS;
    stage_weights<OUT, HID>(sW[0], w.wb[NL - 1]);
    stage_weights<HID, HID>(sW[1], w.wb[2]);
    const float scale = 2.0f / ((float)nrows * (float)nout);
    for (int q = tid; q < ROWS * OUT / 2; q += 32 * WARPS) {   // dZ of the output layer (linear): dL/dY
        const int r = q / (OUT / 2), c = 2 * (q - r * (OUT / 2)), row = row0 + r;
        float v0 = 0.f, v1 = 0.f;
        if (row < nrows) {
            if (c < nout) v0 = scale * (Y[(size_t)row * OUT + c] - T[(size_t)row * nout + c]);
            if (c + 1 < nout) v1 = scale * (Y[(size_t)row * OUT + c + 1] - T[(size_t)row * nout + c + 1]);
        }
        const uint32_t v = pack_bf16(v0, v1);
        *reinterpret_cast<uint32_t *>(&sD[0][r * act_stride(OUT) + c]) = v;
        *reinterpret_cast<uint32_t *>(dZ + dz_off(NL - 1, rows) + (size_t)row * OUT + c) = v;
    }
    const size_t hs = (size_t)nrows * HID;
    const bool z8 = (reinterpret_cast<uintptr_t>(Z) & 7) == 0;   // (elsewhere single floats)
    weights_ready<1>();
    backprop_hidden<OUT>(sD[0], sW[0], Z + 2 * hs, z8, 2 * wp, row0, nrows, lane, dZ + dz_off(2, rows), sD[1]);
    weights_ready<0>();
    stage_weights<HID, HID>(sW[0], w.wb[1]);
    backprop_hidden<HID>(sD[1], sW[1], Z + hs, z8, 2 * wp, row0, nrows, lane, dZ + dz_off(1, rows), sD[0]);
    weights_ready<0>();
    backprop_hidden<HID>(sD[0], sW[0], Z, z8, 2 * wp, row0, nrows, lane, dZ + dz_off(0, rows), sD[1]);
}

// Gradients.  CTA < GRAD_TILES: a 16 x 32 tile of one layer's gW (warp: 16 x 8) over all samples, which
// stream through shared memory 256 at a time; a block of BLOCK samples is one chain of four MMAs, added
// to the running FP32 sum in the order of the blocks.  The other CTAs: four columns of gb, one thread
// per block of samples, then their sums in order.  No partial gradients in memory (26 MB written and read
// back per minibatch of 8192 with one partial per block).
constexpr int GM = 16, GN = 32, GCH = 4 * BLOCK, GST = 3;   // tile, samples per stage, stages
constexpr int SHS = GM + 8, SDS = GN + 8;                   // row strides: 48 and 80 bytes, conflict-free
constexpr int GRAD_THREADS = 128;
constexpr int GRAD_SMEM = GST * GCH * (SHS + SDS) * (int)sizeof(__nv_bfloat16);
__host__ __device__ constexpr int grad_ngroups(int l) { return (layer_out(l) + GN - 1) / GN; }
__host__ __device__ constexpr int grad_tiles(int l) { return layer_in(l) / GM * grad_ngroups(l); }
constexpr int GRAD_TILES = grad_tiles(0) + grad_tiles(1) + grad_tiles(2) + grad_tiles(3);
constexpr int BIAS_CTAS = GB_ELEMS / 4;

__global__ void __launch_bounds__(GRAD_THREADS) mlp_grad_kernel(const __nv_bfloat16 *__restrict__ H0,
                                                                 const __nv_bfloat16 *__restrict__ Hh,
                                                                 const __nv_bfloat16 *__restrict__ dZ, int nrows,
                                                                 int rows, bool h16, float *__restrict__ grad_w,
                                                                 float *__restrict__ grad_b) {
    extern __shared__ __align__(16) __nv_bfloat16 mlp_smem[];
    __nv_bfloat16(*sH)[GCH * SHS] = reinterpret_cast<__nv_bfloat16(*)[GCH * SHS]>(mlp_smem);
    __nv_bfloat16(*sD)[GCH * SDS] = reinterpret_cast<__nv_bfloat16(*)[GCH * SDS]>(mlp_smem + GST * GCH * SHS);
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    if (blockIdx.x >= GRAD_TILES) {
        // bias columns [c, c + 4) of layer l
        int c = (blockIdx.x - GRAD_TILES) * 4, l = 0;
        while (l < NL - 1 && c >= b_off(l + 1)) ++l;
        const int N = layer_out(l), n = c - b_off(l);
        const __nv_bfloat16 *d = dZ + dz_off(l, rows) + n;
        float(*sS)[4] = reinterpret_cast<float(*)[4]>(&sH[0][0]);
        float total = 0.f;
        for (int b0 = 0; b0 < rows / BLOCK; b0 += GRAD_THREADS) {
            const int b = b0 + tid;
            if (b < rows / BLOCK) {
                float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 16
                for (int r = 0; r < BLOCK; ++r) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(d + (size_t)(b * BLOCK + r) * N));
                    const float2 p = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&v.x));
                    const float2 q = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&v.y));
                    s[0] += p.x;
                    s[1] += p.y;
                    s[2] += q.x;
                    s[3] += q.y;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) sS[tid][k] = s[k];
            }
            __syncthreads();
            if (tid < 4) {
                const int nb = min(GRAD_THREADS, rows / BLOCK - b0);
                for (int k = 0; k < nb; ++k) total += sS[k][tid];
            }
            __syncthreads();
        }
        if (tid < 4) grad_b[c + tid] = total;
        return;
    }
    int q = blockIdx.x, l = 0;
    while (l < NL - 1 && q >= grad_tiles(l)) q -= grad_tiles(l++);
    const int K = layer_in(l), N = layer_out(l);
    const int m0 = q / grad_ngroups(l) * GM, n0 = q % grad_ngroups(l) * GN;
    const int ncol = min(GN, N - n0);   // 32, or 16 in the last group of the output layer
    const __nv_bfloat16 *h = (l == 0 ? H0 : Hh + (size_t)(l - 1) * nrows * HID) + m0;
    const __nv_bfloat16 *d = dZ + dz_off(l, rows) + n0;
    const int chunks = (rows + GCH - 1) / GCH;
    auto issue = [&](int ch) {
        const int r0 = ch * GCH, s = ch % GST;
        if (h16) {
            for (int k = tid; k < GCH * GM / 8; k += GRAD_THREADS) {
                const int r = k / (GM / 8), c = 8 * (k % (GM / 8));
                const bool in = r0 + r < nrows;
                cp16(&sH[s][r * SHS + c], h + (in ? (size_t)(r0 + r) * K + c : 0), in);
            }
        } else {   // layer inputs not on 16-byte boundaries: pairs
            for (int k = tid; k < GCH * GM / 2; k += GRAD_THREADS) {
                const int r = k / (GM / 2), c = 2 * (k % (GM / 2));
                *reinterpret_cast<uint32_t *>(&sH[s][r * SHS + c]) =
                    r0 + r < nrows ? *reinterpret_cast<const uint32_t *>(h + (size_t)(r0 + r) * K + c) : 0u;
            }
        }
        for (int k = tid; k < GCH * GN / 8; k += GRAD_THREADS) {
            const int r = k / (GN / 8), c = 8 * (k % (GN / 8));
            const bool in = r0 + r < rows && c < ncol;
            cp16(&sD[s][r * SDS + c], d + (in ? (size_t)(r0 + r) * N + c : 0), in);
        }
    };
#pragma unroll
    for (int ch = 0; ch < GST - 1; ++ch) {
        if (ch < chunks) issue(ch);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
    const int ra = (lane & 7) + ((lane >> 4) & 1) * 8, ca = ((lane >> 3) & 1) * 8;   // A: H^T, transposed reads
    const int rb = lane, cb = 8 * wp;                                               // B: dZ, 32 samples
    for (int ch = 0; ch < chunks; ++ch) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GST - 2) : "memory");
        __syncthreads();   // chunk ch is in shared memory, chunk ch - 1 consumed
        if (ch + GST - 1 < chunks) issue(ch + GST - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const int s = ch % GST;
        // the chunk's blocks are independent chains, then added in their order (blocks past the last
        // sample are zeros)
        constexpr int NB = GCH / BLOCK;
        float acc[NB][4];
#pragma unroll
        for (int bk = 0; bk < NB; ++bk) acc[bk][0] = acc[bk][1] = acc[bk][2] = acc[bk][3] = 0.f;
        const __nv_bfloat16 *ph = &sH[s][ra * SHS + ca], *pd = &sD[s][rb * SDS + cb];
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) {
            uint32_t b[NB][4];
#pragma unroll
            for (int bk = 0; bk < NB; ++bk) ldsm_x4_t(b[bk], pd + (bk * BLOCK + 32 * k2) * SDS);
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                uint32_t a[NB][4];
#pragma unroll
                for (int bk = 0; bk < NB; ++bk) ldsm_x4_t(a[bk], ph + (bk * BLOCK + 32 * k2 + 16 * kk) * SHS);
#pragma unroll
                for (int bk = 0; bk < NB; ++bk) mma_bf16(acc[bk], a[bk], b[bk][2 * kk], b[bk][2 * kk + 1]);
            }
        }
#pragma unroll
        for (int bk = 0; bk < NB; ++bk)
#pragma unroll
            for (int k = 0; k < 4; ++k) sum[k] += acc[bk][k];
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (8 * wp >= ncol) return;
    const int g = lane >> 2, t = lane & 3;
    float *gw = grad_w + w_off(l) + (size_t)(m0 + g) * N + n0 + 8 * wp + 2 * t;
    // (single floats: grad_w may start on any float)
    gw[0] = sum[0];
    gw[1] = sum[1];
    gw[(size_t)8 * N] = sum[2];
    gw[(size_t)8 * N + 1] = sum[3];
}

// Adam on the FP32 master weights [in][out] and biases; refresh both bf16 layouts
__global__ void mlp_adam_kernel(float *__restrict__ master_w, float *__restrict__ master_b,
                                const float *__restrict__ gw, const float *__restrict__ gb,
                                float *__restrict__ mw, float *__restrict__ vw, float *__restrict__ mb,
                                float *__restrict__ vb, __nv_bfloat16 *__restrict__ wf,
                                __nv_bfloat16 *__restrict__ wb, float lr, float b1, float b2, float eps,
                                float bc1, float bc2, float wd) {
    const int nw = GW_ELEMS, nb = GB_ELEMS;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nw + nb; i += gridDim.x * blockDim.x) {
        if (i < nw) {
            const float gr = gw[i];
            const float m = b1 * mw[i] + (1.f - b1) * gr;
            const float v = b2 * vw[i] + (1.f - b2) * gr * gr;
            mw[i] = m;
            vw[i] = v;
            float p = master_w[i];
            p -= lr * ((m / bc1) / (sqrtf(v / bc2) + eps) + wd * p);
            master_w[i] = p;
            // layer and position of element i ([in][out] within the layer)
            int l = 0;
            while (l < NL - 1 && i >= w_off(l + 1)) ++l;
            const int K = layer_in(l), N = layer_out(l);
            const int j = i - w_off(l), k = j / N, n = j - (j / N) * N;
            const __nv_bfloat16 h = __float2bfloat16_rn(p);
            wb[w_off(l) + k * N + n] = h;
            wf[w_off(l) + n * K + k] = h;
        } else {
            const int j = i - nw;
            const float gr = gb[j];
            const float m = b1 * mb[j] + (1.f - b1) * gr;
            const float v = b2 * vb[j] + (1.f - b2) * gr * gr;
            mb[j] = m;
            vb[j] = v;
            master_b[j] -= lr * (m / bc1) / (sqrtf(v / bc2) + eps);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// closure features and correction (coarse grid, order CN = 6)
//   sample (e, i, a, b): x node i of interior x element e, interior velocity element (a, b)
//   features: the element's 6 x 6 nodal patch f[e, i, a, :, b, :], the neighbour traces of the
//   four adjacent velocity elements (their first and second node lines next to the shared face),
//   each divided by the sample's scale max|.|; then a E_i / escale, the element's centre u / umax
//   and v / vmax, and a B; zero padding to IN.
// ---------------------------------------------------------------------------------------------
constexpr int CN = 6;
constexpr int NF = CN * CN + 8 * CN;   // 84 state values

template <typename T>
__global__ void closure_features_kernel(const T *__restrict__ f, int nx, int nu, int nv,
                                        const double *__restrict__ E, double accel, double bfield,
                                        const double *__restrict__ un, const double *__restrict__ vn,
                                        double umax, double vmax, double escale, float *__restrict__ X,
                                        float *__restrict__ scale) {
    const int U = nu + 2, V = nv + 2;
    const long sJ = (long)V * CN, sA = sJ * CN, sI = sA * U, sE = sI * CN;
    const long total = (long)nx * CN * nu * nv;
    for (long s = blockIdx.x * (long)blockDim.x + threadIdx.x; s < total; s += (long)gridDim.x * blockDim.x) {
        long r = s;
        const int b = (int)(r % nv) + 1; r /= nv;
        const int a = (int)(r % nu) + 1; r /= nu;
        const int i = (int)(r % CN); r /= CN;
        const int e = (int)r + 1;
        const T *p = f + e * sE + i * sI;
        float v[NF];
        int q = 0;
        for (int j = 0; j < CN; ++j)
            for (int k = 0; k < CN; ++k) v[q++] = (float)p[a * sA + j * sJ + b * CN + k];
        for (int k = 0; k < CN; ++k) v[q++] = (float)p[(a - 1) * sA + (CN - 1) * sJ + b * CN + k];
        for (int k = 0; k < CN; ++k) v[q++] = (float)p[(a + 1) * sA + 0 * sJ + b * CN + k];
        for (int j = 0; j < CN; ++j) v[q++] = (float)p[a * sA + j * sJ + (b - 1) * CN + CN - 1];
        for (int j = 0; j < CN; ++j) v[q++] = (float)p[a * sA + j * sJ + (b + 1) * CN + 0];
        for (int k = 0; k < CN; ++k) v[q++] = (float)p[(a - 1) * sA + (CN - 2) * sJ + b * CN + k];
        for (int k = 0; k < CN; ++k) v[q++] = (float)p[(a + 1) * sA + 1 * sJ + b * CN + k];
        for (int j = 0; j < CN; ++j) v[q++] = (float)p[a * sA + j * sJ + (b - 1) * CN + CN - 2];
        for (int j = 0; j < CN; ++j) v[q++] = (float)p[a * sA + j * sJ + (b + 1) * CN + 1];
        float m = 0.f;
        for (int c = 0; c < NF; ++c) m = fmaxf(m, fabsf(v[c]));
        m = fmaxf(m, 1e-30f);
        float *x = X + s * IN;
        for (int c = 0; c < NF; ++c) x[c] = v[c] / m;
        x[NF + 0] = (float)(accel * E[e * CN + i] / escale);
        x[NF + 1] = (float)(0.5 * (un[a * CN] + un[a * CN + CN - 1]) / umax);
        x[NF + 2] = (float)(0.5 * (vn[b * CN] + vn[b * CN + CN - 1]) / vmax);
        x[NF + 3] = (float)(accel * bfield);
        for (int c = NF + 4; c < IN; ++c) x[c] = 0.f;
        scale[s] = m;
    }
}

// out[e, i, a, j, b, k] += c2 dt cscale scale[s] clamp(Y[s][j CN + k], +-ymax)
template <typename T>
__global__ void closure_apply_kernel(T *__restrict__ out, int nx, int nu, int nv, const float *__restrict__ Y,
                                     const float *__restrict__ scale, double cscale, float ymax,
                                     const double *__restrict__ dt, double c2,
                                     const vl_run_state *__restrict__ state) {
    if (state != nullptr && state->active == 0) return;
    const int U = nu + 2, V = nv + 2;
    const long sJ = (long)V * CN, sA = sJ * CN, sI = sA * U, sE = sI * CN;
    const long total = (long)nx * CN * nu * nv * CN * CN;
    const double w = c2 * (*dt) * cscale;
    for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < total; p += (long)gridDim.x * blockDim.x) {
        long r = p;
        const int k = (int)(r % CN); r /= CN;
        const int j = (int)(r % CN); r /= CN;
        const long s = r;
        const int b = (int)(r % nv) + 1; r /= nv;
        const int a = (int)(r % nu) + 1; r /= nu;
        const int i = (int)(r % CN); r /= CN;
        const int e = (int)r + 1;
        const long o = e * sE + i * sI + a * sA + j * sJ + b * CN + k;
        const float y = fminf(fmaxf(Y[s * OUT + j * CN + k], -ymax), ymax);
        out[o] = (T)((double)out[o] + w * (double)scale[s] * (double)y);
    }
}

// Charge-conserving form: one CTA per x node (e, i) removes from the correction of that node the
// quadrature mean over all of its velocity nodes, so the correction leaves the zeroth moment -- the
// charge density the field is solved from -- unchanged:
//   c[s, j, k] = scale[s] clamp(Y[s][6 j + k]),  mean = sum w_j w_k c / sum w_j w_k,
//   out += c2 dt cscale (c - mean)
struct NodeWeights {
    double w[CN];
};

constexpr int CONS_THREADS = 256;

template <typename T>
__global__ void __launch_bounds__(CONS_THREADS)
closure_apply_conservative_kernel(T *__restrict__ out, int nx, int nu, int nv, const float *__restrict__ Y,
                                  const float *__restrict__ scale, double cscale, float ymax,
                                  const double *__restrict__ dt, double c2, const vl_run_state *__restrict__ state,
                                  const NodeWeights wq) {
    __shared__ double s_part[CONS_THREADS / 32];
    if (state != nullptr && state->active == 0) return;
    const int node = blockIdx.x;   // e CN + i, e 0-based
    const int e = node / CN + 1, i = node % CN;
    const int U = nu + 2, V = nv + 2;
    const long sJ = (long)V * CN, sA = sJ * CN, sI = sA * U, sE = sI * CN;
    const long nsamp = (long)nu * nv;
    const long s0 = (long)node * nsamp;
    const long count = nsamp * CN * CN;
    double acc = 0.0;
    for (long q = threadIdx.x; q < count; q += blockDim.x) {
        const long s = s0 + q / (CN * CN);
        const int jk = (int)(q % (CN * CN));
        const float y = fminf(fmaxf(Y[s * OUT + jk], -ymax), ymax);
        acc = fma(wq.w[jk / CN] * wq.w[jk % CN], (double)scale[s] * (double)y, acc);
    }
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = acc;
    __syncthreads();
    double tot = 0.0, wsum = 0.0;
    for (int w = 0; w < CONS_THREADS / 32; ++w) tot += s_part[w];
    for (int j = 0; j < CN; ++j)
        for (int k = 0; k < CN; ++k) wsum += wq.w[j] * wq.w[k];
    const double mean = tot / (wsum * (double)nsamp);
    const double w = c2 * (*dt) * cscale;
    for (long q = threadIdx.x; q < count; q += blockDim.x) {
        const long s = s0 + q / (CN * CN);
        const int jk = (int)(q % (CN * CN));
        const int j = jk / CN, k = jk % CN;
        const long sl = s - s0;
        const int a = (int)(sl / nv) + 1, b = (int)(sl % nv) + 1;
        const long o = e * sE + i * sI + a * sA + j * sJ + b * CN + k;
        const float y = fminf(fmaxf(Y[s * OUT + jk], -ymax), ymax);
        out[o] = (T)((double)out[o] + w * ((double)scale[s] * (double)y - mean));
    }
}

MlpWeights weights_of(const __nv_bfloat16 *wf, const __nv_bfloat16 *wb, const float *bias) {
    MlpWeights w;
    for (int l = 0; l < NL; ++l) {
        w.wf[l] = wf + w_off(l);
        w.wb[l] = wb + w_off(l);
        w.bias[l] = bias + b_off(l);
    }
    return w;
}

int fail(int code, const char *msg) {
    vl_internal_set_error(msg);
    return code;
}

int check(const char *where) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        vl_internal_set_error((std::string(where) + ": " + cudaGetErrorString(e)).c_str());
        return VL_ERR_CUDA;
    }
    return VL_OK;
}

// beta^step as the FP32 product of its factors, one after another.  A training loop asks for one step after
// the other, so a thread goes on from the product of its last call where beta is the same (a whole
// product per call takes 25 us at step 16000); the value does not depend on it.
float power(float beta, int step, int slot) {
    struct Last {
        float beta = 0.f, prod = 1.f;
        int step = 0;
    };
    static thread_local Last last[2];
    Last &l = last[slot];
    const int to = step < 100000 ? step : 100000;
    if (l.beta != beta || l.step > to) l = Last{beta, 1.f, 0};
    for (; l.step < to; ++l.step) l.prod *= beta;
    return l.prod;
}

// the kernels' shared-memory limits (per device, set once: an attribute of the function)
int dynamic_smem() {
    static std::mutex mu;
    static bool done[64] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (e == cudaSuccess && dev >= 0 && dev < 64 && done[dev]) return VL_OK;
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MLP_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_backprop_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MLP_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GRAD_SMEM);
    if (e != cudaSuccess) return fail(VL_ERR_CUDA, cudaGetErrorString(e));
    if (dev >= 0 && dev < 64) done[dev] = true;
    return VL_OK;
}

}  // namespace

extern "C" {

VL_API int vl_closure_features(const void *f, int32_t prec, int32_t nx, int32_t nu, int32_t nv,
                               const double *E, double accel, double bfield, const double *u_nodes,
                               const double *v_nodes, double umax, double vmax, double escale, float *X,
                               float *scale, void *stream) {
    if (!f || !E || !u_nodes || !v_nodes || !X || !scale) return fail(VL_ERR_INVALID, "null argument");
    if (nx < 1 || nu < 1 || nv < 1) return fail(VL_ERR_INVALID, "empty grid");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const long total = (long)nx * CN * nu * nv;
    const int blocks = (int)((total + 127) / 128 < 148 * 32 ? (total + 127) / 128 : 148 * 32);
    if (prec == VL_FP64)
        closure_features_kernel<double><<<blocks, 128, 0, s>>>(static_cast<const double *>(f), nx, nu, nv, E, accel,
                                                               bfield, u_nodes, v_nodes, umax, vmax, escale, X, scale);
    else
        closure_features_kernel<float><<<blocks, 128, 0, s>>>(static_cast<const float *>(f), nx, nu, nv, E, accel,
                                                              bfield, u_nodes, v_nodes, umax, vmax, escale, X, scale);
    return check("closure_features_kernel");
}

VL_API int vl_closure_apply(void *out, int32_t prec, int32_t nx, int32_t nu, int32_t nv, const float *Y,
                            const float *scale, double cscale, float ymax, const double *dt, double c2,
                            const vl_run_state *state, int32_t mode, const double *node_weights, void *stream) {
    if (!out || !Y || !scale || !dt) return fail(VL_ERR_INVALID, "null argument");
    if (mode != VL_CLOSURE_PLAIN && mode != VL_CLOSURE_CHARGE) return fail(VL_ERR_INVALID, "closure mode");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (mode == VL_CLOSURE_CHARGE) {
        if (!node_weights) return fail(VL_ERR_INVALID, "null node weights");
        NodeWeights wq;
        for (int j = 0; j < CN; ++j) wq.w[j] = node_weights[j];
        const int blocks = nx * CN;
        if (prec == VL_FP64)
            closure_apply_conservative_kernel<double><<<blocks, CONS_THREADS, 0, s>>>(
                static_cast<double *>(out), nx, nu, nv, Y, scale, cscale, ymax, dt, c2, state, wq);
        else
            closure_apply_conservative_kernel<float><<<blocks, CONS_THREADS, 0, s>>>(
                static_cast<float *>(out), nx, nu, nv, Y, scale, cscale, ymax, dt, c2, state, wq);
        return check("closure_apply_conservative_kernel");
    }
    const long total = (long)nx * CN * nu * nv * CN * CN;
    const int blocks = (int)((total + 255) / 256 < 148 * 32 ? (total + 255) / 256 : 148 * 32);
    if (prec == VL_FP64)
        closure_apply_kernel<double><<<blocks, 256, 0, s>>>(static_cast<double *>(out), nx, nu, nv, Y, scale,
                                                            cscale, ymax, dt, c2, state);
    else
        closure_apply_kernel<float><<<blocks, 256, 0, s>>>(static_cast<float *>(out), nx, nu, nv, Y, scale,
                                                           cscale, ymax, dt, c2, state);
    return check("closure_apply_kernel");
}

VL_API int vl_mlp_dims(int32_t *in, int32_t *hidden, int32_t *out, int32_t *n_weights, int32_t *n_bias) {
    if (in) *in = IN;
    if (hidden) *hidden = HID;
    if (out) *out = OUT;
    if (n_weights) *n_weights = GW_ELEMS;
    if (n_bias) *n_bias = GB_ELEMS;
    return VL_OK;
}

VL_API int vl_mlp_forward(const float *X, int32_t nrows, const void *wf, const void *wb, const float *bias,
                          float *Y, void *H0, void *Hh, float *Z, void *stream) {
    if (!X || !wf || !wb || !bias || !Y || nrows < 0) return fail(VL_ERR_INVALID, "null argument");
    if (nrows == 0) return VL_OK;
    const bool save = H0 || Hh || Z;
    if (save && !(H0 && Hh && Z)) return fail(VL_ERR_INVALID, "training forward needs H0, Hh and Z");
    int rc = dynamic_smem();
    if (rc) return rc;
    mlp_forward_kernel<<<(nrows + ROWS - 1) / ROWS, 32 * WARPS, MLP_SMEM, static_cast<cudaStream_t>(stream)>>>(
        X, nrows, weights_of(static_cast<const __nv_bfloat16 *>(wf), static_cast<const __nv_bfloat16 *>(wb), bias),
        Y, static_cast<__nv_bfloat16 *>(H0), static_cast<__nv_bfloat16 *>(Hh), Z);
    return check("mlp_forward_kernel");
}

VL_API size_t vl_mlp_partial_floats(int32_t nrows) {
    // dZ of every layer, bf16, rows up to a multiple of BLOCK
    const size_t rows = ((size_t)nrows + BLOCK - 1) / BLOCK * BLOCK;
    return rows * (3 * HID + OUT) / 2 + 4;   // (+ a 16-byte boundary at its start)
}

VL_API int vl_mlp_backward(const float *Y, const float *T, int32_t nrows, int32_t nout, const void *wf,
                           const void *wb, const float *bias, const void *H0, const void *Hh, const float *Z,
                           float *partials, float *grad_w, float *grad_b, void *stream) {
    if (!Y || !T || !wf || !wb || !bias || !H0 || !Hh || !Z || !partials || !grad_w || !grad_b)
        return fail(VL_ERR_INVALID, "null argument");
    if (nrows < 1 || nout < 1 || nout > OUT) return fail(VL_ERR_INVALID, "nrows >= 1, nout in 1..48");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int rows = (nrows + BLOCK - 1) / BLOCK * BLOCK;
    __nv_bfloat16 *dZ = reinterpret_cast<__nv_bfloat16 *>((reinterpret_cast<uintptr_t>(partials) + 15) & ~(uintptr_t)15);
    const bool h16 = ((reinterpret_cast<uintptr_t>(H0) | reinterpret_cast<uintptr_t>(Hh)) & 15) == 0;
    int rc = dynamic_smem();
    if (rc) return rc;
    mlp_backprop_kernel<<<rows / ROWS, 32 * WARPS, MLP_SMEM, s>>>(
        Y, T, nrows, nout,
        weights_of(static_cast<const __nv_bfloat16 *>(wf), static_cast<const __nv_bfloat16 *>(wb), bias), Z, dZ, rows);
    if ((rc = check("mlp_backprop_kernel"))) return rc;
    mlp_grad_kernel<<<GRAD_TILES + BIAS_CTAS, GRAD_THREADS, GRAD_SMEM, s>>>(static_cast<const __nv_bfloat16 *>(H0),
                                                                    static_cast<const __nv_bfloat16 *>(Hh), dZ, nrows,
                                                                    rows, h16, grad_w, grad_b);
    return check("mlp_grad_kernel");
}

VL_API int vl_mlp_adam(float *master_w, float *master_b, const float *grad_w, const float *grad_b, float *m_w,
                       float *v_w, float *m_b, float *v_b, void *wf, void *wb, float lr, float beta1,
                       float beta2, float eps, int32_t step, float weight_decay, void *stream) {
    if (!master_w || !master_b || !grad_w || !grad_b || !m_w || !v_w || !m_b || !v_b || !wf || !wb || step < 1)
        return fail(VL_ERR_INVALID, "null argument or step < 1");
    const float bc1 = 1.f - power(beta1, step, 0), bc2 = 1.f - power(beta2, step, 1);
    mlp_adam_kernel<<<148 * 2, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        master_w, master_b, grad_w, grad_b, m_w, v_w, m_b, v_b, static_cast<__nv_bfloat16 *>(wf),
        static_cast<__nv_bfloat16 *>(wb), lr, beta1, beta2, eps, bc1, bc2, weight_decay);
    return check("mlp_adam_kernel");
}

}  // extern "C"
