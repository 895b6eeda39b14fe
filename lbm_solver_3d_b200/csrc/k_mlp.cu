// ============================================================================
//  k_mlp.cu -- the swimmer surrogate network: a 4 -> 64 -> 64 -> 64 -> 3
//  multilayer perceptron with SiLU after each hidden layer, trained and
//  evaluated by the kernels below (no library GEMM, no autograd).
//
//  One CTA owns a tile of MLP_T = 32 samples and runs the whole network on it
//  from shared memory: forward through the four layers, the mean-squared loss,
//  and backward to the weight and bias gradients of the tile, which it writes
//  to its own row of a partials array. k_mlp_adam then sums the rows in a
//  fixed order (deterministic) and applies one Adam step to the FP32 master
//  parameters.
//
//  An Adam step on a minibatch of 512 keeps 16 CTAs busy and is a chain of
//  small products, so it is bound by latency and instruction issue: 16 warps
//  carry the chain, one 16 x 8 tile of every layer's output each, and 16 more
//  form the weight and bias gradients beside it; operand rows are padded so
//  that neither direct nor transposed reads collide in a bank; BF16 operands
//  are rounded once, when they are written, and read by ldmatrix;
//  pre-activations and sigmoids stay in the registers of the thread that needs
//  them again; and launches are programmatic, with a tile's samples fetched
//  while the Adam step before it runs and the optimizer's state while the
//  tiles run. An Adam step of 512 samples in BF16 takes 9.8 us, 31.5 us before
//  (8 warps, FP32 rows of 64 converted at every read, no overlap).
//
//  Every product is a warp-tiled GEMM on 16 x 8 output tiles:
//    BF16 = true   mma.sync m16n8k16 with BF16 operands (rounded from the FP32
//                  values) and FP32 accumulation;
//    BF16 = false  the same tiles with FP32 FMAs (k in ascending order).
//  The layer shapes are padded to multiples of the tile (inputs 4 -> 16,
//  outputs 3 -> 16) with zeros.
//
//  Parameter layout (FP32, the order of the C ABI): W1[64][4] b1[64]
//  W2[64][64] b2[64] W3[64][64] b3[64] W4[3][64] b4[3], W[out][in].
// ============================================================================
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/lbmgpu.h"
#include "pdl.cuh"

namespace {

using lbmgpu::order_acquire;
using lbmgpu::order_publish;
using lbmgpu::pdl_launch_dependents;
using lbmgpu::pdl_wait;

constexpr int NI = LBMGPU_MLP_IN, NH = LBMGPU_MLP_HIDDEN, NO = LBMGPU_MLP_OUT;
constexpr int NP = LBMGPU_MLP_NPARAMS;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + NH * NI, OFF_W2 = OFF_B1 + NH, OFF_B2 = OFF_W2 + NH * NH,
              OFF_W3 = OFF_B2 + NH, OFF_B3 = OFF_W3 + NH * NH, OFF_W4 = OFF_B3 + NH, OFF_B4 = OFF_W4 + NO * NH;
static_assert(OFF_B4 + NO == NP, "parameter layout");
constexpr int NPS = (NP + 31) / 32 * 32;   // row stride of the gradient partials

constexpr int MLP_T = 32;        // samples per CTA
constexpr int MLP_THREADS = 512; // 16 warps: the 16 x 8 tiles of a 32 x 64 layer output
constexpr int PI_ = 16;          // padded input width
constexpr int PO = 16;           // padded output width
constexpr int LOSS_THREADS = 256;   // threads that sum the loss, two outputs each
constexpr int SY = PO + 4;       // row stride of the outputs (FP32)
constexpr int SD = NH + 4;       // row stride of the FP32 dL/dz

// Operand types and row strides of the products: 64-wide (SH) and 16-wide (SI)
// rows, padded so that 8 consecutive rows start in different banks.
template <bool BF16> struct Ops;
template <> struct Ops<true> { using T = __nv_bfloat16; static constexpr int SH = NH + 8, SI = PI_ + 8; };
template <> struct Ops<false> { using T = float; static constexpr int SH = NH + 4, SI = PI_ + 4; };

template <bool BF16>
struct Smem {
    using T = typename Ops<BF16>::T;
    static constexpr int SH = Ops<BF16>::SH, SI = Ops<BF16>::SI;
    alignas(16) T W1[NH * SI], W2[NH * SH], W3[NH * SH], W4[PO * SH];
    alignas(16) T H0[MLP_T * SI], H1[MLP_T * SH], H2[MLP_T * SH], H3[MLP_T * SH];
    alignas(16) T dY[MLP_T * SI], d3[MLP_T * SH], d2[MLP_T * SH], d1[MLP_T * SH];   // dL/dz of each layer
    alignas(16) float Y[MLP_T * SY], fY[MLP_T * SY];                                // outputs, dL/dY
    float f3[MLP_T * SD], f2[MLP_T * SD], f1[MLP_T * SD];                           // dL/dz (bias gradients)
    float b1[NH], b2[NH], b3[NH], b4[PO];
    float red[LOSS_THREADS / 32];
};

// 1 / x for x >= 1, as the division rounds it: the hardware's approximation and
// one Newton step whose residual is exact in an FMA (as Markstein 1990 corrects
// quotients). The approximation's error has no bound from which equality would
// follow; the test compares every float in [1, 2^100). Beyond that, and for
// infinities and NaN, the division itself.
__device__ __forceinline__ float recip_ge1(float x) {
    if (!(x < 1.2676506e30f)) return 1.0f / x;
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return __fmaf_rn(__fmaf_rn(-x, y, 1.0f), y, y);
}
__device__ __forceinline__ float sigmoid(float z) { return recip_ge1(1.0f + expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigmoid(z); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);   // .x (low half) = lo
    uint32_t u;
    memcpy(&u, &v, 4);
    return u;
}

template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __nv_bfloat16* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    if constexpr (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

// The 16 x 8 tile (m0, n0) of C(m, n) = sum_k A(m, k) B(k, n), K a multiple of
// 16, A(m, k) = A[m*AS0 + k*AS1], B(k, n) = B[k*BS0 + n*BS1] (one of each pair of
// strides is 1). A lane holds c[0..3] = C at (m0 + g, n0 + 2t), (.., +1),
// (m0 + g + 8, ..), (.., +1) with g = lane / 4, t = lane % 4.
// BF16: an ldmatrix brings the four 8 x 8 blocks of A's 16 x 16, another B's
// four 8-row blocks of 32 k (16 k: the same two blocks twice); the operand
// whose unit stride runs the other way is transposed on the way.
template <int K, int AS0, int AS1, int BS0, int BS1>
__device__ __forceinline__ void gemm_tile(const __nv_bfloat16* A, const __nv_bfloat16* B, int m0, int n0, float (&c)[4]) {
    const int lane = threadIdx.x & 31, mi = lane >> 3, r = lane & 7;
    c[0] = c[1] = c[2] = c[3] = 0.f;
    const __nv_bfloat16* pa = AS1 == 1 ? A + (m0 + r + (mi & 1) * 8) * AS0 + (mi >> 1) * 8
                                       : A + ((mi >> 1) * 8 + r) * AS1 + m0 + (mi & 1) * 8;
    const int kb = K >= 32 ? mi * 8 : (mi & 1) * 8;
    const __nv_bfloat16* pb = BS0 == 1 ? B + (n0 + r) * BS1 + kb : B + (kb + r) * BS0 + n0;
    uint32_t b[4];
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += 16) {
        uint32_t a[4];
        ldmatrix4<AS1 != 1>(a, pa + k0 * AS1);
        if (k0 % 32 == 0) ldmatrix4<BS0 != 1>(b, pb + k0 * BS0);
        const int h = (k0 % 32) / 8;
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
            "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[h]), "r"(b[h + 1]));
    }
}
template <int K, int AS0, int AS1, int BS0, int BS1>
__device__ __forceinline__ void gemm_tile(const float* A, const float* B, int m0, int n0, float (&c)[4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    c[0] = c[1] = c[2] = c[3] = 0.f;
    const float *p0 = A + (m0 + g) * AS0, *p1 = p0 + 8 * AS0, *q0 = B + (n0 + 2 * tq) * BS1, *q1 = q0 + BS1;
#pragma unroll 8
    for (int k = 0; k < K; ++k) {
        const float x0 = p0[k * AS1], x1 = p1[k * AS1], y0 = q0[k * BS0], y1 = q1[k * BS0];
        c[0] = fmaf(x0, y0, c[0]); c[1] = fmaf(x0, y1, c[1]);
        c[2] = fmaf(x1, y0, c[2]); c[3] = fmaf(x1, y1, c[3]);
    }
}
// two neighbouring operands
__device__ __forceinline__ void put2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void put2(__nv_bfloat16* p, float a, float b) { *reinterpret_cast<uint32_t*>(p) = pack_bf16(a, b); }
__device__ __forceinline__ void put1(float* p, float a) { *p = a; }
__device__ __forceinline__ void put1(__nv_bfloat16* p, float a) { *p = __float2bfloat16_rn(a); }

// A 64-wide weight matrix of `rows` rows (rows >= valid are zero) into its padded place.
template <int SH, class T>
__device__ __forceinline__ void load_w64(T* dst, const float* w, int rows, int valid) {
    for (int e = threadIdx.x; e < rows * (NH / 4); e += blockDim.x) {
        const int r = e / (NH / 4), c = 4 * (e % (NH / 4));
        const float4 v = r < valid ? __ldcg(reinterpret_cast<const float4*>(w + r * NH + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
        put2(dst + r * SH + c, v.x, v.y);
        put2(dst + r * SH + c + 2, v.z, v.w);
    }
}

// Forward (and, when TRAIN, backward) of tiles of MLP_T samples.
//   X [n][4], Yt [n][3] (targets, TRAIN), idx: sample order (NULL: identity);
//   TRAIN: one tile per CTA of 2 MLP_THREADS; grad_part[blockIdx.x][NPS] and
//          loss_part[blockIdx.x] = sum of squared errors of the tile;
//          dL/dY = 2 (Y - Yt) * inv_count; order, tag: published for k_mlp_adam;
//   else:  Yout [n][3]; a CTA of MLP_THREADS takes tiles blockIdx.x, + gridDim.x,
//          ... with the parameters loaded once.
template <bool BF16, bool TRAIN>
__global__ void __launch_bounds__(TRAIN ? 2 * MLP_THREADS : MLP_THREADS)
    k_mlp_tile(const float* params, const float* __restrict__ X, const float* __restrict__ Yt,
               const int* __restrict__ idx, int base, int n, float inv_count, float* __restrict__ grad_part,
               float* __restrict__ loss_part, float* __restrict__ Yout, int* order, int tag) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Sm = Smem<BF16>;
    constexpr int SH = Sm::SH, SI = Sm::SI;
    Sm& S = *reinterpret_cast<Sm*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
    // TRAIN: the second 16 warps form the gradients beside the chain of the first
    const bool chain = !TRAIN || warp < MLP_THREADS / 32;
    const int cw = warp & 15;
    // a chain warp's tile of a layer's 32 x 64 output, and this lane's rows and columns in it
    const int m0 = (cw >> 3) * 16, n0 = (cw & 7) * 8, ra = m0 + g, rb = ra + 8, cc = n0 + 2 * tq;

    for (int tile = blockIdx.x;; tile += gridDim.x) {
    const int t0 = base + tile * MLP_T;   // first sample slot of this tile
    if (!TRAIN && t0 >= n) break;
    // inputs, padded; before the wait: they were copied before the first of the
    // call's kernels was launched and are static since (read past the L1, which
    // may hold an earlier call's)
    float yt = 0.f, yt2 = 0.f;            // TRAIN: this thread's targets
    if (tid < MLP_T * PI_) {
        const int s = tid / PI_, k = tid % PI_, slot = t0 + s;
        float v = 0.f;
        if (k < NI && slot < n) v = __ldcg(X + (size_t)(idx ? __ldcg(idx + slot) : slot) * NI + k);
        put1(S.H0 + s * SI + k, v);
        if (TRAIN && tid < LOSS_THREADS) {
            const int s2 = (tid + LOSS_THREADS) / PO, o = tid % PO;
            if (o < NO && t0 + s < n) yt = __ldcg(Yt + (size_t)(idx ? __ldcg(idx + t0 + s) : t0 + s) * NO + o);
            if (o < NO && t0 + s2 < n) yt2 = __ldcg(Yt + (size_t)(idx ? __ldcg(idx + t0 + s2) : t0 + s2) * NO + o);
        }
    }
    if (TRAIN || tile == (int)blockIdx.x) {
        if (TRAIN) {
            pdl_wait();
            if (blockIdx.x == 0 && tid == 0) order_publish(order, tag);
            pdl_launch_dependents();
        }
        // parameters, padded
        load_w64<SH>(S.W2, params + OFF_W2, NH, NH);
        load_w64<SH>(S.W3, params + OFF_W3, NH, NH);
        load_w64<SH>(S.W4, params + OFF_W4, PO, NO);
        for (int e = tid; e < NH * PI_; e += blockDim.x) {
            const int j = e / PI_, k = e % PI_;
            put1(S.W1 + j * SI + k, k < NI ? __ldcg(params + OFF_W1 + j * NI + k) : 0.f);
        }
        if (tid < NH) S.b1[tid] = __ldcg(params + OFF_B1 + tid);
        else if (tid < 2 * NH) S.b2[tid - NH] = __ldcg(params + OFF_B2 + tid - NH);
        else if (tid < 3 * NH) S.b3[tid - 2 * NH] = __ldcg(params + OFF_B3 + tid - 2 * NH);
        else if (tid < 3 * NH + PO) S.b4[tid - 3 * NH] = tid - 3 * NH < NO ? __ldcg(params + OFF_B4 + tid - 3 * NH) : 0.f;
    }
    __syncthreads();

    // ---- forward: each lane keeps its pre-activations z and sigmoids s ----
    float c[4], z1[4], z2[4], z3[4], s1[4], s2[4], s3[4];
    auto act = [&](const float* b, float (&z)[4], float (&sg)[4], typename Sm::T* H) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            z[e] = c[e] + b[cc + (e & 1)];
            sg[e] = sigmoid(z[e]);
        }
        put2(H + ra * SH + cc, z[0] * sg[0], z[1] * sg[1]);
        put2(H + rb * SH + cc, z[2] * sg[2], z[3] * sg[3]);
    };
    if (chain) {
        gemm_tile<PI_, SI, 1, 1, SI>(S.H0, S.W1, m0, n0, c);
        act(S.b1, z1, s1, S.H1);
    }
    __syncthreads();
    if (chain) {
        gemm_tile<NH, SH, 1, 1, SH>(S.H1, S.W2, m0, n0, c);
        act(S.b2, z2, s2, S.H2);
    }
    __syncthreads();
    if (chain) {
        gemm_tile<NH, SH, 1, 1, SH>(S.H2, S.W3, m0, n0, c);
        act(S.b3, z3, s3, S.H3);
    }
    __syncthreads();
    if (warp < (MLP_T / 16) * (PO / 8)) {
        const int m = (warp >> 1) * 16, q = (warp & 1) * 8, o = q + 2 * tq;
        gemm_tile<NH, SH, 1, 1, SH>(S.H3, S.W4, m, q, c);
        put2(S.Y + (m + g) * SY + o, c[0] + S.b4[o], c[1] + S.b4[o + 1]);
        put2(S.Y + (m + g + 8) * SY + o, c[2] + S.b4[o], c[3] + S.b4[o + 1]);
    }
    __syncthreads();

    if constexpr (!TRAIN) {
        if (tid < MLP_T * NO) {
            const int s = tid / NO, o = tid % NO;
            if (t0 + s < n) Yout[(size_t)(t0 + s) * NO + o] = S.Y[s * SY + o];
        }
        continue;   // the next tile's first writes go to H0, last read before the barriers above
    } else {
        // ---- loss and dL/dY ----
        if (tid < LOSS_THREADS) {
            float se = 0.f;
            const int o = tid % PO;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int s = (tid + h * LOSS_THREADS) / PO;
                float d = 0.f;
                if (o < NO && t0 + s < n) {
                    const float r = S.Y[s * SY + o] - (h ? yt2 : yt);
                    se += r * r;
                    d = 2.f * r * inv_count;
                }
                S.fY[s * SY + o] = d;
                put1(S.dY + s * SI + o, d);
            }
            for (int o2 = 16; o2 > 0; o2 >>= 1) se += __shfl_down_sync(0xffffffffu, se, o2);
            if (lane == 0) S.red[warp] = se;
        }
        __syncthreads();
        float* gp = grad_part + (size_t)blockIdx.x * NPS;
        // a bias gradient: the tile's samples in order
        auto bias = [&](const float* d, int stride, int j) {
            float v[MLP_T], b = 0.f;
#pragma unroll
            for (int q = 0; q < MLP_T; ++q) v[q] = d[q * stride + j];
#pragma unroll
            for (int q = 0; q < MLP_T; ++q) b += v[q];
            return b;
        };
        // dL/dz of a hidden layer from dL/dh in c
        auto back = [&](const float (&z)[4], const float (&sg)[4], typename Sm::T* D, float* F) {
            float d[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) d[e] = c[e] * (sg[e] * (1.0f + z[e] * (1.0f - sg[e])));
            put2(D + ra * SH + cc, d[0], d[1]);
            put2(D + rb * SH + cc, d[2], d[3]);
            put2(F + ra * SD + cc, d[0], d[1]);
            put2(F + rb * SD + cc, d[2], d[3]);
        };
        // a hidden layer's weight gradient (4 x 8 tiles over 16 warps) and bias gradient
        auto grads = [&](const typename Sm::T* D, const typename Sm::T* H, const float* F, int off_w, int off_b) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = m0 + 32 * h;
                float w[4];
                gemm_tile<MLP_T, 1, SH, SH, 1>(D, H, m, n0, w);
                put2(gp + off_w + (m + g) * NH + cc, w[0], w[1]);
                put2(gp + off_w + (m + g + 8) * NH + cc, w[2], w[3]);
            }
            if (cw < NH / 32) gp[off_b + cw * 32 + lane] = bias(F, SD, cw * 32 + lane);
        };
        if (chain) {
            gemm_tile<PO, SI, 1, SH, 1>(S.dY, S.W4, m0, n0, c);
            back(z3, s3, S.d3, S.f3);
        } else {
            if (cw < NH / 8) {   // layer 4
                float w[4];
                gemm_tile<MLP_T, 1, SI, SH, 1>(S.dY, S.H3, 0, cw * 8, w);
                if (g < NO) put2(gp + OFF_W4 + g * NH + cw * 8 + 2 * tq, w[0], w[1]);
            } else if (cw == 8) {
                if (lane < NO) gp[OFF_B4 + lane] = bias(S.fY, SY, lane);
            } else if (cw == 9 && lane == 0) {
                float tot = 0.f;
                for (int w = 0; w < LOSS_THREADS / 32; ++w) tot += S.red[w];
                loss_part[blockIdx.x] = tot;
            }
        }
        __syncthreads();
        if (chain) {
            gemm_tile<NH, SH, 1, SH, 1>(S.d3, S.W3, m0, n0, c);
            back(z2, s2, S.d2, S.f2);
        } else {
            grads(S.d3, S.H2, S.f3, OFF_W3, OFF_B3);
        }
        __syncthreads();
        if (chain) {
            gemm_tile<NH, SH, 1, SH, 1>(S.d2, S.W2, m0, n0, c);
            back(z1, s1, S.d1, S.f1);
        } else {
            grads(S.d2, S.H1, S.f2, OFF_W2, OFF_B2);
        }
        __syncthreads();
        if (warp < NH / 16) {   // layer 1
            float w[4];
            gemm_tile<MLP_T, 1, SH, SI, 1>(S.d1, S.H0, warp * 16, 0, w);
            if (2 * tq < NI) {
                put2(gp + OFF_W1 + (warp * 16 + g) * NI + 2 * tq, w[0], w[1]);
                put2(gp + OFF_W1 + (warp * 16 + g + 8) * NI + 2 * tq, w[2], w[3]);
            }
        } else if (warp >= 8 && warp < 8 + NH / 32) {
            gp[OFF_B1 + (warp - 8) * 32 + lane] = bias(S.f1, SD, (warp - 8) * 32 + lane);
        }
        return;
    }
    }
}

// Sum of the tile partials (tile order) and one Adam step. With lr = 0 only
// the gradient (and loss) is produced. The optimizer's state was last written
// by the Adam step before the tiles, which waited for it and published tag: it
// is fetched before this kernel's own wait. The last CTA sums the loss.
constexpr int ADAM_THREADS = 128, ADAM_GRID = (NP + ADAM_THREADS - 1) / ADAM_THREADS;
__global__ void __launch_bounds__(ADAM_THREADS) k_mlp_adam(float* __restrict__ params, float* __restrict__ m1,
                                                           float* __restrict__ m2, const float* grad_part, int nparts,
                                                           const float* loss_part, float inv_count, float lr,
                                                           float beta1, float beta2, float eps, float bc1, float bc2,
                                                           float* __restrict__ grad_out, float* __restrict__ loss_out,
                                                           const int* order, int tag) {
    const int p = blockIdx.x * ADAM_THREADS + threadIdx.x;
    float w = 0.f, a = 0.f, b = 0.f;
    if (p < NP && lr != 0.f) {
        order_acquire(order, tag);
        w = __ldcg(params + p); a = __ldcg(m1 + p); b = __ldcg(m2 + p);
    }
    pdl_wait();
    pdl_launch_dependents();
    if (blockIdx.x == ADAM_GRID) {
        if (threadIdx.x == 0 && loss_out) {
            float l = 0.f;
#pragma unroll 16
            for (int c = 0; c < nparts; ++c) l += __ldcg(loss_part + c);
            *loss_out = l * inv_count;
        }
        return;
    }
    if (p >= NP) return;
    float g = 0.f;
#pragma unroll 16
    for (int c = 0; c < nparts; ++c) g += __ldcg(grad_part + (size_t)c * NPS + p);
    if (grad_out) grad_out[p] = g;
    if (lr == 0.f) return;
    a = __fmaf_rn(1.f - beta1, g, __fmul_rn(beta1, a));
    b = __fmaf_rn(__fmul_rn(1.f - beta2, g), g, __fmul_rn(beta2, b));
    m1[p] = a; m2[p] = b;
    params[p] = w - lr * (a / bc1) / (sqrtf(b / bc2) + eps);
}

// ---------------------------------------------------------------------------
//  k_mlp_fwd_tc: BF16 inference on the fifth-generation tensor cores.
//
//  One CTA of 128 threads owns 128 samples: thread i is sample i, and row i
//  of every product. Each layer is D[128 x N] = A[128 x K] . W^T with A (the
//  activations) and W (the weights, [out][in]) in shared memory as BF16 and D
//  in tensor memory (FP32, 64 columns allocated per CTA):
//    thread 0 issues tcgen05.mma (kind::f16, cta_group::1, M = 128,
//    N = 64 or 16, K = 16 per instruction) and tcgen05.commit to an mbarrier;
//    every warp then reads its 32 rows of D with tcgen05.ld (32x32b), adds the
//    bias, applies SiLU and writes the next layer's A in BF16.
//  Operand layout in shared memory: K-major with no swizzle. The 8 x 8 BF16
//  core matrices are 128 contiguous bytes (8 rows of 16 bytes). Row r, column k
//  of an R-row operand is at byte ((k / 8) * R + r) * 16 + (k % 8) * 2, so the
//  stride between 8-row groups (SBO) is 128 bytes and the stride between the
//  two 8-column halves of a K = 16 step (LBO) is R * 16 bytes.
//  The grid is one wave of CTAs: each loads and rounds the weights once, holds
//  its tensor memory, and takes tiles of 128 samples in turn. (With a CTA per
//  tile the weights' 35 KB and their index arithmetic were most of the time:
//  98 us for 250,001 samples, 76 us now; 46 -> 24 us for one tile. A call is
//  mostly its copies from and to pageable memory: 550 us for 250,001 samples.)
//  Waits on the mbarrier are bounded; a timeout sets *err, and the tensor
//  memory is released on every path.
// ---------------------------------------------------------------------------
constexpr int TC_M = 128;              // samples per CTA
constexpr int TC_COLS = 64;            // tensor-memory columns (FP32 accumulators)
constexpr int TC_CTAS = 5;             // CTAs per SM: shared memory holds 5 x 38 KB, tensor memory 8 x 64 columns

struct TcSmem {
    alignas(128) __nv_bfloat16 A[NH / 8][TC_M][8];       // activations, K-major core matrices
    alignas(128) __nv_bfloat16 W1[PI_ / 8][NH][8];
    alignas(128) __nv_bfloat16 W2[NH / 8][NH][8];
    alignas(128) __nv_bfloat16 W3[NH / 8][NH][8];
    alignas(128) __nv_bfloat16 W4[NH / 8][PO][8];
    float b1[NH], b2[NH], b3[NH], b4[PO];
    alignas(8) uint64_t mbar;
    uint32_t tmem_base;
};

__device__ __forceinline__ uint64_t umma_desc(const void* smem, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    uint64_t d = 0;
    d |= (uint64_t)((a >> 4) & 0x3FFFu);                     // start address
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;       // leading dimension byte offset
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;       // stride dimension byte offset
    d |= (uint64_t)1 << 46;                                  // descriptor version (sm_100)
    return d;                                                // base offset 0, no swizzle
}

// BF16 x BF16 -> FP32, both operands K-major, M = 128
__host__ __device__ constexpr uint32_t umma_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
}

__device__ __forceinline__ bool tc_wait(uint64_t* m, uint32_t parity) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(m);
    for (int it = 0; it < (1 << 22); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok) : "r"(a), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

// D[tmem] = A . W^T over K (multiple of 16), issued by one thread, completion on mbar
__device__ __forceinline__ void tc_layer(uint32_t tmem, const void* A, const void* W, int K, int N, uint64_t* mbar) {
    const uint32_t idesc = umma_idesc(N);
    for (int k16 = 0; k16 < K / 16; ++k16) {
        const uint64_t da = umma_desc((const char*)A + (size_t)k16 * 2 * TC_M * 16, TC_M * 16, 128);
        const uint64_t db = umma_desc((const char*)W + (size_t)k16 * 2 * N * 16, N * 16, 128);
        const uint32_t acc = k16 > 0;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n}"
            :: "r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0)
            : "memory");
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"((uint32_t)__cvta_generic_to_shared(mbar)) : "memory");
}

// 16 FP32 columns of this thread's row of D
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

// W[out][in] (FP32, global) -> BF16 K-major core matrices with R rows (outputs,
// VALID of them given, the others zero) and KP columns (inputs, KIN of them
// given, a multiple of 4): four inputs per load, all of a thread's in flight.
template <int R, int VALID, int KP, int KIN>
__device__ __forceinline__ void tc_load_w(__nv_bfloat16* dst, const float* __restrict__ w) {
#pragma unroll
    for (int e0 = 0; e0 < R * KP / 4; e0 += TC_M) {
        const int e = e0 + threadIdx.x, r = e / (KP / 4), k = 4 * (e % (KP / 4));
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < VALID && k < KIN) v = *reinterpret_cast<const float4*>(w + r * KIN + k);
        *reinterpret_cast<uint2*>(dst + ((size_t)(k / 8) * R + r) * 8 + (k % 8)) =
            make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
    }
}
static_assert(NH * PI_ / 4 % TC_M == 0 && PO * NH / 4 % TC_M == 0, "whole rounds");

__global__ void __launch_bounds__(TC_M) k_mlp_fwd_tc(const float* __restrict__ params, const float* __restrict__ X,
                                                     int n, float* __restrict__ Yout, int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char tc_raw[];
    TcSmem& S = *reinterpret_cast<TcSmem*>(tc_raw);
    const int tid = threadIdx.x, warp = tid >> 5;

    if (warp == 0) {   // tensor memory: one warp allocates, the same warp frees
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"((uint32_t)__cvta_generic_to_shared(&S.tmem_base)), "r"(TC_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"((uint32_t)__cvta_generic_to_shared(&S.mbar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_load_w<NH, NH, PI_, NI>(&S.W1[0][0][0], params + OFF_W1);
    tc_load_w<NH, NH, NH, NH>(&S.W2[0][0][0], params + OFF_W2);
    tc_load_w<NH, NH, NH, NH>(&S.W3[0][0][0], params + OFF_W3);
    tc_load_w<PO, NO, NH, NH>(&S.W4[0][0][0], params + OFF_W4);
    for (int e = tid; e < NH; e += TC_M) { S.b1[e] = params[OFF_B1 + e]; S.b2[e] = params[OFF_B2 + e]; S.b3[e] = params[OFF_B3 + e]; }
    if (tid < PO) S.b4[tid] = tid < NO ? params[OFF_B4 + tid] : 0.f;
    float4 xin = make_float4(0.f, 0.f, 0.f, 0.f);   // the next tile's input row of this thread
    const int ntiles = (n + TC_M - 1) / TC_M;
    if ((int)blockIdx.x * TC_M + tid < n) xin = reinterpret_cast<const float4*>(X)[(size_t)blockIdx.x * TC_M + tid];
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();   // tmem_base, the barrier
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = S.tmem_base;
    const uint32_t my_lanes = tmem + ((uint32_t)(warp * 32) << 16);

    bool ok = true;
    uint32_t phase = 0, last = 0;   // last: the phase of the most recent commit
    const void* Ws[3] = {&S.W1[0][0][0], &S.W2[0][0][0], &S.W3[0][0][0]};
    const float* bs[3] = {S.b1, S.b2, S.b3};
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const int row = tile * TC_M + tid;
        {   // this thread's input row, padded to 16
            static_assert(NI == 4 && PI_ == 16, "one float4 of inputs, a zero second half");
            uint4 v = make_uint4(pack_bf16(xin.x, xin.y), pack_bf16(xin.z, xin.w), 0u, 0u);
            *reinterpret_cast<uint4*>(&S.A[0][tid][0]) = v;
            *reinterpret_cast<uint4*>(&S.A[1][tid][0]) = make_uint4(0u, 0u, 0u, 0u);
            const int nrow = row + (int)gridDim.x * TC_M;   // fetched while this tile is computed
            xin = nrow < n && nrow > row ? reinterpret_cast<const float4*>(X)[nrow] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // operands visible to the tensor cores
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int l = 0; l < 3 && ok; ++l) {
            if (tid == 0) tc_layer(tmem, &S.A[0][0][0], Ws[l], l == 0 ? PI_ : NH, NH, &S.mbar);
            last = phase;
            ok = __all_sync(0xffffffffu, tc_wait(&S.mbar, phase));   // warp-uniform: tcgen05.ld is .sync.aligned
            phase ^= 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (ok) {
                // 16 columns at a time, in a loop: all 64 SiLUs unrolled are
                // 25 KB of instructions, which every layer fetched anew (12 us)
#pragma unroll 1
                for (int q = 0; q < NH / 16; ++q) {
                    float h[16];
                    tc_ld16(my_lanes + q * 16, h);
                    const float* b = bs[l] + q * 16;
                    uint32_t w[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        w[j] = pack_bf16(silu(h[2 * j] + b[2 * j]), silu(h[2 * j + 1] + b[2 * j + 1]));
                    *reinterpret_cast<uint4*>(&S.A[2 * q][tid][0]) = make_uint4(w[0], w[1], w[2], w[3]);
                    *reinterpret_cast<uint4*>(&S.A[2 * q + 1][tid][0]) = make_uint4(w[4], w[5], w[6], w[7]);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            ok = __syncthreads_and(ok);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        if (ok) {
            if (tid == 0) tc_layer(tmem, &S.A[0][0][0], &S.W4[0][0][0], NH, PO, &S.mbar);
            last = phase;
            ok = __all_sync(0xffffffffu, tc_wait(&S.mbar, phase));
            phase ^= 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (ok) {
                float y[16];
                tc_ld16(my_lanes, y);
                if (row < n)
#pragma unroll
                    for (int o = 0; o < NO; ++o) Yout[(size_t)row * NO + o] = y[o] + S.b4[o];
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            ok = __syncthreads_and(ok);   // the tile's columns and operands may be reused; one verdict for all
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
    }
    ok = __syncthreads_and(ok);   // the same verdict in every warp
    if (!ok) {
        // A wait gave up while the last layer's MMAs may still be writing
        // tensor memory: wait (bounded) for their commit before the columns
        // are freed.
        if (tid == 0) {
            atomicExch(err, 1);
            tc_wait(&S.mbar, last);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(TC_COLS));
}

template <bool BF16, bool TRAIN>
cudaError_t prepare_tile() {
    return cudaFuncSetAttribute(k_mlp_tile<BF16, TRAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem<BF16>));
}

thread_local std::string g_mlp_error;

}  // namespace

struct lbmgpu_mlp {
    int device = 0, bf16 = 0, sms = 148;
    cudaStream_t stream = nullptr;
    float *params = nullptr, *m1 = nullptr, *m2 = nullptr;
    float *X = nullptr, *Y = nullptr;   // training set
    int n = 0, cap = 0;
    int* idx = nullptr;
    int idx_cap = 0;
    float* grad_part = nullptr;
    float* loss_part = nullptr;
    float* losses = nullptr;            // an epoch's minibatch losses
    int losses_cap = 0;
    int part_cap = 0;                   // tiles
    float *xin = nullptr, *yout = nullptr;
    int xin_cap = 0, yout_cap = 0;      // floats
    float* small = nullptr;             // [0] loss, [1..NP] gradient
    int* d_err = nullptr;               // tensor-core forward: a bounded wait gave up; then the order word (pdl.cuh)
    unsigned batches = 0;               // minibatches launched: the order word's value
    long long t = 0;                    // Adam steps taken
    float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    std::string err;
};

namespace {

int mfail(lbmgpu_mlp* m, int code, const std::string& msg) {
    if (m) m->err = msg; else g_mlp_error = msg;
    return code;
}

#define MTRY(m, call)                                                                               \
    do {                                                                                            \
        cudaError_t e_ = (call);                                                                    \
        if (e_ != cudaSuccess)                                                                      \
            return mfail(m, e_ == cudaErrorMemoryAllocation ? LBMGPU_ERR_NOMEM : LBMGPU_ERR_CUDA,     \
                         std::string(#call) + ": " + cudaGetErrorString(e_));                       \
    } while (0)

cudaError_t grow(float** p, int* cap, long long need_elems) {
    if (need_elems <= *cap) return cudaSuccess;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    cudaError_t e = cudaMalloc(p, (size_t)need_elems * sizeof(float));
    if (e == cudaSuccess) *cap = (int)need_elems;
    return e;
}

int ensure_parts(lbmgpu_mlp* m, int tiles) {
    if (tiles <= m->part_cap) return LBMGPU_OK;
    if (m->grad_part) cudaFree(m->grad_part);
    if (m->loss_part) cudaFree(m->loss_part);
    m->grad_part = m->loss_part = nullptr;
    m->part_cap = 0;
    MTRY(m, cudaMalloc(&m->grad_part, (size_t)tiles * NPS * sizeof(float)));
    MTRY(m, cudaMalloc(&m->loss_part, (size_t)tiles * sizeof(float)));
    m->part_cap = tiles;
    return LBMGPU_OK;
}

// Launch that may start while its predecessor in the stream finishes (pdl_wait).
template <class... KArgs, class... Args>
cudaError_t launch_pdl(void (*kern)(KArgs...), int grid, int block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// fwd + bwd over samples [0, count) of the order `idx` (or identity), then
// the reduction (and Adam step when lr > 0)
int train_batch(lbmgpu_mlp* m, const int* idx, int base, int count, float lr, float* d_grad, float* d_loss) {
    const int tiles = (count + MLP_T - 1) / MLP_T;
    int rc = ensure_parts(m, tiles);
    if (rc) return rc;
    const float inv = 1.0f / (float)(count * NO);
    const int tag = (int)++m->batches;   // another value than the minibatch before left
    // the tile kernel sees slots [base, base + count) of idx as its samples
    MTRY(m, launch_pdl(m->bf16 ? k_mlp_tile<true, true> : k_mlp_tile<false, true>, tiles, 2 * MLP_THREADS,
                       m->bf16 ? sizeof(Smem<true>) : sizeof(Smem<false>), m->stream, (const float*)m->params, (const float*)m->X, (const float*)m->Y, idx, base,
                       base + count, inv, m->grad_part, m->loss_part, (float*)nullptr, m->d_err + 1, tag));
    float bc1 = 1.f, bc2 = 1.f;
    if (lr > 0.f) {
        m->t += 1;
        bc1 = 1.f - powf(m->beta1, (float)m->t);
        bc2 = 1.f - powf(m->beta2, (float)m->t);
    }
    MTRY(m, launch_pdl(k_mlp_adam, ADAM_GRID + 1, ADAM_THREADS, 0, m->stream, m->params, m->m1, m->m2,
                       (const float*)m->grad_part, tiles, (const float*)m->loss_part, inv, lr, m->beta1, m->beta2,
                       m->eps, bc1, bc2, d_grad, d_loss, (const int*)(m->d_err + 1), tag));
    return LBMGPU_OK;
}

}  // namespace

extern "C" {

int lbmgpu_mlp_create(int device, int bf16, lbmgpu_mlp** out) {
    if (!out) return mfail(nullptr, LBMGPU_ERR_INVALID, "null output pointer");
    *out = nullptr;
    lbmgpu_mlp* m = new lbmgpu_mlp();
    m->device = device;
    m->bf16 = bf16 ? 1 : 0;
    auto bail = [&](cudaError_t e, const char* what) {
        g_mlp_error = std::string(what) + ": " + cudaGetErrorString(e);
        lbmgpu_mlp_destroy(m);
        return e == cudaErrorMemoryAllocation ? LBMGPU_ERR_NOMEM : LBMGPU_ERR_CUDA;
    };
    cudaError_t e;
    if ((e = cudaSetDevice(device)) != cudaSuccess) return bail(e, "cudaSetDevice");
    if ((e = cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess)
        return bail(e, "cudaDeviceGetAttribute");
    if ((e = prepare_tile<true, true>()) != cudaSuccess) return bail(e, "smem attribute");
    if ((e = prepare_tile<false, true>()) != cudaSuccess) return bail(e, "smem attribute");
    if ((e = prepare_tile<true, false>()) != cudaSuccess) return bail(e, "smem attribute");
    if ((e = prepare_tile<false, false>()) != cudaSuccess) return bail(e, "smem attribute");
    if ((e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking)) != cudaSuccess) return bail(e, "stream");
    if ((e = cudaMalloc(&m->params, NP * sizeof(float))) != cudaSuccess) return bail(e, "cudaMalloc");
    if ((e = cudaMalloc(&m->m1, NP * sizeof(float))) != cudaSuccess) return bail(e, "cudaMalloc");
    if ((e = cudaMalloc(&m->m2, NP * sizeof(float))) != cudaSuccess) return bail(e, "cudaMalloc");
    if ((e = cudaMalloc(&m->small, (NP + 1) * sizeof(float))) != cudaSuccess) return bail(e, "cudaMalloc");
    if ((e = cudaMalloc(&m->d_err, 2 * sizeof(int))) != cudaSuccess) return bail(e, "cudaMalloc");
    if ((e = cudaMemsetAsync(m->d_err, 0, 2 * sizeof(int), m->stream)) != cudaSuccess) return bail(e, "memset");
    if ((e = cudaMemsetAsync(m->params, 0, NP * sizeof(float), m->stream)) != cudaSuccess) return bail(e, "memset");
    if ((e = cudaMemsetAsync(m->m1, 0, NP * sizeof(float), m->stream)) != cudaSuccess) return bail(e, "memset");
    if ((e = cudaMemsetAsync(m->m2, 0, NP * sizeof(float), m->stream)) != cudaSuccess) return bail(e, "memset");
    if ((e = cudaStreamSynchronize(m->stream)) != cudaSuccess) return bail(e, "sync");
    *out = m;
    return LBMGPU_OK;
}

int lbmgpu_mlp_destroy(lbmgpu_mlp* m) {
    if (!m) return LBMGPU_OK;
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    void* ptrs[] = {m->params, m->m1, m->m2, m->X, m->Y, m->idx, m->grad_part, m->loss_part, m->losses, m->xin, m->yout, m->small,
                    m->d_err};
    for (void* p : ptrs) if (p) cudaFree(p);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return LBMGPU_OK;
}

int lbmgpu_mlp_set_params(lbmgpu_mlp* m, const float* params, int reset_optimizer) {
    if (!m || !params) return LBMGPU_ERR_INVALID;
    MTRY(m, cudaSetDevice(m->device));
    MTRY(m, cudaMemcpyAsync(m->params, params, NP * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    if (reset_optimizer) {
        MTRY(m, cudaMemsetAsync(m->m1, 0, NP * sizeof(float), m->stream));
        MTRY(m, cudaMemsetAsync(m->m2, 0, NP * sizeof(float), m->stream));
        m->t = 0;
    }
    MTRY(m, cudaStreamSynchronize(m->stream));
    return LBMGPU_OK;
}

int lbmgpu_mlp_get_params(lbmgpu_mlp* m, float* params) {
    if (!m || !params) return LBMGPU_ERR_INVALID;
    MTRY(m, cudaSetDevice(m->device));
    MTRY(m, cudaMemcpyAsync(params, m->params, NP * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MTRY(m, cudaStreamSynchronize(m->stream));
    return LBMGPU_OK;
}

int lbmgpu_mlp_set_adam(lbmgpu_mlp* m, float beta1, float beta2, float eps) {
    if (!m || !(beta1 >= 0.f && beta1 < 1.f) || !(beta2 >= 0.f && beta2 < 1.f) || !(eps > 0.f))
        return mfail(m, LBMGPU_ERR_INVALID, "Adam needs 0 <= beta1, beta2 < 1 and eps > 0");
    m->beta1 = beta1; m->beta2 = beta2; m->eps = eps;
    return LBMGPU_OK;
}

int lbmgpu_mlp_set_data(lbmgpu_mlp* m, const float* x, const float* y, int n) {
    if (!m || !x || !y || n < 1) return mfail(m, LBMGPU_ERR_INVALID, "need n >= 1 samples");
    MTRY(m, cudaSetDevice(m->device));
    if (n > m->cap) {
        if (m->X) cudaFree(m->X);
        if (m->Y) cudaFree(m->Y);
        m->X = m->Y = nullptr;
        m->cap = 0;
        MTRY(m, cudaMalloc(&m->X, (size_t)n * NI * sizeof(float)));
        MTRY(m, cudaMalloc(&m->Y, (size_t)n * NO * sizeof(float)));
        m->cap = n;
    }
    MTRY(m, cudaMemcpyAsync(m->X, x, (size_t)n * NI * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    MTRY(m, cudaMemcpyAsync(m->Y, y, (size_t)n * NO * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    MTRY(m, cudaStreamSynchronize(m->stream));
    m->n = n;
    return LBMGPU_OK;
}

int lbmgpu_mlp_train_epoch(lbmgpu_mlp* m, const int* order, int n_order, int batch, float lr, float* mean_loss) {
    if (!m || !order || n_order < 1 || batch < 1 || !(lr > 0.f))
        return mfail(m, LBMGPU_ERR_INVALID, "need an order of >= 1 samples, batch >= 1 and lr > 0");
    if (m->n < 1) return mfail(m, LBMGPU_ERR_INVALID, "no training data (lbmgpu_mlp_set_data)");
    for (int k = 0; k < n_order; ++k)
        if (order[k] < 0 || order[k] >= m->n) return mfail(m, LBMGPU_ERR_INVALID, "order holds an index out of range");
    MTRY(m, cudaSetDevice(m->device));
    if (n_order > m->idx_cap) {
        if (m->idx) cudaFree(m->idx);
        m->idx = nullptr;
        m->idx_cap = 0;
        MTRY(m, cudaMalloc(&m->idx, (size_t)n_order * sizeof(int)));
        m->idx_cap = n_order;
    }
    MTRY(m, cudaMemcpyAsync(m->idx, order, (size_t)n_order * sizeof(int), cudaMemcpyHostToDevice, m->stream));
    const int steps = (n_order + batch - 1) / batch;
    std::vector<float> losses(steps);
    MTRY(m, grow(&m->losses, &m->losses_cap, steps));
    float* const d_losses = m->losses;
    for (int s = 0; s < steps; ++s) {
        const int base = s * batch, count = std::min(batch, n_order - base);
        const int rc = train_batch(m, m->idx, base, count, lr, nullptr, d_losses + s);
        if (rc) return rc;
    }
    cudaError_t e = cudaMemcpyAsync(losses.data(), d_losses, (size_t)steps * sizeof(float), cudaMemcpyDeviceToHost,
                                    m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    MTRY(m, e);
    if (mean_loss) {
        double acc = 0;
        for (float l : losses) acc += l;
        *mean_loss = (float)(acc / steps);
    }
    return LBMGPU_OK;
}

int lbmgpu_mlp_loss_grad(lbmgpu_mlp* m, float* loss, float* grad) {
    if (!m || !loss) return LBMGPU_ERR_INVALID;
    if (m->n < 1) return mfail(m, LBMGPU_ERR_INVALID, "no training data (lbmgpu_mlp_set_data)");
    MTRY(m, cudaSetDevice(m->device));
    const int rc = train_batch(m, nullptr, 0, m->n, 0.f, m->small + 1, m->small);
    if (rc) return rc;
    MTRY(m, cudaMemcpyAsync(loss, m->small, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    if (grad) MTRY(m, cudaMemcpyAsync(grad, m->small + 1, NP * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MTRY(m, cudaStreamSynchronize(m->stream));
    return LBMGPU_OK;
}

int lbmgpu_mlp_forward_ex(lbmgpu_mlp* m, const float* x, int n, float* y, int path) {
    if (!m || !x || !y || n < 1) return mfail(m, LBMGPU_ERR_INVALID, "need n >= 1 inputs");
    if (path != LBMGPU_MLP_PATH_AUTO && path != LBMGPU_MLP_PATH_WARP && path != LBMGPU_MLP_PATH_TCGEN05)
        return mfail(m, LBMGPU_ERR_INVALID, "unknown forward path");
    if (path == LBMGPU_MLP_PATH_TCGEN05 && !m->bf16)
        return mfail(m, LBMGPU_ERR_INVALID, "the tensor-memory path computes in BF16: create the network with bf16 = 1");
    MTRY(m, cudaSetDevice(m->device));
    MTRY(m, grow(&m->xin, &m->xin_cap, (long long)n * NI));
    MTRY(m, grow(&m->yout, &m->yout_cap, (long long)n * NO));
    MTRY(m, cudaMemcpyAsync(m->xin, x, (size_t)n * NI * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    const bool tc = m->bf16 && path != LBMGPU_MLP_PATH_WARP;
    if (tc) {
        k_mlp_fwd_tc<<<std::min((n + TC_M - 1) / TC_M, m->sms * TC_CTAS), TC_M, sizeof(TcSmem), m->stream>>>(m->params, m->xin, n, m->yout, m->d_err);
    } else {
        // two CTAs fit an SM; each takes its share of the tiles
        const int tiles = std::min((n + MLP_T - 1) / MLP_T, 2 * m->sms);
        const size_t sm = m->bf16 ? sizeof(Smem<true>) : sizeof(Smem<false>);
        if (m->bf16)
            k_mlp_tile<true, false><<<tiles, MLP_THREADS, sm, m->stream>>>(m->params, m->xin, nullptr, nullptr, 0, n,
                                                                           0.f, nullptr, nullptr, m->yout, nullptr, 0);
        else
            k_mlp_tile<false, false><<<tiles, MLP_THREADS, sm, m->stream>>>(m->params, m->xin, nullptr, nullptr, 0, n,
                                                                            0.f, nullptr, nullptr, m->yout, nullptr, 0);
    }
    MTRY(m, cudaGetLastError());
    int err = 0;
    MTRY(m, cudaMemcpyAsync(y, m->yout, (size_t)n * NO * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    if (tc) MTRY(m, cudaMemcpyAsync(&err, m->d_err, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    MTRY(m, cudaStreamSynchronize(m->stream));
    if (err) return mfail(m, LBMGPU_ERR_WATCHDOG, "a tensor-core layer did not complete in time");
    return LBMGPU_OK;
}

int lbmgpu_mlp_forward(lbmgpu_mlp* m, const float* x, int n, float* y) {
    return lbmgpu_mlp_forward_ex(m, x, n, y, LBMGPU_MLP_PATH_AUTO);
}

const char* lbmgpu_mlp_last_error(const lbmgpu_mlp* m) { return m ? m->err.c_str() : g_mlp_error.c_str(); }

}  // extern "C"
