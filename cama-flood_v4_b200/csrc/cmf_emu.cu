// cmf_emu.cu -- device kernels of the learned per-cell emulator (no counterpart in the reference).
//
// A 4-layer MLP (input 32 -> 128 -> 128 -> 128 -> 1, ReLU) maps local state plus 8-hop upstream
// messages of every cell to its mean outflow over the next coupling step.  BF16 operands, FP32
// accumulation on the tensor cores: tcgen05 MMAs into tensor memory for the training step, the layer-by-layer
// GEMMs and the inference; mma.sync m16n8k16 tiles for the cross-checks of both (k_gemm, k_mlp_fused).  FP32
// master weights updated by Adam.
// The rollout kernel turns predicted outflows into a mass-conserving storage update along the
// same upstream CSR the physics uses; the stage scheme then recomputes depths.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/cmf_gpu.h"

namespace {

thread_local std::string g_emu_err;

int emu_err(int code, const std::string &m) {
    g_emu_err = m;
    return code;
}

#define EMU_TRY(expr)                                                                         \
    do {                                                                                      \
        cudaError_t e_ = (expr);                                                              \
        if (e_ != cudaSuccess) return emu_err(CMF_E_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// ------------------------------------------------------------------------------------------
// GEMM: C[M,N] (+)= op(A)[M,K] * op(B)[K,N], bf16 in, fp32 accumulate.
// A is [M][K] (transA=0) or [K][M] (transA=1); B is [K][N] (transB=0) or [N][K] (transB=1); all
// row-major with leading dimensions lda/ldb.  Tiles of 64x64 per CTA (4 warps of 32x32), K steps
// of 32 staged in shared memory with both operands stored K-contiguous ([m][k], [n][k]), so the
// m16n8k16 fragments are plain 32-bit shared loads:
//   A frag  a0={A[g][2t..]}, a1={A[g+8][2t..]}, a2={A[g][2t+8..]}, a3={A[g+8][2t+8..]}
//   B frag  b0={B[k=2t..][n=g]}, b1={B[k=2t+8..][n=g]}          (g = lane/4, t = lane%4)
//   C frag  c0,c1 = C[g][2t..], c2,c3 = C[g+8][2t..]
// Epilogue: +bias[n], optional ReLU, store fp32 and/or bf16, or atomic-add fp32 (split-K).
// M, N must be multiples of 64 and K of 32 (callers pad); K may be split over gridDim.z.
// ------------------------------------------------------------------------------------------
constexpr int TM = 64, TN = 64, TK = 32, PAD = 8;

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__global__ void __launch_bounds__(128) k_gemm(int M, int N, int K, const __nv_bfloat16 *__restrict__ A, int lda, int transA,
                                              const __nv_bfloat16 *__restrict__ B, int ldb, int transB,
                                              float *C, int ldc, __nv_bfloat16 *Cb, int ldcb, const float *__restrict__ bias,
                                              int relu, int accumulate, int k_per_split) {
    __shared__ __align__(16) __nv_bfloat16 As[TM][TK + PAD];
    __shared__ __align__(16) __nv_bfloat16 Bs[TN][TK + PAD];
    const int m0 = blockIdx.x * TM, n0 = blockIdx.y * TN;   // row tiles on x: up to 2^31-1 of them
    const int kbeg = blockIdx.z * k_per_split, kend = min(K, kbeg + k_per_split);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int g = lane >> 2, t = lane & 3;
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int r = 0; r < 4; r++) acc[i][j][r] = 0.f;
    for (int k0 = kbeg; k0 < kend; k0 += TK) {
        // stage A tile as [m][k] and B tile as [n][k]
        for (int e = tid; e < TM * TK; e += blockDim.x) {
            const int mm = e / TK, kk = e % TK;
            const int gm = m0 + mm, gk = k0 + kk;
            As[mm][kk] = transA ? A[(size_t)gk * lda + gm] : A[(size_t)gm * lda + gk];
            const int nn = mm;
            const int gn = n0 + nn;
            Bs[nn][kk] = transB ? B[(size_t)gn * ldb + gk] : B[(size_t)gk * ldb + gn];
        }
        __syncthreads();
#pragma unroll
        for (int ks = 0; ks < TK; ks += 16) {
            uint32_t af[2][4], bfr[4][2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int r = wm + i * 16 + g;
                af[i][0] = *reinterpret_cast<const uint32_t *>(&As[r][ks + 2 * t]);
                af[i][1] = *reinterpret_cast<const uint32_t *>(&As[r + 8][ks + 2 * t]);
                af[i][2] = *reinterpret_cast<const uint32_t *>(&As[r][ks + 2 * t + 8]);
                af[i][3] = *reinterpret_cast<const uint32_t *>(&As[r + 8][ks + 2 * t + 8]);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int c = wn + j * 8 + g;
                bfr[j][0] = *reinterpret_cast<const uint32_t *>(&Bs[c][ks + 2 * t]);
                bfr[j][1] = *reinterpret_cast<const uint32_t *>(&Bs[c][ks + 2 * t + 8]);
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) mma_bf16(acc[i][j], af[i], bfr[j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int row = m0 + wm + i * 16 + g + h * 8;
                const int col = n0 + wn + j * 8 + 2 * t;
                float v0 = acc[i][j][2 * h], v1 = acc[i][j][2 * h + 1];
                if (accumulate) {
                    atomicAdd(&C[(size_t)row * ldc + col], v0);
                    atomicAdd(&C[(size_t)row * ldc + col + 1], v1);
                    continue;
                }
                if (bias) { v0 += bias[col]; v1 += bias[col + 1]; }
                if (relu) { v0 = fmaxf(v0, 0.f); v1 = fmaxf(v1, 0.f); }
                if (C) { C[(size_t)row * ldc + col] = v0; C[(size_t)row * ldc + col + 1] = v1; }
                if (Cb) {
                    Cb[(size_t)row * ldcb + col] = __float2bfloat16_rn(v0);
                    Cb[(size_t)row * ldcb + col + 1] = __float2bfloat16_rn(v1);
                }
            }
}

// ------------------------------------------------------------------------------------------
// Fused inference: y[r] = w3 . relu(W2' relu(W1' relu(W0' x_r + b0) + b1) + b2) + b3[0]
//
// One warp owns 16 rows through all four layers.  The m16n8k16 accumulator of two adjacent
// n-tiles (columns 16k..16k+7 and 16k+8..16k+15) holds, lane by lane, exactly the A fragment of
// the k-slab 16k..16k+15 of the next layer, so activations never leave registers: bias, ReLU and
// the bf16 rounding happen on the accumulator and the packed pairs feed the next layer's MMAs.
// The weights are packed once in fragment order (kMlpPack* below: [layer][kslab][ntile][lane] of
// {b0b1, b2b3}) and copied into shared memory by every CTA of a persistent grid; a warp's B
// fragment is one 8-byte shared load per lane.  The chain of MMAs, bias/ReLU/bf16 points and the
// K order are those of the layer-by-layer forward (k_gemm), so y equals its column 0 bit for bit.
// Input columns 32..63 of X are zero padding (the first layer reads k-slabs 0 and 1 only).
// ------------------------------------------------------------------------------------------
constexpr int kMlpKs0 = 2, kMlpKsH = 8, kMlpNt = 16;
constexpr int kMlpOff1 = kMlpKs0 * kMlpNt * 32;                 // uint2 offsets of each layer
constexpr int kMlpOff2 = kMlpOff1 + kMlpKsH * kMlpNt * 32;
constexpr int kMlpOff3 = kMlpOff2 + kMlpKsH * kMlpNt * 32;
constexpr int kMlpPackWords = kMlpOff3 + kMlpKsH * 32;          // last layer: one n-tile (column 0 real)
constexpr int kMlpThreads = 256, kMlpRowsPerCta = 128;

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);   // .x = lo (lower address / lower 16 bits)
    return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ uint32_t bf16_pair(const __nv_bfloat16 *W, int ldw, int k, int n) {
    __nv_bfloat162 v;
    v.x = W[(size_t)k * ldw + n];
    v.y = W[(size_t)(k + 1) * ldw + n];
    return *reinterpret_cast<const uint32_t *>(&v);
}

// W0..W2 bf16 [K][128] row-major, W3 bf16 [128][ldw3]; one thread per packed uint2
__global__ void k_mlp_pack(const __nv_bfloat16 *__restrict__ W0, const __nv_bfloat16 *__restrict__ W1,
                           const __nv_bfloat16 *__restrict__ W2, const __nv_bfloat16 *__restrict__ W3, int ldw3, uint2 *out) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= kMlpPackWords) return;
    const __nv_bfloat16 *W;
    int ldw, rel;
    if (e < kMlpOff1) { W = W0; ldw = 128; rel = e; }
    else if (e < kMlpOff2) { W = W1; ldw = 128; rel = e - kMlpOff1; }
    else if (e < kMlpOff3) { W = W2; ldw = 128; rel = e - kMlpOff2; }
    else { W = W3; ldw = ldw3; rel = e - kMlpOff3; }
    const int nts = (e < kMlpOff3) ? kMlpNt : 1;
    const int lane = rel & 31, nt = (rel >> 5) % nts, ks = (rel >> 5) / nts;
    const int g = lane >> 2, t = lane & 3;
    const int n = nt * 8 + g, k = ks * 16 + 2 * t;
    out[e] = make_uint2(bf16_pair(W, ldw, k, n), bf16_pair(W, ldw, k + 8, n));
}

template <int KS>
__device__ __forceinline__ void mlp_layer(float (&acc)[kMlpNt][4], const uint32_t (&a)[kMlpKsH][4], const uint2 *__restrict__ w,
                                          int lane) {
#pragma unroll
    for (int nt = 0; nt < kMlpNt; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < KS; ks++)
#pragma unroll
        for (int nt = 0; nt < kMlpNt; nt++) {
            const uint2 b2 = w[(ks * kMlpNt + nt) * 32 + lane];
            const uint32_t b[2] = {b2.x, b2.y};
            mma_bf16(acc[nt], a[ks], b);
        }
}

// bias + ReLU + bf16 on the accumulator, repacked as the next layer's A fragments
__device__ __forceinline__ void mlp_chain(const float (&acc)[kMlpNt][4], const float *__restrict__ bias, uint32_t (&a)[kMlpKsH][4],
                                          int t) {
#pragma unroll
    for (int nt = 0; nt < kMlpNt; nt++) {
        const int col = nt * 8 + 2 * t;
        const float b0 = bias[col], b1 = bias[col + 1];
        const float v0 = fmaxf(acc[nt][0] + b0, 0.f), v1 = fmaxf(acc[nt][1] + b1, 0.f);
        const float v2 = fmaxf(acc[nt][2] + b0, 0.f), v3 = fmaxf(acc[nt][3] + b1, 0.f);
        a[nt >> 1][(nt & 1) * 2 + 0] = pack_bf16x2(v0, v1);   // row g
        a[nt >> 1][(nt & 1) * 2 + 1] = pack_bf16x2(v2, v3);   // row g + 8
    }
}

__global__ void __launch_bounds__(kMlpThreads, 2) k_mlp_fused(const __nv_bfloat16 *__restrict__ X, int ldx, int rows,
                                                              const uint2 *__restrict__ wpack, const float *__restrict__ b0,
                                                              const float *__restrict__ b1, const float *__restrict__ b2,
                                                              const float *__restrict__ b3, float *__restrict__ y) {
    extern __shared__ __align__(16) uint2 sw[];
    __shared__ float sb[3 * 128 + 4];
    for (int e = threadIdx.x; e < kMlpPackWords; e += blockDim.x) sw[e] = wpack[e];
    for (int e = threadIdx.x; e < 128; e += blockDim.x) { sb[e] = b0[e]; sb[128 + e] = b1[e]; sb[256 + e] = b2[e]; }
    if (threadIdx.x == 0) sb[384] = b3[0];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int ntiles = (rows + kMlpRowsPerCta - 1) / kMlpRowsPerCta;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int r0 = tile * kMlpRowsPerCta + warp * 16;
        if (r0 >= rows) continue;                    // rows is a multiple of 16: groups are whole
        uint32_t a[kMlpKsH][4];
        const __nv_bfloat16 *x0 = X + (size_t)(r0 + g) * ldx, *x1 = X + (size_t)(r0 + g + 8) * ldx;
#pragma unroll
        for (int ks = 0; ks < kMlpKs0; ks++) {
            a[ks][0] = *reinterpret_cast<const uint32_t *>(x0 + ks * 16 + 2 * t);
            a[ks][1] = *reinterpret_cast<const uint32_t *>(x1 + ks * 16 + 2 * t);
            a[ks][2] = *reinterpret_cast<const uint32_t *>(x0 + ks * 16 + 8 + 2 * t);
            a[ks][3] = *reinterpret_cast<const uint32_t *>(x1 + ks * 16 + 8 + 2 * t);
        }
        float acc[kMlpNt][4];
        mlp_layer<kMlpKs0>(acc, a, sw, lane);
        mlp_chain(acc, sb, a, t);
        mlp_layer<kMlpKsH>(acc, a, sw + kMlpOff1, lane);
        mlp_chain(acc, sb + 128, a, t);
        mlp_layer<kMlpKsH>(acc, a, sw + kMlpOff2, lane);
        mlp_chain(acc, sb + 256, a, t);
        float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < kMlpKsH; ks++) {
            const uint2 b2 = sw[kMlpOff3 + ks * 32 + lane];
            const uint32_t b[2] = {b2.x, b2.y};
            mma_bf16(o, a[ks], b);
        }
        if (t == 0) {
            y[r0 + g] = o[0] + sb[384];
            y[r0 + g + 8] = o[2] + sb[384];
        }
    }
}

// dZ = dA * (act > 0) -> bf16, for ReLU layers (act stored in bf16 by the forward pass)
__global__ void k_relu_bwd(int n, const float *__restrict__ dA, const __nv_bfloat16 *__restrict__ act, __nv_bfloat16 *dZ,
                           float *dZf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = __bfloat162float(act[i]) > 0.f ? dA[i] : 0.f;
    dZ[i] = __float2bfloat16_rn(v);
    if (dZf) dZf[i] = v;
}

// column sums of a [rows][cols] fp32 matrix into out[cols] (bias gradients), one block per column
__global__ void k_colsum(int rows, int cols, const float *__restrict__ X, float *out) {
    const int c = blockIdx.x;
    float s = 0.f;
    for (int r = threadIdx.x; r < rows; r += blockDim.x) s += X[(size_t)r * cols + c];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    __shared__ float w[32];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += w[k];
        out[c] = t;
    }
}

// Adam on fp32 master weights, bf16 copy for the tensor cores; up to 8 tensors in one launch, tensor
// k on blockIdx.y (the 8 tensors of a training step took 8 launches, each far below a wave)
constexpr int kAdamMax = 8;
struct AdamSet {
    int n[kAdamMax];
    float *w[kAdamMax];
    __nv_bfloat16 *wb[kAdamMax];
    const float *grad[kAdamMax];
    float *m[kAdamMax], *v[kAdamMax];
    float wd[kAdamMax];
};
__global__ void k_adam(AdamSet a, float lr, float b1, float b2, float eps, float bc1, float bc2) {
    const int k = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n[k]) return;
    float *w = a.w[k], *m = a.m[k], *v = a.v[k];
    const float gr = a.grad[k][i] + a.wd[k] * w[i];
    const float mi = b1 * m[i] + (1.f - b1) * gr;
    const float vi = b2 * v[i] + (1.f - b2) * gr * gr;
    m[i] = mi;
    v[i] = vi;
    const float upd = lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    const float wn = w[i] - upd;
    w[i] = wn;
    if (a.wb[k]) a.wb[k][i] = __float2bfloat16_rn(wn);
}

// mean-squared-error gradient on column 0 of Y [rows][ldy]: dY = 2 (Y - t) / rows (other columns 0),
// bf16 copy for the tensor cores, per-block loss partials
__global__ void k_mse_grad(int rows, int valid, int ldy, const float *__restrict__ Y, const float *__restrict__ t, float *dY,
                           __nv_bfloat16 *dYb, float *loss_part) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.f;
    if (r < rows) {
        const float e = (r < valid) ? Y[(size_t)r * ldy] - t[r] : 0.f;
        l = e * e;
        for (int c = 0; c < ldy; c++) {
            const float v = (c == 0) ? 2.f * e / (float)valid : 0.f;
            dY[(size_t)r * ldy + c] = v;
            dYb[(size_t)r * ldy + c] = __float2bfloat16_rn(v);
        }
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
    __shared__ float w[32];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) s += w[k];
        loss_part[blockIdx.x] = s;
    }
}

// ------------------------------------------------------------------------------------------
// features: 14 local + 16 message channels + 2 hydraulic estimates = 32 per cell (bf16 rows)
//
// The upstream messages are computed first as fp32 planes (one coalesced pass per hop), then one
// assembly pass writes each cell's 32 features as four 16-byte stores; nothing writes X columns
// one at a time (rows are 128 bytes apart, so column writes would touch every row's sector per hop).
// ------------------------------------------------------------------------------------------
struct EmuNet {
    int N, R;
    const int *next, *up_ptr, *up_idx;
    const double *rivelv, *elevtn, *nxtdst, *rivwth, *rivhgt, *rivlen, *rivstomax, *qref, *rivman;
    double pmanfld;
};


// one hop of upstream message passing: out[i] = sum over upstream j of in[j], ascending upstream order.  The
// first hop reads the fp64 last-step outflow and runoff (rounded to fp32), the later ones the hop before's
// planes.  Bound by its gathers through L1, so a hop of its own: two hops in one pass gather a cell's second
// ring anew, through two more index loads, for a third less memory traffic.  Two upstream cells are in flight
// at a time.  Eight hops and the assembly for 32 x 299k cells: 1215 us with two hops a pass, 1081 us with one.
template <bool FromState>
__global__ void __launch_bounds__(256) k_emu_hop(EmuNet n, const float *__restrict__ in_a, const float *__restrict__ in_b,
                                                 const double *__restrict__ qa, const double *__restrict__ qb, float *out_a,
                                                 float *out_b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n.N) return;
    const size_t mo = (size_t)blockIdx.y * n.N;
    auto va = [&](int j) { return FromState ? (float)qa[mo + j] : in_a[mo + j]; };
    auto vb = [&](int j) { return FromState ? (float)qb[mo + j] : in_b[mo + j]; };
    float a = 0.f, b = 0.f;
    const int k1 = n.up_ptr[i + 1];
    for (int k = n.up_ptr[i]; k < k1; k += 2) {
        const int j0 = n.up_idx[k], j1 = k + 1 < k1 ? n.up_idx[k + 1] : -1;
        const float a0 = va(j0), b0 = vb(j0);
        float a1 = 0.f, b1 = 0.f;
        if (j1 >= 0) {
            a1 = va(j1);
            b1 = vb(j1);
        }
        a += a0;
        b += b0;
        if (j1 >= 0) {
            a += a1;
            b += b1;
        }
    }
    out_a[mo + i] = a;
    out_b[mo + i] = b;
}

// Features feed a bf16 network (8-bit mantissa), so they are computed in fp32 with fast
// reciprocals and the hardware log/exp approximations: one reciprocal of the discharge scale per
// cell instead of a division per feature.  Training and inference use this same kernel.
// sign(x) log(1 + |x|); below 1e-3 the two-term series a - a^2/2 (relative error < a^2/3), where
// the hardware logarithm of 1 + a would lose the small ratios (runoff over a large river's scale)
__device__ __forceinline__ float fslog(float x) {
    const float a = fabsf(x);
    return copysignf(a < 1e-3f ? a * (1.f - 0.5f * a) : __logf(1.f + a), x);
}

// Manning discharge of a rectangular section of area A, hydraulic depth h and friction slope s
__device__ __forceinline__ float manning_q(float area, float h, float s, float inv_man) {
    if (!(area > 0.f) || !(h > 0.f)) return 0.f;
    return copysignf(area * __expf(0.6666667f * __logf(h)) * sqrtf(fabsf(s)) * inv_man, s);
}

// Bound by the latency of its 35 loads a cell, so six blocks per SM are asked for (54 registers and four
// blocks without it); a row leaves through shared memory, four lanes writing its 64 bytes together, where a
// lane per row wrote half a sector at a time.  32 x 299k cells, four passes of two hops included: 1337 us as
// one row a lane, 1313 us through shared memory, 1218 us with six blocks (seven: 1262 us).
// features of cell i of member blockIdx.y; planes [2*(hops+1)][M*N] (0, 1 unused; 2h+2, 2h+3 = hop h)
__global__ void __launch_bounds__(256, 6) k_emu_assemble(EmuNet n, const double *__restrict__ rivsto, const double *__restrict__ fldsto,
                               const double *__restrict__ levsto, const double *__restrict__ rivdph,
                               const double *__restrict__ flddph, const double *__restrict__ fldfrc,
                               const double *__restrict__ qprev, const double *__restrict__ runoff,
                               const float *__restrict__ planes, size_t plane, int hops, __nv_bfloat16 *X, int ldx,
                               int rows_per_member) {
    __shared__ uint4 rows_s[8][128];
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = min(i0, n.N - 1);
    // member blockIdx.y: state arrays are member-major [M][N], X rows [M][rows_per_member]
    const size_t mo = (size_t)blockIdx.y * n.N, gi = mo + i;
    const float qf = (float)n.qref[i];
    const float iq = __frcp_rn(qf);
    const double Sd = rivsto[gi] + fldsto[gi] + (levsto ? levsto[gi] : 0.0);
    const float S = (float)Sd;
    const float rdph = (float)rivdph[gi], fdph = (float)flddph[gi];
    const float len = (float)n.rivlen[i], wth = (float)n.rivwth[i], hgt = (float)n.rivhgt[i];
    float f[32];
    f[0] = fslog(S * __frcp_rn((float)n.rivstomax[i]));
    f[1] = rdph * __frcp_rn(hgt);
    f[2] = fslog(fdph);
    f[3] = fslog((float)qprev[gi] * iq);
    f[4] = fslog((float)runoff[gi] * iq);
    f[5] = (float)fldfrc[gi];
    const bool mouth = i >= n.R;
    const int j = mouth ? i : n.next[i];
    const float inv_dst = __frcp_rn(mouth ? 10000.f : (float)n.nxtdst[i]);
    const double sfc = n.rivelv[i] + rivdph[gi], sfcn = mouth ? n.elevtn[i] : n.rivelv[j] + rivdph[mo + j];
    const float slope = (float)(sfc - sfcn) * inv_dst;   // elevations subtracted in fp64
    f[6] = fslog(1000.f * slope);
    f[7] = fslog(1000.f * (float)(n.elevtn[i] - (mouth ? n.elevtn[i] : n.elevtn[j])) * __frcp_rn((float)n.nxtdst[i]));
    f[8] = __logf(len) - 9.5f;
    f[9] = __logf(wth) - 4.0f;
    f[10] = __logf(hgt) - 1.0f;
    f[11] = __logf(qf) - 3.0f;
    f[12] = mouth ? 1.f : 0.f;
    f[13] = fslog(S * iq * (1.f / 3600.f));
#pragma unroll
    for (int h = 0; h < 8; h++) {
        if (h < hops) {
            f[14 + 2 * h] = fslog(planes[(size_t)(2 + 2 * h) * plane + gi] * iq);
            f[15 + 2 * h] = fslog(planes[(size_t)(3 + 2 * h) * plane + gi] * iq);
        } else {
            f[14 + 2 * h] = f[15 + 2 * h] = 0.f;
        }
    }
    // hydraulic estimates: Manning discharge of the channel and of the floodplain at the current
    // water-surface slope (the state the local-inertial scheme relaxes towards within an hour)
    const float af = fmaxf((float)fldsto[gi] * __frcp_rn(len) - fdph * wth, 0.f);
    f[30] = fslog(manning_q(wth * rdph, rdph, slope, __frcp_rn((float)n.rivman[i])) * iq);
    f[31] = fslog(manning_q(af, fdph, fmaxf(-0.005f, fminf(0.005f, slope)), __frcp_rn((float)n.pmanfld)) * iq);
    const int lane = threadIdx.x & 31;
    uint4 *ws = rows_s[threadIdx.x >> 5];
#pragma unroll
    for (int v = 0; v < 4; v++) {
        uint4 u;
        u.x = pack_bf16x2(f[8 * v + 0], f[8 * v + 1]);
        u.y = pack_bf16x2(f[8 * v + 2], f[8 * v + 3]);
        u.z = pack_bf16x2(f[8 * v + 4], f[8 * v + 5]);
        u.w = pack_bf16x2(f[8 * v + 6], f[8 * v + 7]);
        ws[lane * 4 + (v ^ ((lane >> 1) & 3))] = u;
    }
    __syncwarp();
    __nv_bfloat16 *xw = X + ((size_t)blockIdx.y * rows_per_member + (i0 - lane)) * ldx;
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const int r = 8 * v + (lane >> 2), c = lane & 3;
        if (i0 - lane + r < n.N) *reinterpret_cast<uint4 *>(xw + (size_t)r * ldx + 8 * c) = ws[r * 4 + (c ^ ((r >> 1) & 3))];
    }
}

// Mass-conserving rollout of one coupling step from the predicted transformed mean outflow:
// Q_i = qref_i * expm1(max(base_i + y_i, 0)) with base_i = log1p(Qprev_i/qref_i) when the network
// predicts the change over the step (residual != 0) and 0 when it predicts the value itself, limited
// to the storage the cell holds plus its own runoff over DT (so storage never goes negative whatever
// its upstream delivers); storage then changes by (inflow + runoff - outflow) * DT with the inflow
// gathered over the upstream CSR.
__global__ void k_emu_rollout(EmuNet n, const float *y, int ldy, int rows_per_member, const int *active, double dt,
                              int residual, const double *runoff, const double *rivsto, const double *fldsto,
                              const double *levsto, const double *qprev, double *qout) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n.N || !active[blockIdx.y]) return;
    const size_t mo = (size_t)blockIdx.y * n.N;
    y += (size_t)blockIdx.y * rows_per_member * ldy;
    runoff += mo; rivsto += mo; fldsto += mo; if (levsto) levsto += mo; qout += mo;
    const double S = rivsto[i] + fldsto[i] + (levsto ? levsto[i] : 0.0);
    // the network predicts the change of log1p(Q/qref) over the step (residual on the last outflow)
    const double base = residual ? log1p(fmax(qprev[mo + i], 0.0) / n.qref[i]) : 0.0;
    const double yi = fmax(base + (double)y[(size_t)i * ldy], 0.0);
    double q = n.qref[i] * expm1(yi);
    q = fmin(q, S / dt + runoff[i]);
    qout[i] = fmax(q, 0.0);
}

__global__ void k_emu_update(EmuNet n, const int *active, double dt, const double *runoff, const double *qout, double *rivsto,
                             double *fldsto, double *levsto, double *rivout_pre, double *fldout_pre, double *qprev) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n.N || !active[blockIdx.y]) return;
    const size_t mo = (size_t)blockIdx.y * n.N;
    runoff += mo; qout += mo; rivsto += mo; fldsto += mo; if (levsto) levsto += mo; rivout_pre += mo; fldout_pre += mo;
    qprev += mo;
    double inflow = 0.0;
    for (int k = n.up_ptr[i]; k < n.up_ptr[i + 1]; k++) inflow += qout[n.up_idx[k]];
    const double S = rivsto[i] + fldsto[i] + (levsto ? levsto[i] : 0.0);
    const double Snew = fmax(S + (inflow + runoff[i] - qout[i]) * dt, 0.0);
    rivsto[i] = Snew;   // the stage scheme re-splits river / floodplain / protected storage
    fldsto[i] = 0.0;
    if (levsto) levsto[i] = 0.0;
    rivout_pre[i] = qout[i];
    fldout_pre[i] = 0.0;
    qprev[i] = qout[i];
}


// ------------------------------------------------------------------------------------------
// Fused inference on the 5th-generation tensor cores (tcgen05, sm_100a).
//
// One CTA per SM (a persistent grid) holds all four layers' weights in shared memory once, as the MMAs'
// B operands, and runs two 128-row tiles at a time.  A tile's activations never touch shared memory:
// slot s (warps 16s..16s+15) owns 192 of the SM's tensor-memory columns, 128 for the fp32 accumulator and 64
// for the next layer's A operand (row = lane, two bf16 of consecutive k per column), which tcgen05.mma
// reads from there.  With both operands in shared memory one 128x128x16 product reads 8 KB in the 64
// cycles it takes, all of the SM's shared-memory bandwidth, next to the epilogue's stores; so it reads
// 4 KB.  B is 128-byte swizzled (sw128_off).  Per layer of a slot: its warps (warp
// 16s+4g+q: TMEM lanes 32q..32q+31, columns 32g..32g+31) wait for the layer's products, read the
// accumulator with tcgen05.ld, add the bias, apply ReLU and the bf16 rounding in one cvt and write the
// next A columns; after the slot's one barrier its first warp issues the next layer's tcgen05.mma chain
// (one elected thread; M=128, N=128 or 16, K=16 per instruction) and commits it to the slot's mbarrier.  While one slot runs
// its epilogue the tensor pipe serves the other; sixteen warps keep the epilogue to 32 columns per thread,
// as a layer's time is the chain wait, load, convert, store, barrier, issue, product.  The last layer
// (N=16, column 0 real) adds b3 and writes y, and the next tile's X goes in.  Tiles are dealt to the CTAs
// first and to their slots second, so that a small call spreads over the SMs.  Every wait is bounded: a
// wait that runs out ends the slot's loop at its next barrier (a vote), and its first warp drains the
// MMAs it issued (one more commit, waited for with the full bound) before the tensor memory is released.
// The rounding points equal the layer-by-layer chain (bf16 inputs, fp32 accumulation, bf16 activations) and
// the K=16 steps run in the same order, so the outputs equal that chain bit for bit.
// 4.2M rows: 511 us with four 128-thread slots, activations in shared memory and a polling issuer warp;
// 582 us in this form with the MMAs issued under a branch on the thread index; 401 us as it stands, where the
// products alone would take 202 us at the measured bf16 rate.  26.6k rows: 16.4 and 10.4 us.
// ------------------------------------------------------------------------------------------
constexpr int kTcRows = 128;
constexpr int kTcSlots = 2;                           // tiles in flight per CTA
constexpr int kTcSlotThreads = 512;
constexpr int kTcThreads = kTcSlotThreads * kTcSlots;
constexpr int kTcW0 = 0;                              // byte offsets inside the packed image
constexpr int kTcW1 = kTcW0 + 128 * 64 * 2;           // layer 0: N=128, K=32 (of a 64-column block)
constexpr int kTcW2 = kTcW1 + 128 * 128 * 2;          // layers 1, 2: N=128, K=128
constexpr int kTcW3 = kTcW2 + 128 * 128 * 2;          // layer 3: N=16, K=128
constexpr int kTcWBytes = kTcW3 + 16 * 128 * 2;
constexpr int kTcBias = kTcWBytes;                    // b0 b1 b2 (3 x 128 floats), b3[0]
constexpr int kTcMisc = kTcBias + (3 * 128 + 4) * 4;  // done[2], drain[2] mbarriers; TMEM address
constexpr int kTcSmem = kTcMisc + 2 * kTcSlots * 8 + 16;
constexpr int kTcSlotCols = 192, kTcACol = 128;       // a slot's tensor-memory columns, the A operand's place
constexpr int kTcCols = 512;                          // allocated (a power of two)
#ifndef CMF_TC_WAIT_LIMIT
#define CMF_TC_WAIT_LIMIT (1 << 20)
#endif
constexpr int kTcWaitLimit = CMF_TC_WAIT_LIMIT;        // polls of an MMA completion before giving up
int g_tc_wait_limit = kTcWaitLimit;                   // host side: the bound the next launches use

__device__ int g_mlp_tc_status;                       // 0 ok; 1: an MMA completion wait ran out

__host__ __device__ constexpr uint64_t umma_smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    // start address, leading- and stride-dimension byte offsets (16-byte units), version 1,
    // base offset 0, no swizzle
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// The layout of the inference image: 128-byte swizzled, a matrix of R rows cut into
// blocks of 64 bf16 columns, block-major, a row's 128 bytes together, its 16-byte chunk c at c ^ (row % 8).
__host__ __device__ constexpr uint32_t sw128_off(int r, int c, int R) {
    return (uint32_t)((c >> 6) * (R * 128) + r * 128 + ((((c >> 3) & 7) ^ (r & 7)) << 4) + (c & 7) * 2);
}
__host__ __device__ constexpr uint64_t sw128_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return umma_smem_desc(saddr, lbo, sbo) | (2ull << 61);
}
// K=16 step s of a matrix at `base` (1024-byte aligned)
__device__ __forceinline__ uint64_t sw128_kmajor(uint32_t base, int R, int s) {
    return sw128_desc(base + (s >> 2) * (R * 128) + (s & 3) * 32, 16, 1024);
}
__host__ __device__ constexpr uint32_t umma_idesc_bf16_f32(int M, int N) {
    // D fp32, A and B bf16, both K-major, N/8 and M/16
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// byte offset of element (r, k) of an R-row K-major operand in the canonical layout
__host__ __device__ constexpr uint32_t canon_off(int r, int k, int R) {
    return (uint32_t)((k >> 3) * (R * 16) + (r >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// B operands of the four layers as one shared-memory image: element (n, k) = W[k][n], columns 32.. of
// layer 0 zero
__global__ void k_mlp_tc_pack(const __nv_bfloat16 *__restrict__ W0, const __nv_bfloat16 *__restrict__ W1,
                              const __nv_bfloat16 *__restrict__ W2, const __nv_bfloat16 *__restrict__ W3, int ldw3,
                              __nv_bfloat16 *out) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    const int n0 = 128 * 64, n1 = 128 * 128, n3 = 16 * 128;
    if (e >= n0 + 2 * n1 + n3) return;
    int n, k, R, base;
    const __nv_bfloat16 *W;
    int ldw;
    if (e < n0) { n = e / 64; k = e % 64; R = 128; base = kTcW0; W = W0; ldw = 128; }
    else if (e < n0 + n1) { const int q = e - n0; n = q / 128; k = q % 128; R = 128; base = kTcW1; W = W1; ldw = 128; }
    else if (e < n0 + 2 * n1) { const int q = e - n0 - n1; n = q / 128; k = q % 128; R = 128; base = kTcW2; W = W2; ldw = 128; }
    else { const int q = e - n0 - 2 * n1; n = q / 128; k = q % 128; R = 16; base = kTcW3; W = W3; ldw = ldw3; }
    out[(base + sw128_off(n, k, R)) / 2] = (e < n0 && k >= 32) ? __float2bfloat16_rn(0.f) : W[(size_t)k * ldw + n];
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        :: "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}

// one thread of a converged warp, chosen by the hardware: the form in which ptxas keeps the operands of
// tcgen05 instructions in uniform registers (under a branch on the thread index each MMA took about 200
// cycles to issue)
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\tselp.u32 %0, 1, 0, e;\n\t}\n" : "=r"(p));
    return p != 0;
}

// the same with A in tensor memory (K-major: lane = row, two consecutive k per 32-bit column)
__device__ __forceinline__ void umma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        :: "r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void umma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(mbar) : "memory");
}

// bounded wait on an mbarrier phase; false when the limit ran out
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, int limit) {
    for (int i = 0; i < limit; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok) : "r"(mbar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld1(uint32_t taddr, uint32_t &v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        :: "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
           "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint4 &a, const uint4 &b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 :: "r"(taddr), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ReLU and round-to-nearest bf16 of two fp32 values in one instruction (ReLU commutes with the
// rounding, so this equals rounding max(x, 0)); lo goes to the lower half
__device__ __forceinline__ uint32_t relu_bf16x2(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// layer epilogue of 32 columns of one row: bias + ReLU + bf16 into 16 columns of the next A operand
__device__ __forceinline__ void tc_epilogue_hidden(uint32_t tmem_d, const float *bias, uint32_t tmem_a) {
    uint32_t v[32], w[16];
    tmem_ld32(tmem_d, v);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; j++)
        w[j] = relu_bf16x2(__uint_as_float(v[2 * j]) + bias[2 * j], __uint_as_float(v[2 * j + 1]) + bias[2 * j + 1]);
    tmem_st16(tmem_a, w);
    tmem_wait_st();
}

// named barrier with an OR over the participants' flags: every participant gets the same answer
__device__ __forceinline__ bool named_bar_or(int id, int nthreads, bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.or.pred p, %2, %3, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(r) : "r"((uint32_t)v), "r"(id), "r"(nthreads) : "memory");
    return r != 0;
}
__global__ void __launch_bounds__(kTcThreads, 1) k_mlp_tc(const __nv_bfloat16 *__restrict__ X, int ldx, int rows,
                                                        const uint4 *__restrict__ wimg, const float *__restrict__ b0,
                                                        const float *__restrict__ b1, const float *__restrict__ b2,
                                                        const float *__restrict__ b3, float *__restrict__ y,
                                                        int wait_limit) {
    extern __shared__ __align__(1024) unsigned char sm[];
    float *sb = reinterpret_cast<float *>(sm + kTcBias);
    uint64_t *done = reinterpret_cast<uint64_t *>(sm + kTcMisc), *drain = done + kTcSlots;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(drain + kTcSlots);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // weights and biases into shared memory
    for (int e = tid; e < kTcWBytes / 16; e += kTcThreads) reinterpret_cast<uint4 *>(sm)[e] = wimg[e];
    for (int e = tid; e < 128; e += kTcThreads) { sb[e] = b0[e]; sb[128 + e] = b1[e]; sb[256 + e] = b2[e]; }
    if (tid == 0) {
        sb[384] = b3[0];
        for (int q = 0; q < 2 * kTcSlots; q++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(done + q)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {   // one warp allocates the CTA's accumulator columns and releases the allocation permit
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(tslot)), "r"(kTcCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tslot, 0);
    const int ntiles = (rows + kTcRows - 1) / kTcRows;
    const int stride = kTcSlots * (int)gridDim.x;             // tiles of slot s: first + j * stride
    const int sl = __shfl_sync(0xffffffffu, warp >> 4, 0), g = (warp >> 2) & 3, q = warp & 3;
    const int r = 32 * q + lane;                              // this thread's row == TMEM lane
    const uint32_t td = tmem + (uint32_t)(kTcSlotCols * sl), trow = td + ((uint32_t)(32 * q) << 16);
    const uint32_t dn = smem_u32(done + sl), sw = smem_u32(sm);
    const bool lead = __shfl_sync(0xffffffffu, (warp & 15) == 0, 0);      // the slot's first warp
    // issues layer L of the slot's tile (one thread of the lead warp): A from the slot's columns, B from
    // the image
    auto issue = [&](int L) {
        tc_fence_after();
        if (!elect_one()) return;
        const uint32_t wb = sw + (L == 0 ? kTcW0 : L == 1 ? kTcW1 : L == 2 ? kTcW2 : kTcW3);
        const uint32_t id = L == 3 ? umma_idesc_bf16_f32(128, 16) : umma_idesc_bf16_f32(128, 128);
        const int ksteps = L == 0 ? 2 : 8, R = L == 3 ? 16 : 128;
#pragma unroll
        for (int st = 0; st < 8; st++)
            if (st < ksteps) umma_bf16_ta(td, td + kTcACol + 8 * st, sw128_kmajor(wb, R, st), id, st > 0 ? 1u : 0u);
        umma_commit(dn);
    };
    // this row's quarter pair of X (16 bf16: columns 16g..16g+15, g < 2) of a tile
    uint4 xn[2];
    auto load_x = [&](int tile) {
        xn[0] = xn[1] = make_uint4(0u, 0u, 0u, 0u);
        if (g < 2 && tile < ntiles && tile * kTcRows + r < rows) {
            const uint4 *p = reinterpret_cast<const uint4 *>(X + (size_t)(tile * kTcRows + r) * ldx + 16 * g);
            xn[0] = p[0];
            xn[1] = p[1];
        }
    };
    auto put_x = [&]() {
        if (g < 2) tmem_st8(trow + kTcACol + 8 * g, xn[0], xn[1]);
        tmem_wait_st();
    };
    bool ok = true, issued = false;
    uint32_t phase = 0;
    int t = blockIdx.x + sl * (int)gridDim.x;
    if (t < ntiles) {
        load_x(t);
        put_x();
        load_x(t + stride);                                   // fetched while the tile before it runs
        tc_fence_before();
        named_bar_or(1 + sl, kTcSlotThreads, false);
        if (lead) { issue(0); issued = true; }
    }
    for (; t < ntiles && ok; t += stride) {
        const int row = t * kTcRows + r;
#pragma unroll 1
        for (int layer = 0; layer < 4; layer++) {
            const bool fail = !mbar_wait(dn, phase, wait_limit);
            phase ^= 1u;
            tc_fence_after();
            if (layer < 3) {
                tc_epilogue_hidden(trow + 32 * g, sb + 128 * layer + 32 * g, trow + kTcACol + 16 * g);
            } else {
                if (g == 0) {
                    uint32_t v;
                    tmem_ld1(trow, v);
                    tmem_wait_ld();
                    if (row < rows) y[row] = __uint_as_float(v) + sb[384];
                }
                put_x();
                load_x(t + 2 * stride);
            }
            tc_fence_before();
            ok = !named_bar_or(1 + sl, kTcSlotThreads, fail);
            if (!ok) break;
            if (lead && (layer < 3 || t + stride < ntiles)) issue((layer + 1) & 3);
        }
    }
    if (issued) {
        // every MMA this thread issued completes before the columns are released: one more commit
        // tracks them all, waited for with the full bound
        if (elect_one()) umma_commit(smem_u32(drain + sl));
        mbar_wait(smem_u32(drain + sl), 0u, kTcWaitLimit);
    }
    if (lead && lane == 0 && !ok) atomicExch(&g_mlp_tc_status, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(kTcCols) : "memory");
}

// ------------------------------------------------------------------------------------------
// Training GEMM on the 5th-generation tensor cores: the contract of k_gemm (C (+)= op(A) op(B),
// bias + ReLU, fp32 and/or bf16 output, or split-K atomic accumulation), with the products on
// tcgen05.  CTA tile 128 rows x NT columns (NT = 128, or 64 when N is not a multiple of 128); K in
// chunks of 64 staged into two shared-memory buffers in the canonical K-major no-swizzle layout
// (operands stored transposed in global memory are written element by element); one thread issues
// the chunk's MMAs (M=128, N=NT, K=16, bf16 x bf16 -> fp32) into a tensor-memory accumulator and
// commits them to the buffer's mbarrier, which completes (bounded wait) before the buffer is refilled.
// Epilogue: thread t owns row t (TMEM lane t) and reads its NT accumulator columns 32 at a time.
// With `zstride` > 0 every K slice stores its own partial product at C + blockIdx.z * zstride
// (plain stores, no bias or ReLU); k_splitk_reduce then adds the slices to the output in slice
// order, so a split-K product is the same bits on every run.
// ------------------------------------------------------------------------------------------
constexpr int kGThreads = 128;                          // = rows of the tile = TMEM lanes
constexpr int kGK = 64;                                 // K per staged chunk
constexpr int kGTileBytes = 128 * kGK * 2;              // one 128-row operand chunk (bf16)
constexpr int kGBuf = 2 * kGTileBytes;                  // A and B chunks of one buffer
constexpr int kGSmem = 2 * kGBuf + 64;                  // two buffers, two mbarriers, TMEM address

// stages rows [r0, r0 + 128) (rows >= rmax zero) x k [k0, k0 + kc) of an operand whose element
// (r, k) is at P[r * ld + k] (kmajor) or P[k * ld + r] (r contiguous) into the canonical layout
__device__ __forceinline__ void gemm_stage(unsigned char *dst, int R, const __nv_bfloat16 *__restrict__ P, int ld,
                                           bool kmajor, int r0, int rmax, int k0, int kc) {
    const int tid = threadIdx.x;
    if (kmajor) {
        const int cpr = kc / 8;                          // 16-byte chunks per row
        for (int e = tid; e < R * cpr; e += kGThreads) {
            const int r = e / cpr, kq = e - r * cpr;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (r0 + r < rmax) v = *reinterpret_cast<const uint4 *>(P + (size_t)(r0 + r) * ld + k0 + kq * 8);
            *reinterpret_cast<uint4 *>(dst + canon_off(r, kq * 8, R)) = v;
        }
    } else {
        const int cpk = R / 8;                           // 16-byte chunks along r per k
        for (int e = tid; e < kc * cpk; e += kGThreads) {
            const int k = e / cpk, rq = e - k * cpk;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (r0 + rq * 8 < rmax) v = *reinterpret_cast<const uint4 *>(P + (size_t)(k0 + k) * ld + r0 + rq * 8);
            const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
            for (int j = 0; j < 8; j++) *reinterpret_cast<__nv_bfloat16 *>(dst + canon_off(rq * 8 + j, k, R)) = h[j];
        }
    }
}

template <int NT>
__global__ void __launch_bounds__(kGThreads) k_gemm_tc(int M, int N, int K, const __nv_bfloat16 *__restrict__ A, int lda,
                                                       int transA, const __nv_bfloat16 *__restrict__ B, int ldb, int transB,
                                                       float *C, int ldc, __nv_bfloat16 *Cb, int ldcb,
                                                       const float *__restrict__ bias, int relu, int accumulate,
                                                       int k_per_split, int wait_limit, size_t zstride) {
    extern __shared__ __align__(1024) unsigned char sm[];
    if (zstride) C += blockIdx.z * zstride;
    uint64_t *mbar = reinterpret_cast<uint64_t *>(sm + 2 * kGBuf);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + 2 * kGBuf + 16);
    const int tid = threadIdx.x, warp = tid >> 5;
    const int m0 = blockIdx.x * 128, n0 = blockIdx.y * NT;
    const int kbeg = blockIdx.z * k_per_split, kend = min(K, kbeg + k_per_split);
    if (tid == 0) {
        for (int b = 0; b < 2; b++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&mbar[b])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tslot)), "r"(NT)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t idesc = umma_idesc_bf16_f32(128, NT);
    uint32_t phase[2] = {0u, 0u};
    bool issued[2] = {false, false};
    bool failed = false;
    int chunk = 0;
    for (int k0 = kbeg; k0 < kend; k0 += kGK, chunk++) {
        const int buf = chunk & 1;
        unsigned char *sA = sm + buf * kGBuf, *sB = sA + kGTileBytes;
        if (issued[buf]) {   // the MMAs that read this buffer two chunks ago must have finished
            const bool ok = mbar_wait(smem_u32(&mbar[buf]), phase[buf], wait_limit);
            if (__syncthreads_or(ok ? 0 : 1)) { failed = true; break; }   // block-uniform
            phase[buf] ^= 1u;
            issued[buf] = false;
            tc_fence_after();
        }
        const int kc = min(kGK, kend - k0);             // a multiple of 32
        gemm_stage(sA, 128, A, lda, !transA, m0, M, k0, kc);
        gemm_stage(sB, NT, B, ldb, transB != 0, n0, N, k0, kc);
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            for (int s = 0; s < kc / 16; s++) {
                const uint64_t ad = umma_smem_desc(smem_u32(sA) + 2 * s * (128 * 16), 128 * 16, 128);
                const uint64_t bd = umma_smem_desc(smem_u32(sB) + 2 * s * (NT * 16), NT * 16, 128);
                umma_bf16(tmem, ad, bd, idesc, (chunk > 0 || s > 0) ? 1u : 0u);
            }
            umma_commit(smem_u32(&mbar[buf]));
        }
        issued[buf] = true;
    }
    // the outstanding commits, oldest first (after a failure: drain them with the full bound
    // before the accumulator columns are released)
    for (int q = 0; q < 2; q++) {
        const int b = (chunk + q) & 1;
        if (!issued[b]) continue;
        const bool ok = mbar_wait(smem_u32(&mbar[b]), phase[b], failed ? kTcWaitLimit : wait_limit);
        if (__syncthreads_or(ok ? 0 : 1)) failed = true;
        phase[b] ^= 1u;
    }
    tc_fence_after();
    if (failed) {
        if (tid == 0) atomicExch(&g_mlp_tc_status, 1);
    } else {
        const uint32_t trow = tmem + ((uint32_t)(32 * warp) << 16);
        const int row = m0 + tid;
        const bool vec = ((ldc & 3) == 0) && (((uintptr_t)C & 15) == 0);
#pragma unroll 1
        for (int c0 = 0; c0 < NT; c0 += 32) {
            uint32_t v[32];
            tmem_ld32(trow + c0, v);
            tmem_wait_ld();
            if (row >= M) continue;
            const int col = n0 + c0;
            float x[32];
#pragma unroll
            for (int j = 0; j < 32; j++) x[j] = __uint_as_float(v[j]);
            if (accumulate) {
#pragma unroll
                for (int j = 0; j < 32; j++) atomicAdd(&C[(size_t)row * ldc + col + j], x[j]);
                continue;
            }
#pragma unroll
            for (int j = 0; j < 32; j++) {
                if (bias) x[j] += bias[col + j];
                if (relu) x[j] = fmaxf(x[j], 0.f);
            }
            if (C) {
                float *dst = C + (size_t)row * ldc + col;
                if (vec) {
#pragma unroll
                    for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4 *>(dst + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) dst[j] = x[j];
                }
            }
            if (Cb) {
#pragma unroll
                for (int j = 0; j < 32; j++) Cb[(size_t)row * ldcb + col + j] = __float2bfloat16_rn(x[j]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(NT) : "memory");
}

// C[r][c] = ((C[r][c] + P_0[r][c]) + P_1[r][c]) + ...: the split-K slices in slice order
__global__ void k_splitk_reduce(int M, int N, int splits, const float *__restrict__ ws, float *C, int ldc) {
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t MN = (size_t)M * N;
    if (e >= MN) return;
    const int r = (int)(e / N), c = (int)(e - (size_t)r * N);
    float x = C[(size_t)r * ldc + c];
    for (int z = 0; z < splits; z++) x += ws[z * MN + e];
    C[(size_t)r * ldc + c] = x;
}


// ------------------------------------------------------------------------------------------
// Fused training step on tcgen05: loss, every weight gradient and every bias gradient of the 4-layer
// MLP in one pass over the rows (k_train), then one reduction over the CTAs (k_train_reduce).
//
// A persistent grid of at most one CTA per SM keeps the bf16 weights in shared memory and takes
// 128-row tiles t = b, b + G, ...; a tile's activations and dZ never leave the SM, and the weight
// gradients accumulate in tensor memory over all tiles of the CTA.  Every matrix (rows x columns,
// column-contiguous in global memory) is stored once, in the canonical no-swizzle layout, and serves
// each product it enters through the descriptor's major-ness:
//   forward      D[r][n]  = a[r][k]  W[k][n]     A K-major,  B MN-major
//   data grad    D[r][k]  = dZ[r][n] W[k][n]     A K-major,  B K-major
//   weight grad  D[n][k] += dZ[r][n] a[r][k]     A MN-major, B MN-major
// dZ of a layer replaces that layer's activations in place once their products are done.  The
// rounding points are those of the layer-by-layer chain (bf16 inputs, weights, activations and dZ;
// fp32 accumulation, bias, loss and bias gradients), and the K=16 steps of the forward and data
// products run in its order, so the dZ are its bits; the row sums of the gradients are taken per CTA
// and then in CTA order, the same on every run.
// Tensor memory: D 0..127, gW1 128..255, gW2 256..383, gW0 384..447, gW3 448..463, Y 464..479.
// Bound: a tile's 10 products, seven of which wait for the one before and its epilogue: about 9.3 us a tile
// with one tile in flight (131,072 rows take seven per CTA), the tensor pipe busy a fifth of the time; 16 warps
// share every epilogue (32 columns of one row per thread) to keep that half of the chain short.  Measured with
// k_adam (loss_and_grad + adam, per step): 16,384 rows 2136 us (layer by layer, about 45 launches) -> 34.2
// us; 131,072 rows 4934 -> 90.3 us.
// ------------------------------------------------------------------------------------------
constexpr int kTrThreads = 512;
constexpr int kTrW0 = 0;                                  // [64 k][128 n]
constexpr int kTrW1 = kTrW0 + 64 * 128 * 2;               // [128 k][128 n]
constexpr int kTrW2 = kTrW1 + 128 * 128 * 2;
constexpr int kTrW3 = kTrW2 + 128 * 128 * 2;              // [128 k][16 n], column 0 real
constexpr int kTrX = kTrW3 + 128 * 16 * 2;                // two [128 r][64 k] tiles
constexpr int kTrXBytes = 128 * 64 * 2;
constexpr int kTrAct = kTrX + 2 * kTrXBytes;              // a1, a2, a3 (then dZ0, dZ1, dZ2): [128 r][128]
constexpr int kTrActBytes = 128 * 128 * 2;
constexpr int kTrDY = kTrAct + 3 * kTrActBytes;           // [128 r][16], column 0 real
constexpr int kTrBias = kTrDY + 128 * 16 * 2;             // b0 b1 b2 (3 x 128 floats), W3 column 0, dY (bf16 values)
constexpr int kTrMisc = kTrBias + 5 * 128 * 4;            // three mbarriers, TMEM address, b3
constexpr int kTrSmem = kTrMisc + 3 * 8 + 8;
constexpr int kTrCols = 512;
constexpr uint32_t kTrGW1 = 128, kTrGW2 = 256, kTrGW0 = 384, kTrGW3 = 448, kTrY = 464;
// one CTA's partial sums in the workspace (floats)
constexpr int kTrPW0 = 0, kTrPW1 = kTrPW0 + 64 * 128, kTrPW2 = kTrPW1 + 128 * 128, kTrPW3 = kTrPW2 + 128 * 128;
constexpr int kTrPb = kTrPW3 + 128;                       // gb0 gb1 gb2, then gb3[0] and the loss
constexpr int kTrPart = kTrPb + 3 * 128 + 2;

// rows [0, rows) of a global matrix (columns [0, C), C % 8 == 0) into the canonical layout of an
// R-row matrix, rows past `rows` zero; 8 consecutive threads write one 128-byte core matrix
__device__ __forceinline__ void tr_load(unsigned char *dst, int R, int C, const __nv_bfloat16 *__restrict__ src, int ld,
                                        int rows) {
    const int chunks = C / 8;
    for (int e = threadIdx.x; e < R * chunks; e += kTrThreads) {
        const int q = e >> 3, c = q % chunks, r = (q / chunks) * 8 + (e & 7);
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (r < rows) v = *reinterpret_cast<const uint4 *>(src + (size_t)r * ld + c * 8);
        *reinterpret_cast<uint4 *>(dst + canon_off(r, c * 8, R)) = v;
    }
}

// one product of `steps` K=16 instructions; a and b are matrices of ra and rb rows in the canonical
// layout, taken K-major (K = columns) or MN-major (K = rows)
template <bool AMn, bool BMn>
__device__ __forceinline__ void tr_mma(uint32_t d, uint32_t a, int ra, uint32_t b, int rb, int N, int steps, bool acc) {
    const uint32_t idesc = umma_idesc_bf16_f32(128, N) | (AMn ? 1u << 15 : 0u) | (BMn ? 1u << 16 : 0u);
    const uint32_t pa = ra * 16, pb = rb * 16;            // byte distance of 8-column groups
    for (int s = 0; s < steps; s++) {
        const uint64_t ad = AMn ? umma_smem_desc(a + s * 256, 128, pa) : umma_smem_desc(a + s * 2 * pa, pa, 128);
        const uint64_t bd = BMn ? umma_smem_desc(b + s * 256, 128, pb) : umma_smem_desc(b + s * 2 * pb, pb, 128);
        umma_bf16(d, ad, bd, idesc, (acc || s > 0) ? 1u : 0u);
    }
}

// sums of v[0..31] over the warp's 32 lanes by halving exchanges: lane l returns the sum of v[l]
__device__ __forceinline__ float tr_colsum(float (&v)[32], int lane) {
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
        const bool up = lane & h;
#pragma unroll
        for (int j = 0; j < h; j++) {
            const float send = up ? v[j] : v[j + h], keep = up ? v[j + h] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    return v[0];
}

// hidden layer epilogue of row r, columns c0..c0+31: bias, ReLU, bf16 into the activation buffer
__device__ __forceinline__ void tr_hidden(uint32_t taddr, const float *bias, unsigned char *act, int r, int c0) {
    uint32_t v[32];
    tmem_ld32(taddr, v);
    tmem_wait_ld();
#pragma unroll
    for (int q = 0; q < 4; q++) {
        uint4 u;
        uint32_t *w = reinterpret_cast<uint32_t *>(&u);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int c = 8 * q + 2 * j;
            w[j] = pack_bf16x2(fmaxf(__uint_as_float(v[c]) + bias[c0 + c], 0.f),
                               fmaxf(__uint_as_float(v[c + 1]) + bias[c0 + c + 1], 0.f));
        }
        *reinterpret_cast<uint4 *>(act + canon_off(r, c0 + 8 * q, 128)) = u;
    }
}

__device__ __forceinline__ float bf16_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// dZ = dA where the activation is positive: fp32 values stay in v (for the bias gradient), their
// bf16 roundings come back packed
__device__ __forceinline__ void tr_mask(float (&v)[32], const unsigned char *act, int r, int c0, uint4 (&u)[4]) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint4 a = *reinterpret_cast<const uint4 *>(act + canon_off(r, c0 + 8 * q, 128));
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
        uint32_t *w = reinterpret_cast<uint32_t *>(&u[q]);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int c = 8 * q + 2 * j;
            v[c] = bf16_lo(aw[j]) > 0.f ? v[c] : 0.f;
            v[c + 1] = bf16_hi(aw[j]) > 0.f ? v[c + 1] : 0.f;
            w[j] = pack_bf16x2(v[c], v[c + 1]);
        }
    }
}
__device__ __forceinline__ void tr_put(unsigned char *act, int r, int c0, const uint4 (&u)[4]) {
#pragma unroll
    for (int q = 0; q < 4; q++) *reinterpret_cast<uint4 *>(act + canon_off(r, c0 + 8 * q, 128)) = u[q];
}

struct TrainArgs {
    const __nv_bfloat16 *X, *W[4];
    const float *t, *b[4];
    int rows, valid;
    float *ws;
};

__global__ void __launch_bounds__(kTrThreads, 1) k_train(TrainArgs a, int wait_limit) {
    extern __shared__ __align__(1024) unsigned char sm[];
    float *sbias = reinterpret_cast<float *>(sm + kTrBias), *sw3 = sbias + 3 * 128, *sdy = sw3 + 128;
    uint64_t *mbar = reinterpret_cast<uint64_t *>(sm + kTrMisc);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + 3);
    float *sb3 = reinterpret_cast<float *>(tslot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, G = gridDim.x;
    const int ntiles = (a.rows + 127) / 128;
    // ---- weights, biases and the first tile into shared memory
    tr_load(sm + kTrW0, 64, 128, a.W[0], 128, 64);
    tr_load(sm + kTrW1, 128, 128, a.W[1], 128, 128);
    tr_load(sm + kTrW2, 128, 128, a.W[2], 128, 128);
    tr_load(sm + kTrW3, 128, 16, a.W[3], 64, 128);
    tr_load(sm + kTrX, 128, 64, a.X + (size_t)blockIdx.x * 128 * 64, 64, a.rows - (int)blockIdx.x * 128);
    for (int e = tid; e < 128 * 16 * 2 / 16; e += kTrThreads) reinterpret_cast<uint4 *>(sm + kTrDY)[e] = make_uint4(0u, 0u, 0u, 0u);
    if (tid < 128) {
        for (int l = 0; l < 3; l++) sbias[l * 128 + tid] = a.b[l][tid];
        sw3[tid] = __bfloat162float(a.W[3][(size_t)tid * 64]);
    }
    if (tid == 0) {
        *sb3 = a.b[3][0];
        for (int q = 0; q < 3; q++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(mbar + q)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(tslot)), "r"(kTrCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot, sb = smem_u32(sm), m0 = smem_u32(mbar), m1 = smem_u32(mbar + 1);
    const int q = warp & 3, cg = warp >> 2;              // TMEM lanes 32q.., columns 32cg..
    const int r = 32 * q + lane, c0 = 32 * cg;           // this thread's row and first column
    const uint32_t trow = tmem + ((uint32_t)(32 * q) << 16);
    unsigned char *act[3] = {sm + kTrAct, sm + kTrAct + kTrActBytes, sm + kTrAct + 2 * kTrActBytes};
    const uint32_t sact[3] = {sb + kTrAct, sb + kTrAct + kTrActBytes, sb + kTrAct + 2 * kTrActBytes};
    const uint32_t sw[3] = {sb + kTrW0, sb + kTrW1, sb + kTrW2};
    uint32_t p0 = 0, p1 = 0;                             // phases of the two mbarriers
    float gb[3] = {0.f, 0.f, 0.f}, gb3 = 0.f, loss = 0.f;
    bool fail = false;
    // a bounded wait for a commit; one that runs out ends the tile loop at the next block barrier
    auto wait = [&](uint32_t mb, uint32_t &ph) {
        if (!mbar_wait(mb, ph, wait_limit)) fail = true;
        ph ^= 1u;
        tc_fence_after();
    };
    // shared-memory operands and tensor-memory reads of every thread are done: the next product may
    // start; false, for every thread alike, when a thread's wait ran out
    auto publish = [&]() -> bool {
        fence_async_smem();
        tc_fence_before();
        const bool bad = __syncthreads_or(fail);
        tc_fence_after();
        return !bad;
    };
    const bool issuer = tid == 0;
    bool ok = true;
    int it = 0;
    for (int t = blockIdx.x; t < ntiles; t += G, it++) {
        const bool more = it > 0;                        // gradients accumulate after the first tile
        const uint32_t sx = sb + kTrX + (it & 1) * kTrXBytes;
        // the next tile's rows: two 16-byte chunks per thread, stored below into the other buffer
        uint4 xn[2];
        const int tn = t + G;
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int i = tid + e * kTrThreads, c = (i >> 3) & 7, rr = (i >> 6) * 8 + (i & 7);
            xn[e] = make_uint4(0u, 0u, 0u, 0u);
            if (tn < ntiles && tn * 128 + rr < a.rows)
                xn[e] = *reinterpret_cast<const uint4 *>(a.X + ((size_t)tn * 128 + rr) * 64 + c * 8);
        }
        const int row = t * 128 + r;
        const float target = (cg == 0 && row < a.valid && row < a.rows) ? a.t[row] : 0.f;
        // ---- forward
        if (issuer) { tr_mma<false, true>(tmem, sx, 128, sw[0], 64, 128, 4, false); umma_commit(m0); }
        wait(m0, p0);
        if (tn < ntiles)                                 // the other buffer's last reader (gW0 of the previous tile) is done
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int i = tid + e * kTrThreads, c = (i >> 3) & 7, rr = (i >> 6) * 8 + (i & 7);
                *reinterpret_cast<uint4 *>(sm + kTrX + ((it + 1) & 1) * kTrXBytes + canon_off(rr, c * 8, 128)) = xn[e];
            }
        tr_hidden(trow + c0, sbias, act[0], r, c0);
        if (!(ok = publish())) break;
#pragma unroll
        for (int l = 1; l < 3; l++) {
            if (issuer) { tr_mma<false, true>(tmem, sact[l - 1], 128, sw[l], 128, 128, 8, false); umma_commit(m0); }
            wait(m0, p0);
            tr_hidden(trow + c0, sbias + 128 * l, act[l], r, c0);
            if (!(ok = publish())) break;
        }
        if (!ok) break;
        // ---- output layer, loss and dY
        if (issuer) { tr_mma<false, true>(tmem + kTrY, sact[2], 128, sb + kTrW3, 128, 16, 8, false); umma_commit(m0); }
        wait(m0, p0);
        if (cg == 0) {
            uint32_t yv;
            tmem_ld1(trow + kTrY, yv);
            tmem_wait_ld();
            const float e = (row < a.valid && row < a.rows) ? (__uint_as_float(yv) + *sb3) - target : 0.f;
            const float dy = 2.f * e / (float)a.valid;
            const __nv_bfloat16 dyb = __float2bfloat16_rn(row < a.rows ? dy : 0.f);
            loss += e * e;
            gb3 += row < a.rows ? dy : 0.f;
            *reinterpret_cast<__nv_bfloat16 *>(sm + kTrDY + canon_off(r, 0, 128)) = dyb;
            sdy[r] = __bfloat162float(dyb);
        }
        if (!(ok = publish())) break;
        // ---- gW3 += a3^T dY;  dZ2 = dY W3^T where a3 > 0 (one exact product per element)
        if (issuer) { tr_mma<true, true>(tmem + kTrGW3, sact[2], 128, sb + kTrDY, 128, 16, 8, more); umma_commit(m0); }
        float v[32];
        uint4 u[4];
        {
            const float dy = sdy[r];
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = dy * sw3[c0 + j];
            tr_mask(v, act[2], r, c0, u);
            gb[2] += tr_colsum(v, lane);
        }
        wait(m0, p0);
        tr_put(act[2], r, c0, u);
        if (!(ok = publish())) break;
        // ---- layers 2 and 1: dA = dZ W^T, gW += dZ^T a, dZ of the layer below in place of its activations
#pragma unroll
        for (int l = 2; l >= 1; l--) {
            if (issuer) {
                tr_mma<false, false>(tmem, sact[l], 128, sw[l], 128, 128, 8, false);
                umma_commit(m0);
                tr_mma<true, true>(tmem + (l == 2 ? kTrGW2 : kTrGW1), sact[l], 128, sact[l - 1], 128, 128, 8, more);
                umma_commit(m1);
            }
            wait(m0, p0);
            uint32_t d[32];
            tmem_ld32(trow + c0, d);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = __uint_as_float(d[j]);
            tr_mask(v, act[l - 1], r, c0, u);
            gb[l - 1] += tr_colsum(v, lane);
            wait(m1, p1);                                // the weight gradient has read the activations
            tr_put(act[l - 1], r, c0, u);
            if (!(ok = publish())) break;
        }
        if (!ok) break;
        // ---- gW0 += dZ0^T X; completes before the next tile's first product, which is issued after it
        if (issuer) tr_mma<true, true>(tmem + kTrGW0, sact[0], 128, sx, 128, 64, 8, more);
    }
    // every product issued so far completes (one more commit tracks them all, waited for with the full
    // bound also after a failure) before the sums are read and the columns released
    if (issuer) umma_commit(smem_u32(mbar + 2));
    fail = !mbar_wait(smem_u32(mbar + 2), 0u, kTcWaitLimit) || !ok;
    const bool failed = __syncthreads_or(fail);
    tc_fence_after();
    float *out = a.ws + (size_t)blockIdx.x * kTrPart;
    if (failed) {
        // no sums: NaN, so that the loss and every gradient show it whether or not the status is read
        for (int e = tid; e < kTrPart; e += kTrThreads) out[e] = __int_as_float(0x7fc00000);
        if (tid == 0) atomicExch(&g_mlp_tc_status, 1);
    } else {
        uint32_t d[32];
        // D lanes are n, columns k: consecutive lanes store consecutive n of one k
#pragma unroll
        for (int l = 1; l < 3; l++) {
            tmem_ld32(trow + (l == 1 ? kTrGW1 : kTrGW2) + c0, d);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; j++) out[(l == 1 ? kTrPW1 : kTrPW2) + (c0 + j) * 128 + r] = __uint_as_float(d[j]);
        }
        if (cg < 2) {
            tmem_ld32(trow + kTrGW0 + c0, d);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; j++) out[kTrPW0 + (c0 + j) * 128 + r] = __uint_as_float(d[j]);
        } else if (cg == 2) {
            uint32_t g;
            tmem_ld1(trow + kTrGW3, g);
            tmem_wait_ld();
            out[kTrPW3 + r] = __uint_as_float(g);
        }
        // bias gradients: thread (q, cg, lane) holds column c0 + lane over rows 32q..; the four row
        // quarters are added in order (the activation buffers are free now)
        float *sg = reinterpret_cast<float *>(sm + kTrAct);
#pragma unroll
        for (int l = 0; l < 3; l++) sg[(l * 4 + q) * 128 + c0 + lane] = gb[l];
        if (cg == 0) {
            for (int o = 16; o > 0; o >>= 1) {
                gb3 += __shfl_down_sync(0xffffffffu, gb3, o);
                loss += __shfl_down_sync(0xffffffffu, loss, o);
            }
            if (lane == 0) { sg[12 * 128 + q] = gb3; sg[12 * 128 + 4 + q] = loss; }
        }
        __syncthreads();
        if (tid < 3 * 128) {
            const float *p = sg + (tid >> 7) * 4 * 128 + (tid & 127);
            out[kTrPb + tid] = ((p[0] + p[128]) + p[256]) + p[384];
        } else if (tid < 3 * 128 + 2) {
            const float *p = sg + 12 * 128 + 4 * (tid - 3 * 128);
            out[kTrPb + tid] = ((p[0] + p[1]) + p[2]) + p[3];
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(kTrCols) : "memory");
}

// Gradients and loss from the CTAs' partial sums.  32 consecutive outputs per block, 8 slices of the
// CTAs each: a slice adds its partials in CTA order, the slices are added in order.
struct TrainOut {
    float *gW[4], *gb[4], *loss;
    int parts, valid;
};
constexpr int kTrOutW3 = kTrPW3, kTrOutB = kTrOutW3 + 128 * 64, kTrOutN = kTrOutB + 3 * 128 + 64 + 1;
constexpr int kTrSlices = 8;
__global__ void __launch_bounds__(32 * kTrSlices) k_train_reduce(const float *__restrict__ ws, TrainOut o) {
    const int e = blockIdx.x * 32 + (threadIdx.x & 31), sl = threadIdx.x >> 5;
    // output e: gW0 gW1 gW2 as in the partials, gW3 [128][64] (column 0 real), gb0 gb1 gb2, gb3 [64], loss
    int src = -1;
    if (e < kTrOutW3) src = e;
    else if (e < kTrOutB) src = ((e - kTrOutW3) & 63) == 0 ? kTrPW3 + ((e - kTrOutW3) >> 6) : -1;
    else if (e < kTrOutB + 3 * 128 + 1) src = kTrPb + (e - kTrOutB);
    else if (e == kTrOutN - 1) src = kTrPb + 3 * 128 + 1;
    const int per = (o.parts + kTrSlices - 1) / kTrSlices, p0 = sl * per, p1 = min(o.parts, p0 + per);
    float x = 0.f;
    if (src >= 0)
#pragma unroll 8
        for (int p = p0; p < p1; p++) x += ws[(size_t)p * kTrPart + src];
    __shared__ float s[kTrSlices][32];
    s[sl][threadIdx.x & 31] = x;
    __syncthreads();
    if (sl != 0 || e >= kTrOutN) return;
    for (int k = 1; k < kTrSlices; k++) x += s[k][threadIdx.x];
    if (e < kTrPW1) o.gW[0][e - kTrPW0] = x;
    else if (e < kTrPW2) o.gW[1][e - kTrPW1] = x;
    else if (e < kTrOutW3) o.gW[2][e - kTrPW2] = x;
    else if (e < kTrOutB) o.gW[3][e - kTrOutW3] = x;
    else if (e < kTrOutB + 3 * 128) o.gb[(e - kTrOutB) >> 7][(e - kTrOutB) & 127] = x;
    else if (e < kTrOutN - 1) o.gb[3][e - kTrOutB - 3 * 128] = x;
    else *o.loss = x / (float)o.valid;
}

}  // namespace

extern "C" {

const char *cmf_emu_last_error(void) { return g_emu_err.c_str(); }

int cmf_emu_gemm(int M, int N, int K, const void *A, int lda, int transA, const void *B, int ldb, int transB, float *C,
                 int ldc, void *Cb, int ldcb, const float *bias, int relu, int accumulate, int ksplit, void *stream) {
    if (M % TM || N % TN || K % TK || M <= 0 || N <= 0 || K <= 0)
        return emu_err(CMF_E_ARG, "cmf_emu_gemm: M,N must be multiples of 64 and K of 32");
    if ((lda % 8) || (ldb % 8) || ((uintptr_t)A & 15) || ((uintptr_t)B & 15))
        return emu_err(CMF_E_ARG, "cmf_emu_gemm: lda, ldb must be multiples of 8 and A, B 16-byte aligned");
    int dev = 0, major = 0;
    EMU_TRY(cudaGetDevice(&dev));
    EMU_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    if (major != 10) return emu_err(CMF_E_NO_DEVICE, "cmf_emu_gemm: needs an sm_100 device");
    if (ksplit < 1) ksplit = 1;
    const int kps = ((K / ksplit + kGK - 1) / kGK) * kGK;   // whole chunks per split
    const int splits = (K + kps - 1) / kps;
    if (splits > 1 && !accumulate) return emu_err(CMF_E_ARG, "cmf_emu_gemm: split-K needs accumulate=1");
    cudaStream_t st = (cudaStream_t)stream;
    if (N % 128 == 0) {
        EMU_TRY(cudaFuncSetAttribute(k_gemm_tc<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGSmem));
        dim3 grid((M + 127) / 128, N / 128, splits);
        k_gemm_tc<128><<<grid, kGThreads, kGSmem, st>>>(M, N, K, (const __nv_bfloat16 *)A, lda, transA, (const __nv_bfloat16 *)B,
                                                       ldb, transB, C, ldc, (__nv_bfloat16 *)Cb, ldcb, bias, relu, accumulate,
                                                       kps, g_tc_wait_limit, (size_t)0);
    } else {
        EMU_TRY(cudaFuncSetAttribute(k_gemm_tc<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGSmem));
        dim3 grid((M + 127) / 128, N / 64, splits);
        k_gemm_tc<64><<<grid, kGThreads, kGSmem, st>>>(M, N, K, (const __nv_bfloat16 *)A, lda, transA, (const __nv_bfloat16 *)B,
                                                      ldb, transB, C, ldc, (__nv_bfloat16 *)Cb, ldcb, bias, relu, accumulate,
                                                      kps, g_tc_wait_limit, (size_t)0);
    }
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

size_t cmf_emu_gemm_splitk_ws_floats(int M, int N, int K, int ksplit) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    if (ksplit < 1) ksplit = 1;
    const int kps = ((K / ksplit + kGK - 1) / kGK) * kGK;
    return (size_t)((K + kps - 1) / kps) * (size_t)M * (size_t)N;
}

int cmf_emu_gemm_splitk(int M, int N, int K, const void *A, int lda, int transA, const void *B, int ldb, int transB,
                        float *C, int ldc, int ksplit, float *workspace, size_t workspace_floats, void *stream) {
    if (M % TM || N % TN || K % TK || M <= 0 || N <= 0 || K <= 0)
        return emu_err(CMF_E_ARG, "cmf_emu_gemm_splitk: M,N must be multiples of 64 and K of 32");
    if ((lda % 8) || (ldb % 8) || ((uintptr_t)A & 15) || ((uintptr_t)B & 15))
        return emu_err(CMF_E_ARG, "cmf_emu_gemm_splitk: lda, ldb must be multiples of 8 and A, B 16-byte aligned");
    if (!C || !workspace) return emu_err(CMF_E_ARG, "cmf_emu_gemm_splitk: C and workspace are required");
    int dev = 0, major = 0;
    EMU_TRY(cudaGetDevice(&dev));
    EMU_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    if (major != 10) return emu_err(CMF_E_NO_DEVICE, "cmf_emu_gemm_splitk: needs an sm_100 device");
    if (ksplit < 1) ksplit = 1;
    const int kps = ((K / ksplit + kGK - 1) / kGK) * kGK;
    const int splits = (K + kps - 1) / kps;
    const size_t MN = (size_t)M * N;
    if (workspace_floats < (size_t)splits * MN)
        return emu_err(CMF_E_ARG, "cmf_emu_gemm_splitk: workspace smaller than cmf_emu_gemm_splitk_ws_floats()");
    cudaStream_t st = (cudaStream_t)stream;
    if (N % 128 == 0) {
        EMU_TRY(cudaFuncSetAttribute(k_gemm_tc<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGSmem));
        dim3 grid((M + 127) / 128, N / 128, splits);
        k_gemm_tc<128><<<grid, kGThreads, kGSmem, st>>>(M, N, K, (const __nv_bfloat16 *)A, lda, transA, (const __nv_bfloat16 *)B,
                                                       ldb, transB, workspace, N, nullptr, 0, nullptr, 0, 0, kps,
                                                       g_tc_wait_limit, MN);
    } else {
        EMU_TRY(cudaFuncSetAttribute(k_gemm_tc<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGSmem));
        dim3 grid((M + 127) / 128, N / 64, splits);
        k_gemm_tc<64><<<grid, kGThreads, kGSmem, st>>>(M, N, K, (const __nv_bfloat16 *)A, lda, transA, (const __nv_bfloat16 *)B,
                                                      ldb, transB, workspace, N, nullptr, 0, nullptr, 0, 0, kps,
                                                      g_tc_wait_limit, MN);
    }
    EMU_TRY(cudaGetLastError());
    k_splitk_reduce<<<(unsigned)((MN + 255) / 256), 256, 0, st>>>(M, N, splits, workspace, C, ldc);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

int cmf_emu_gemm_mma(int M, int N, int K, const void *A, int lda, int transA, const void *B, int ldb, int transB, float *C,
                     int ldc, void *Cb, int ldcb, const float *bias, int relu, int accumulate, int ksplit, void *stream) {
    if (M % TM || N % TN || K % TK || M <= 0 || N <= 0 || K <= 0)
        return emu_err(CMF_E_ARG, "cmf_emu_gemm_mma: M,N must be multiples of 64 and K of 32");
    if (ksplit < 1) ksplit = 1;
    int kps = ((K / ksplit + TK - 1) / TK) * TK;
    const int splits = (K + kps - 1) / kps;
    if (splits > 1 && !accumulate) return emu_err(CMF_E_ARG, "cmf_emu_gemm: split-K needs accumulate=1");
    dim3 grid(M / TM, N / TN, splits);
    k_gemm<<<grid, 128, 0, (cudaStream_t)stream>>>(M, N, K, (const __nv_bfloat16 *)A, lda, transA, (const __nv_bfloat16 *)B,
                                                  ldb, transB, C, ldc, (__nv_bfloat16 *)Cb, ldcb, bias, relu, accumulate, kps);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

int cmf_emu_relu_bwd(int n, const float *dA, const void *act, void *dZ, float *dZf, void *stream) {
    k_relu_bwd<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(n, dA, (const __nv_bfloat16 *)act, (__nv_bfloat16 *)dZ, dZf);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

int cmf_emu_mse_grad(int rows, int valid, int ldy, const float *Y, const float *t, float *dY, void *dYb, float *loss_part,
                     void *stream) {
    k_mse_grad<<<(rows + 255) / 256, 256, 0, (cudaStream_t)stream>>>(rows, valid, ldy, Y, t, dY, (__nv_bfloat16 *)dYb, loss_part);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

int cmf_emu_colsum(int rows, int cols, const float *X, float *out, void *stream) {
    k_colsum<<<cols, 256, 0, (cudaStream_t)stream>>>(rows, cols, X, out);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

int cmf_emu_adam_set(int count, const int32_t *n, float *const *w, void *const *wb, const float *const *grad, float *const *m,
                     float *const *v, const float *wd, float lr, float b1, float b2, float eps, int step, void *stream) {
    if (count < 1 || count > kAdamMax || !n || !w || !wb || !grad || !m || !v || !wd)
        return emu_err(CMF_E_ARG, "cmf_emu_adam_set: 1 to 8 tensors");
    AdamSet a{};
    int most = 0;
    for (int k = 0; k < count; k++) {
        a.n[k] = n[k]; a.w[k] = w[k]; a.wb[k] = (__nv_bfloat16 *)wb[k]; a.grad[k] = grad[k];
        a.m[k] = m[k]; a.v[k] = v[k]; a.wd[k] = wd[k];
        if (n[k] > most) most = n[k];
    }
    const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
    k_adam<<<dim3((most + 255) / 256, count), 256, 0, (cudaStream_t)stream>>>(a, lr, b1, b2, eps, bc1, bc2);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

int cmf_emu_adam(int n, float *w, void *wb, const float *grad, float *m, float *v, float lr, float b1, float b2, float eps,
                 int step, float wd, void *stream) {
    const int32_t nn = n;
    return cmf_emu_adam_set(1, &nn, &w, &wb, &grad, &m, &v, &wd, lr, b1, b2, eps, step, stream);
}

size_t cmf_emu_loss_grad_ws_floats(int rows) {
    if (rows <= 0) return 0;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    const int ntiles = (rows + 127) / 128;
    return (size_t)(ntiles < sms ? ntiles : sms) * kTrPart;
}

int cmf_emu_loss_grad(int rows, int valid, const void *X, const float *t, const void *const *W, const float *const *b,
                      float *const *gW, float *const *gb, float *loss, float *workspace, size_t workspace_floats,
                      void *stream) {
    if (rows <= 0 || rows % 64 || !X || !t || !W || !b || !gW || !gb || !loss || !workspace)
        return emu_err(CMF_E_ARG, "cmf_emu_loss_grad: null argument, or rows not a multiple of 64");
    TrainArgs a{};
    TrainOut o{};
    uintptr_t align = (uintptr_t)X;
    for (int l = 0; l < 4; l++) {
        if (!W[l] || !b[l] || !gW[l] || !gb[l]) return emu_err(CMF_E_ARG, "cmf_emu_loss_grad: null parameter tensor");
        a.W[l] = (const __nv_bfloat16 *)W[l];
        a.b[l] = b[l];
        o.gW[l] = gW[l];
        o.gb[l] = gb[l];
        align |= (uintptr_t)W[l];
    }
    if (align & 15) return emu_err(CMF_E_ARG, "cmf_emu_loss_grad: X and the weights must be 16-byte aligned");
    int dev = 0, major = 0, sms = 0;
    EMU_TRY(cudaGetDevice(&dev));
    EMU_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    if (major != 10) return emu_err(CMF_E_NO_DEVICE, "cmf_emu_loss_grad: needs an sm_100 device");
    EMU_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int ntiles = (rows + 127) / 128, grid = ntiles < sms ? ntiles : sms;
    if (workspace_floats < (size_t)grid * kTrPart)
        return emu_err(CMF_E_ARG, "cmf_emu_loss_grad: workspace smaller than cmf_emu_loss_grad_ws_floats()");
    a.X = (const __nv_bfloat16 *)X;
    a.t = t;
    a.rows = rows;
    a.valid = valid;
    a.ws = workspace;
    o.loss = loss;
    o.parts = grid;
    o.valid = valid;
    EMU_TRY(cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrSmem));
    k_train<<<grid, kTrThreads, kTrSmem, (cudaStream_t)stream>>>(a, g_tc_wait_limit);
    EMU_TRY(cudaGetLastError());
    k_train_reduce<<<(kTrOutN + 31) / 32, 32 * kTrSlices, 0, (cudaStream_t)stream>>>(workspace, o);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

size_t cmf_emu_mlp_pack_bytes(void) { return (size_t)kMlpPackWords * sizeof(uint2); }

int cmf_emu_mlp_pack(const void *W0, const void *W1, const void *W2, const void *W3, int ldw3, void *pack, void *stream) {
    if (!W0 || !W1 || !W2 || !W3 || !pack || ldw3 < 8) return emu_err(CMF_E_ARG, "cmf_emu_mlp_pack: bad arguments");
    k_mlp_pack<<<(kMlpPackWords + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16 *)W0, (const __nv_bfloat16 *)W1, (const __nv_bfloat16 *)W2, (const __nv_bfloat16 *)W3, ldw3,
        (uint2 *)pack);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

int cmf_emu_mlp_fused(const void *X, int ldx, int rows, const void *pack, const float *b0, const float *b1, const float *b2,
                      const float *b3, float *y, void *stream) {
    if (!X || !pack || !b0 || !b1 || !b2 || !b3 || !y || ldx < 32 || (ldx & 1) || rows < 0 || rows % 16)
        return emu_err(CMF_E_ARG, "cmf_emu_mlp_fused: bad arguments (ldx >= 32 and even, rows % 16 == 0)");
    if (((uintptr_t)X & 3) || ((uintptr_t)pack & 7)) return emu_err(CMF_E_ARG, "cmf_emu_mlp_fused: misaligned X or pack");
    if (rows == 0) return CMF_OK;
    int dev = 0, sms = 0;
    EMU_TRY(cudaGetDevice(&dev));
    EMU_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int smem = (int)cmf_emu_mlp_pack_bytes();
    EMU_TRY(cudaFuncSetAttribute(k_mlp_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const int ntiles = (rows + kMlpRowsPerCta - 1) / kMlpRowsPerCta;
    const int grid = ntiles < 2 * sms ? ntiles : 2 * sms;
    k_mlp_fused<<<grid, kMlpThreads, smem, (cudaStream_t)stream>>>((const __nv_bfloat16 *)X, ldx, rows, (const uint2 *)pack,
                                                                   b0, b1, b2, b3, y);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

size_t cmf_emu_mlp_tc_pack_bytes(void) { return (size_t)kTcWBytes; }

int cmf_emu_mlp_tc_pack(const void *W0, const void *W1, const void *W2, const void *W3, int ldw3, void *pack, void *stream) {
    if (!W0 || !W1 || !W2 || !W3 || !pack || ldw3 < 16 || ((uintptr_t)pack & 15))
        return emu_err(CMF_E_ARG, "cmf_emu_mlp_tc_pack: bad arguments (ldw3 >= 16, pack 16-byte aligned)");
    const int n = 128 * 64 + 2 * 128 * 128 + 16 * 128;
    k_mlp_tc_pack<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16 *)W0, (const __nv_bfloat16 *)W1, (const __nv_bfloat16 *)W2, (const __nv_bfloat16 *)W3, ldw3,
        (__nv_bfloat16 *)pack);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

int cmf_emu_mlp_tc(const void *X, int ldx, int rows, const void *pack, const float *b0, const float *b1, const float *b2,
                   const float *b3, float *y, void *stream) {
    if (!X || !pack || !b0 || !b1 || !b2 || !b3 || !y || ldx < 32 || (ldx % 8) || rows < 0)
        return emu_err(CMF_E_ARG, "cmf_emu_mlp_tc: bad arguments (ldx >= 32 and a multiple of 8)");
    if (((uintptr_t)X & 15) || ((uintptr_t)pack & 15)) return emu_err(CMF_E_ARG, "cmf_emu_mlp_tc: X and pack must be 16-byte aligned");
    if (rows == 0) return CMF_OK;
    int dev = 0, sms = 0, major = 0;
    EMU_TRY(cudaGetDevice(&dev));
    EMU_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    if (major != 10) return emu_err(CMF_E_NO_DEVICE, "cmf_emu_mlp_tc: needs an sm_100 device");
    EMU_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    EMU_TRY(cudaFuncSetAttribute(k_mlp_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem));
    const int ntiles = (rows + kTcRows - 1) / kTcRows;
    const int grid = ntiles < sms ? ntiles : sms;
    k_mlp_tc<<<grid, kTcThreads, kTcSmem, (cudaStream_t)stream>>>((const __nv_bfloat16 *)X, ldx, rows, (const uint4 *)pack,
                                                                  b0, b1, b2, b3, y, g_tc_wait_limit);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

int cmf_emu_mlp_tc_status(void) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_mlp_tc_status, sizeof v) != cudaSuccess) return emu_err(CMF_E_CUDA, "cmf_emu_mlp_tc_status: read failed");
    if (!v) return CMF_OK;
    const int zero = 0;                                       // clear on read: the next check starts clean
    if (cudaMemcpyToSymbol(g_mlp_tc_status, &zero, sizeof zero) != cudaSuccess)
        return emu_err(CMF_E_CUDA, "cmf_emu_mlp_tc_status: reset failed");
    return emu_err(CMF_E_CUDA, "cmf_emu_mlp_tc: an MMA completion wait ran out its bound (the kernel returned early)");
}

int cmf_emu_mlp_tc_set_wait_limit(int32_t limit) {
    g_tc_wait_limit = limit < 0 ? kTcWaitLimit : limit;
    return CMF_OK;
}

// Features of every member: X rows [M][rows_per_member][ldx] bf16 (columns 0..31 written);
// planes: fp32 [2 * (hops + 1)][M * N] scratch for the message passes.
int cmf_emu_features(const cmf_emu_net *net, const cmf_emu_member *mb, int nmembers, void *X, int ldx, int rows_per_member,
                     int hops, float *planes, void *stream) {
    if (!net || !mb || !X || !planes || hops < 0 || hops > 8 || ldx < 32 || (ldx % 8) || nmembers < 1 ||
        rows_per_member < net->nseqall || ((uintptr_t)X & 15) || !net->rivman)
        return emu_err(CMF_E_ARG, "cmf_emu_features: bad arguments (hops <= 8, ldx % 8 == 0, X 16-byte aligned)");
    EmuNet n{net->nseqall, net->nseqriv, net->next, net->up_ptr, net->up_idx, net->rivelv, net->elevtn, net->nxtdst,
             net->rivwth, net->rivhgt, net->rivlen, net->rivstomax, net->qref, net->rivman, net->pmanfld};
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 blocks((n.N + 255) / 256, nmembers);
    const size_t plane = (size_t)nmembers * n.N;
    auto pl = [&](int k) { return planes + (size_t)k * plane; };   // hop h: planes 2h+2 (outflow), 2h+3 (runoff)
    if (hops >= 1) k_emu_hop<true><<<blocks, 256, 0, st>>>(n, nullptr, nullptr, mb->qprev, mb->runoff, pl(2), pl(3));
    for (int h = 1; h < hops; h++)
        k_emu_hop<false><<<blocks, 256, 0, st>>>(n, pl(2 * h), pl(2 * h + 1), nullptr, nullptr, pl(2 * h + 2), pl(2 * h + 3));
    k_emu_assemble<<<blocks, 256, 0, st>>>(n, mb->rivsto, mb->fldsto, mb->levsto, mb->rivdph, mb->flddph, mb->fldfrc,
                                           mb->qprev, mb->runoff, planes, plane, hops, (__nv_bfloat16 *)X, ldx,
                                           rows_per_member);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

int cmf_emu_rollout(const cmf_emu_net *net, const cmf_emu_member *mb, int nmembers, const int *active_dev, const float *y,
                    int ldy, int rows_per_member, double dt, int residual, double *qout, void *stream) {
    if (!net || !mb || !y || !qout || !active_dev || nmembers < 1) return emu_err(CMF_E_ARG, "cmf_emu_rollout: null argument");
    EmuNet n{net->nseqall, net->nseqriv, net->next, net->up_ptr, net->up_idx, net->rivelv, net->elevtn, net->nxtdst,
             net->rivwth, net->rivhgt, net->rivlen, net->rivstomax, net->qref, net->rivman, net->pmanfld};
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 blocks((n.N + 255) / 256, nmembers);
    k_emu_rollout<<<blocks, 256, 0, st>>>(n, y, ldy, rows_per_member, active_dev, dt, residual, mb->runoff, mb->rivsto, mb->fldsto,
                                          mb->levsto, mb->qprev, qout);
    k_emu_update<<<blocks, 256, 0, st>>>(n, active_dev, dt, mb->runoff, qout, mb->rivsto, mb->fldsto, mb->levsto,
                                         mb->rivout_pre, mb->fldout_pre, mb->qprev);
    EMU_TRY(cudaGetLastError());
    return CMF_OK;
}

}  // extern "C"
