// Small multilayer perceptron for the learned variant picker: forward,
// backward and Adam training kernels with bf16 weights and activations and
// fp32 accumulation.
//
// Shape: in -> H -> H -> H -> out (3 hidden layers of width H, GELU after
// each hidden layer, exact erf form).  All dimensions are multiples of 16.
// GEMMs use warp-level tensor-core tiles (mma m16n8k16, bf16 in, fp32
// accumulate); at this model size (H = 256) the network is bound by latency,
// not by tensor throughput.
//
//   forward:  pre_l = act_{l-1} W_l^T + b_l (fp32), act_l = bf16(gelu(pre_l))
//   loss:     masked mean squared error of the output against targets
//   backward: d_pre = d_act * gelu'(pre) (rounded to bf16 for the GEMMs),
//             dW_l = d_pre^T act_{l-1}, db_l = column sums, d_act_{l-1} = d_pre W_l
//   update:   Adam on fp32 master weights, refreshed bf16 copies.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <memory>
#include <random>
#include <string>
#include <vector>

#include "../../include/bine_b200.h"

namespace {

using bf16 = __nv_bfloat16;

thread_local std::string g_mlp_err;

int mfail(int code, const std::string& m) {
    g_mlp_err = m;
    return code;
}

#define MLP_TRY(expr)                                                                         \
    do {                                                                                      \
        cudaError_t e_ = (expr);                                                              \
        if (e_ != cudaSuccess) return mfail(BINE_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
    } while (0)

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

// ------------------------------------------------- layered forward/backward
// Every GEMM of the layered path is a few hundred rows and columns: bound by
// the latency of its operand loads and of the launches between dependent
// stages, not by tensor throughput.  So a block owns one 32 x 32 tile (four
// warps of 16 x 16), requests its operands for 2 * kStageK steps of the
// reduction at once (cp.async, double-buffered beyond that), and what
// follows a GEMM runs in its epilogue on the accumulators: bias and GELU,
// loss and output gradient, GELU' of the backward pass, bias gradients (from
// the staged tiles).  One stage per dependent step remains: a prepare kernel,
// 4 forward, 4 backward (the weight gradient of a layer beside the next
// layer's input gradient).  Each accumulator adds its k-steps of 16 in
// ascending order.
//
// B200, 256 rows, 16 -> 256 -> 256 -> 256 -> 144, host call included, against
// one launch per GEMM (64 x 64 tiles, operands loaded step by step), bias,
// loss, GELU' and column sum, with the mask counted on the host: gradients
// 559 -> 124 us (about 60 of them the copy of 690 KB to the host and its
// fresh pages), training step 400 -> 73, forward 57 -> 22.
constexpr int kTile = 32;      // rows and columns of a block's tile
constexpr int kStageK = 128;   // reduction steps per buffer
constexpr int kGemmThreads = 128;
constexpr int kPitchK = kStageK + 8;  // operand stored [row][k]: 16-byte rows fall on distinct banks
constexpr int kPitchT = kTile + 8;    // operand stored [k][row]

struct GemmSmem {
    // One buffer holds a [kTile][kPitchK] or a [kStageK][kPitchT] tile.
    static constexpr int kElems = kStageK * kPitchT > kTile * kPitchK ? kStageK * kPitchT : kTile * kPitchK;
    __align__(128) bf16 a[2][kElems];
    __align__(128) bf16 b[2][kElems];
};

__device__ __forceinline__ void cp_async16(void* smem, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
                 : "memory");
}
template <bool TRANS>
__device__ __forceinline__ void ldmatrix_x4(uint32_t* r, const void* smem) {
    const uint32_t p = (uint32_t)__cvta_generic_to_shared(smem);
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(p)
                     : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(p)
                     : "memory");
}
__device__ __forceinline__ void mma_bf16_16816(float* d, const uint32_t* a, const uint32_t* b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Requests k-steps [k0, k0 + kn) of a tile's 32 rows from `row0` of an
// operand: stored [row][k] (ld elements per row), or [k][row] when T.  Rows
// from `rows` on are not requested (their results are not used); all
// dimensions are multiples of 16, so every request is 16 aligned bytes.
template <bool T>
__device__ __forceinline__ void gemm_request(bf16* smem, const bf16* __restrict__ g, int ld, int row0, int rows,
                                             int k0, int kn) {
    const int nr = min(kTile, rows - row0);
    if (!T) {
        const int per = kn / 8;  // 16-byte pieces per row
        for (int i = threadIdx.x; i < nr * per; i += kGemmThreads) {
            const int r = i / per, c = i - r * per;
            cp_async16(smem + r * kPitchK + c * 8, g + (size_t)(row0 + r) * ld + k0 + c * 8);
        }
    } else {
        const int per = nr / 8;
        for (int i = threadIdx.x; i < kn * per; i += kGemmThreads) {
            const int k = i / per, c = i - k * per;
            cp_async16(smem + k * kPitchT + c * 8, g + (size_t)(k0 + k) * ld + row0 + c * 8);
        }
    }
}

// acc (two 16 x 8 fragments of the warp's 16 x 16) = A[row0.., :] B[:, col0..]
// over K.  A is stored [M][K] (lda), or [K][M] when TA; B [N][K] (ldb), or
// [K][N] when TB.  `each(buffer, steps)` sees every staged A tile.
template <bool TA, bool TB, typename Each>
__device__ __forceinline__ void gemm_tile(GemmSmem& S, float (&acc)[2][4], const bf16* __restrict__ A, int lda,
                                          const bf16* __restrict__ B, int ldb, int row0, int col0, int M, int N,
                                          int K, const Each& each) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * 16;
    const bool active = row0 + wm < M && col0 + wn < N;
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[h][i] = 0.f;
    const int stages = (K + kStageK - 1) / kStageK;
    auto request = [&](int s) {
        if (s < stages) {
            const int k0 = s * kStageK, kn = min(kStageK, K - k0);
            gemm_request<TA>(S.a[s & 1], A, lda, row0, M, k0, kn);
            gemm_request<TB>(S.b[s & 1], B, ldb, col0, N, k0, kn);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    request(0);
    request(1);
    for (int s = 0; s < stages; s++) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const int kn = min(kStageK, K - s * kStageK);
        const bf16* sa = S.a[s & 1];
        const bf16* sb = S.b[s & 1];
        if (active) {
            // ldmatrix: lanes 8q .. 8q + 7 address the rows of matrix q.
            const int q = lane >> 3, r = lane & 7;
#pragma unroll 4
            for (int k = 0; k < kn; k += 16) {
                uint32_t a[4], b[4];
                if (!TA) ldmatrix_x4<false>(a, sa + (wm + (q & 1) * 8 + r) * kPitchK + k + (q >> 1) * 8);
                else ldmatrix_x4<true>(a, sa + (k + (q >> 1) * 8 + r) * kPitchT + wm + (q & 1) * 8);
                if (!TB) ldmatrix_x4<false>(b, sb + (wn + (q >> 1) * 8 + r) * kPitchK + k + (q & 1) * 8);
                else ldmatrix_x4<true>(b, sb + (k + (q & 1) * 8 + r) * kPitchT + wn + (q >> 1) * 8);
                mma_bf16_16816(acc[0], a, b);
                mma_bf16_16816(acc[1], a, b + 2);
            }
        }
        each(sa, kn);
        __syncthreads();  // the buffer is free for the request after next
        request(s + 2);
    }
}

// Calls f(row, column, value 0, value 1) for the warp's accumulators: two
// adjacent columns at a time.
template <typename F>
__device__ __forceinline__ void gemm_each(const float (&acc)[2][4], int row0, int col0, int M, int N, const F& f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r = row0 + (warp >> 1) * 16 + (lane >> 2), c = col0 + (warp & 1) * 16 + (lane & 3) * 2;
    if (row0 + (warp >> 1) * 16 >= M || col0 + (warp & 1) * 16 >= N) return;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        f(r, c + 8 * h, acc[h][0], acc[h][1]);
        f(r + 8, c + 8 * h, acc[h][2], acc[h][3]);
    }
}

// x in bf16, and per block the valid (mask != 0) targets it counted.
constexpr int kPrepBlocks = 64;
__global__ void __launch_bounds__(256) k_prepare(const float* __restrict__ x, bf16* __restrict__ xb, long long n,
                                                 const float* __restrict__ mask, long long m, int* counts) {
    const long long step = (long long)gridDim.x * blockDim.x, first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (long long i = first; i < n; i += step) xb[i] = __float2bfloat16(x[i]);
    if (!mask) return;
    int c = 0;
    for (long long i = first; i < m; i += step) c += mask[i] != 0.f;
    __shared__ int warp_sum[8];
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) c += warp_sum[w];
        counts[blockIdx.x] = c;
    }
}

// One layer: pre = in W^T + bias.  Hidden: pre and act = bf16(gelu(pre)).
// Output (act null): y = pre, and with targets the masked MSE (d = mask (y -
// t); loss = mean of d^2 over the valid entries, one partial sum per block;
// grad = bf16(2 d / count)).
struct ForwardArgs {
    const bf16 *in, *w;
    const float* bias;
    float* pre;
    bf16* act;
    float* y;
    const float *t, *mask;
    const int* counts;
    float* losses;
    bf16* grad;
    int M, N, K;
    int nx;  // tiles per row of tiles
};
__global__ void __launch_bounds__(kGemmThreads) k_forward(const ForwardArgs a) {
    __shared__ GemmSmem S;
    float acc[2][4];
    const int row0 = blockIdx.x / a.nx * kTile, col0 = blockIdx.x % a.nx * kTile;
    gemm_tile<false, false>(S, acc, a.in, a.K, a.w, a.K, row0, col0, a.M, a.N, a.K, [](const bf16*, int) {});
    if (a.act) {
        gemm_each(acc, row0, col0, a.M, a.N, [&](int r, int c, float v0, float v1) {
            const size_t i = (size_t)r * a.N + c;
            v0 += a.bias[c];
            v1 += a.bias[c + 1];
            *reinterpret_cast<float2*>(a.pre + i) = make_float2(v0, v1);
            *reinterpret_cast<__nv_bfloat162*>(a.act + i) = __floats2bfloat162_rn(gelu(v0), gelu(v1));
        });
        return;
    }
    float inv = 0.f, sum = 0.f;
    if (a.t) {
        __shared__ int total[2];
        if (threadIdx.x < kPrepBlocks) {
            const int c = __reduce_add_sync(0xffffffffu, a.counts[threadIdx.x]);
            if ((threadIdx.x & 31) == 0) total[threadIdx.x >> 5] = c;
        }
        __syncthreads();
        const int count = total[0] + total[1];
        inv = count > 0 ? (float)(1.0 / count) : 0.f;
    }
    gemm_each(acc, row0, col0, a.M, a.N, [&](int r, int c, float v0, float v1) {
        const size_t i = (size_t)r * a.N + c;
        v0 += a.bias[c];
        v1 += a.bias[c + 1];
        if (a.y) {  // the caller's array: any float alignment
            a.y[i] = v0;
            a.y[i + 1] = v1;
        }
        if (a.t) {
            const float d0 = a.mask[i] * (v0 - a.t[i]), d1 = a.mask[i + 1] * (v1 - a.t[i + 1]);
            sum += d0 * d0;
            sum += d1 * d1;
            *reinterpret_cast<__nv_bfloat162*>(a.grad + i) = __floats2bfloat162_rn(2.0f * d0 * inv, 2.0f * d1 * inv);
        }
    });
    if (a.t) {
        __shared__ float part[kGemmThreads / 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
        __syncthreads();
        if (threadIdx.x == 0)
            a.losses[blockIdx.x] = (part[0] + part[1] + part[2] + part[3]) * inv;
    }
}

// One backward stage from a layer's gradient `g` [n][N].  Blocks below
// nx * ny: the gradient of the layer below, bf16((g W) gelu'(pre)) [n][K].
// The others: dW = g^T in [N][K] and, from the staged gradients, db = column
// sums of g.  The first block also adds up the loss (deterministic).
struct BackwardArgs {
    const bf16 *g, *w, *in;
    const float* pre;
    bf16* below;
    float *dw, *db;
    int n, N, K;
    int nx, ny;  // tiles of the gradient below (0: first layer)
    const float* losses;
    int nlosses;
    float* loss;
};
__global__ void __launch_bounds__(kGemmThreads) k_backward(const BackwardArgs a) {
    __shared__ GemmSmem S;
    float acc[2][4];
    int tile = blockIdx.x;
    if (tile < a.nx * a.ny) {
        const int row0 = tile / a.nx * kTile, col0 = tile % a.nx * kTile;
        gemm_tile<false, true>(S, acc, a.g, a.N, a.w, a.K, row0, col0, a.n, a.K, a.N, [](const bf16*, int) {});
        gemm_each(acc, row0, col0, a.n, a.K, [&](int r, int c, float v0, float v1) {
            const size_t i = (size_t)r * a.K + c;
            const float2 p = *reinterpret_cast<const float2*>(a.pre + i);
            *reinterpret_cast<__nv_bfloat162*>(a.below + i) =
                __floats2bfloat162_rn(v0 * gelu_grad(p.x), v1 * gelu_grad(p.y));
        });
    } else {
        tile -= a.nx * a.ny;
        const int tx = (a.K + kTile - 1) / kTile;
        const int row0 = tile / tx * kTile, col0 = tile % tx * kTile;
        const bool sums = col0 == 0;
        float db = 0.f;  // thread (q, c): column row0 + c of g, rows q mod 4
        const int c = threadIdx.x & 31, q = threadIdx.x >> 5;
        gemm_tile<true, true>(S, acc, a.g, a.N, a.in, a.K, row0, col0, a.N, a.K, a.n, [&](const bf16* sg, int kn) {
            if (sums && row0 + c < a.N)
                for (int k = q; k < kn; k += 4) db += __bfloat162float(sg[k * kPitchT + c]);
        });
        gemm_each(acc, row0, col0, a.N, a.K, [&](int r, int cc, float v0, float v1) {
            *reinterpret_cast<float2*>(a.dw + (size_t)r * a.K + cc) = make_float2(v0, v1);
        });
        if (sums) {
            __shared__ float part[4][kTile];
            part[q][c] = db;
            __syncthreads();
            if (q == 0 && row0 + c < a.N) a.db[row0 + c] = (part[0][c] + part[1][c]) + (part[2][c] + part[3][c]);
        }
    }
    if (a.losses && blockIdx.x == 0 && threadIdx.x < 32) {
        float sum = 0.f;
        for (int i = threadIdx.x; i < a.nlosses; i += 32) sum += a.losses[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (threadIdx.x == 0) *a.loss = sum;
    }
}

__global__ void k_to_bf16(const float* x, bf16* y, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] = __float2bfloat16(x[i]);
}

__global__ void k_adam(float* w, const float* g, float* m, float* v, bf16* wb, long long n, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        w[i] = wi;
        if (wb) wb[i] = __float2bfloat16(wi);
    }
}

unsigned grid1(long long n) { return (unsigned)std::max(1LL, std::min((n + 255) / 256, 148LL * 8)); }

// ------------------------------------------------- fused ensemble inference
// The picker evaluates a handful of models on one 16-row batch per pick:
// at that size the per-layer GEMM, bias and GELU launches cost far more
// than the arithmetic.  One launch does it all: CTA (m, t) runs model m on
// rows [16t, 16t + 16) through every layer, with the activations in shared
// memory (bf16, as the layered path rounds them), warp-level bf16 tensor-core
// tiles (mma m16n8k16, fp32 accumulation) whose B operands stream straight
// from the model's bf16 weights in L2, and bias + GELU fused into the tile
// epilogue.  The models of one row tile form a thread-block cluster; once
// every model's output tile is in its CTA's shared memory, CTA 0 of the
// cluster reads them through distributed shared memory and writes their
// mean, summed in model order (deterministic).
constexpr int kEnsMaxModels = 8;  // portable cluster size
constexpr int kEnsH = 256;        // hidden width the fused kernel is built for
constexpr int kEnsMaxOut = 256;
constexpr int kEnsThreads = 1024;  // 32 warps: one 8-column tile each (widths up to 256)

struct EnsModel {
    const bf16* wb;   // bf16 weights (layer l at woff[l], [out][in] row-major)
    const float* w;   // fp32 arena (biases at boff[l])
};
struct EnsArgs {
    EnsModel m[kEnsMaxModels];
    long long woff[4], boff[4];
    int nmodels, din, dout;
    const float* x;  // [n][din]
    float* y;        // [n][dout], the mean over the models
};

// One layer for 16 rows: out[16][N] = act[16][K] W^T + bias, then GELU into
// the next activation buffer (hidden) or fp32 into `outf` (last layer).
// Warp w owns the n-tile w (8 columns; N <= 8 * warps).  Its weight
// fragments for the whole K (at most 16 k-steps, two 32-bit registers each)
// and its two bias values are loaded in one round (ens_fetch), and the
// kernel issues the next layer's round as soon as this layer's mma chain
// has consumed the fragments, so that the L2 latency of layer l + 1 runs
// under layer l's epilogue and block barrier.
//
// Which columns of a 32-column block feed which k slots of the mma is free,
// as long as A and B agree: lane (g, t) gives k-step 2j the columns
// 32j + 8t + {0,1} (slots 2t, 2t+1) and 32j + 8t + {2,3} (slots 2t+8,
// 2t+9), and k-step 2j+1 the columns 32j + 8t + {4..7}.  Each lane then
// reads 16 contiguous bytes of its weight row per two k-steps (one
// fully-used 32-byte sector pair per row and instruction, a quarter of the
// load instructions of the mma's natural column order) and 16 contiguous
// bytes of each activation row.  A trailing single k-step (K not a
// multiple of 32) takes columns 4t + {0,1} and 4t + {2,3} of its 16.
struct EnsFrag {
    uint32_t b[16][2];
    float b0, b1;
};

__device__ __forceinline__ void ens_fetch(EnsFrag& f, int K, const bf16* __restrict__ W, const float* __restrict__ bias,
                                          int N) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    if (warp * 8 >= N) return;
    const int npair = K / 32;
    const bf16* wr = W + (size_t)(warp * 8 + g) * K;
#pragma unroll
    for (int j = 0; j < 8; j++) {  // unrolled: the fragment indices stay static (registers)
        if (j < npair) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(wr + 32 * j + 8 * t));
            f.b[2 * j][0] = v.x;
            f.b[2 * j][1] = v.y;
            f.b[2 * j + 1][0] = v.z;
            f.b[2 * j + 1][1] = v.w;
        } else if (j == npair && (K % 32)) {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(wr + 32 * j + 4 * t));
            f.b[2 * j][0] = v.x;
            f.b[2 * j][1] = v.y;
        }
    }
    const int c = warp * 8 + 2 * t;
    f.b0 = __ldg(bias + c);
    f.b1 = __ldg(bias + c + 1);
}

// The mma chain of one layer from fragments already in registers.
__device__ __forceinline__ void ens_mma(float* acc, const bf16* __restrict__ act, int lda, int K, const EnsFrag& f) {
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int npair = K / 32;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        if (j < npair) {
            const uint4 r0 = *reinterpret_cast<const uint4*>(act + g * lda + 32 * j + 8 * t);
            const uint4 r1 = *reinterpret_cast<const uint4*>(act + (g + 8) * lda + 32 * j + 8 * t);
            const uint32_t a0[4] = {r0.x, r1.x, r0.y, r1.y};
            const uint32_t a1[4] = {r0.z, r1.z, r0.w, r1.w};
            mma_bf16_16816(acc, a0, f.b[2 * j]);
            mma_bf16_16816(acc, a1, f.b[2 * j + 1]);
        } else if (j == npair && (K % 32)) {
            const uint2 r0 = *reinterpret_cast<const uint2*>(act + g * lda + 32 * j + 4 * t);
            const uint2 r1 = *reinterpret_cast<const uint2*>(act + (g + 8) * lda + 32 * j + 4 * t);
            const uint32_t a[4] = {r0.x, r1.x, r0.y, r1.y};
            mma_bf16_16816(acc, a, f.b[2 * j]);
        }
    }
}

// Bias and GELU into the next activation buffer, or fp32 output.
__device__ __forceinline__ void ens_epilogue(const float* acc, float b0, float b1, bf16* next, int ldn, float* outf,
                                             int ldo) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int c = warp * 8 + 2 * t;
    const float v[4] = {acc[0] + b0, acc[1] + b1, acc[2] + b0, acc[3] + b1};
    if (next) {
        *(__nv_bfloat162*)(next + g * ldn + c) = __floats2bfloat162_rn(gelu(v[0]), gelu(v[1]));
        *(__nv_bfloat162*)(next + (g + 8) * ldn + c) = __floats2bfloat162_rn(gelu(v[2]), gelu(v[3]));
    } else {
        outf[g * ldo + c] = v[0];
        outf[g * ldo + c + 1] = v[1];
        outf[(g + 8) * ldo + c] = v[2];
        outf[(g + 8) * ldo + c + 1] = v[3];
    }
}

__global__ void __launch_bounds__(kEnsThreads) k_mlp_ensemble(EnsArgs a) {
    namespace cg = cooperative_groups;
    // Padded rows (144 words, 16 mod 32): the 16-byte activation loads of a
    // quarter warp (rows g, g + 1; t = 0..3) fall on all 32 banks once.
    constexpr int kLd = kEnsH + 32;
    __shared__ __align__(16) bf16 s_act[2][16 * kLd];
    __shared__ __align__(16) float s_out[16 * kEnsMaxOut];
    cg::cluster_group cluster = cg::this_cluster();
    const int model = (int)cluster.block_rank();
    const int row0 = blockIdx.y * 16;
    const EnsModel M = a.m[model];
    const int dims[5] = {a.din, kEnsH, kEnsH, kEnsH, a.dout};
    const int warp = threadIdx.x >> 5;
    EnsFrag f;
    ens_fetch(f, dims[0], M.wb + a.woff[0], M.w + a.boff[0], dims[1]);
    for (int i = threadIdx.x; i < 16 * a.din; i += kEnsThreads) {
        const int r = i / a.din, k = i % a.din;
        s_act[0][r * kLd + k] = __float2bfloat16(a.x[(size_t)(row0 + r) * a.din + k]);
    }
    __syncthreads();
#pragma unroll 1
    for (int l = 0; l < 4; l++) {
        const bf16* in = s_act[l & 1];
        bf16* nxt = l < 3 ? s_act[(l + 1) & 1] : nullptr;
        if (warp * 8 < dims[l + 1]) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            ens_mma(acc, in, kLd, dims[l], f);
            const float b0 = f.b0, b1 = f.b1;
            if (l < 3) ens_fetch(f, dims[l + 1], M.wb + a.woff[l + 1], M.w + a.boff[l + 1], dims[l + 2]);
            ens_epilogue(acc, b0, b1, nxt, kLd, s_out, a.dout);
        } else if (l < 3) {
            ens_fetch(f, dims[l + 1], M.wb + a.woff[l + 1], M.w + a.boff[l + 1], dims[l + 2]);
        }
        __syncthreads();
    }
    cluster.sync();
    if (model == 0) {
        const float inv = 1.0f / (float)a.nmodels;
        for (int i = threadIdx.x; i < 16 * a.dout; i += kEnsThreads) {
            float sum = 0.f;
            for (int m = 0; m < a.nmodels; m++) sum += cluster.map_shared_rank(s_out, m)[i];
            a.y[(size_t)(row0 + i / a.dout) * a.dout + i % a.dout] = sum * inv;
        }
    }
    cluster.sync();  // keep every CTA's shared memory alive until CTA 0 has read it
}

}  // namespace

struct bine_mlp_s {
    int din, h, dout, max_batch;
    int nlayer = 4;
    int in_dim[4], out_dim[4];
    // fp32 master weights and biases (one arena), gradients, Adam moments.
    float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
    bf16* wb = nullptr;  // bf16 weights (same offsets as w, biases unused)
    size_t woff[4], boff[4], nparams = 0;
    long long step = 0;
    // Activations for max_batch rows.
    bf16* x = nullptr;           // input, bf16
    float* pre[3] = {nullptr};   // hidden pre-activations (fp32)
    bf16* act[3] = {nullptr};    // hidden activations (bf16)
    bf16* dpre[2] = {nullptr};   // bf16 gradients of two consecutive layers
    int* counts = nullptr;       // valid targets per prepare block
    float* losses = nullptr;     // loss per output tile, then the loss, then `side`
    float* loss = nullptr;
    float* side = nullptr;       // output, or targets and mask, where the caller's are not this device's
    float* staged = nullptr;     // pinned host copy of the gradients and the loss
    cudaEvent_t inputs_read = nullptr;  // a step's last read of the caller's arrays
    ~bine_mlp_s() {
        cudaFree(w);
        cudaFree(g);
        cudaFree(m);
        cudaFree(v);
        cudaFree(wb);
        cudaFree(x);
        for (float* p : pre) cudaFree(p);
        for (bf16* p : act) cudaFree(p);
        for (bf16* p : dpre) cudaFree(p);
        cudaFree(counts);
        cudaFree(losses);
        cudaFreeHost(staged);
        if (inputs_read) cudaEventDestroy(inputs_read);
    }
};

namespace {

int tiles(int n) { return (n + kTile - 1) / kTile; }

// Rows of the batch (and the targets' mask, for a loss) to the layered path.
void prepare_batch(bine_mlp_t mlp, const float* d_x, const float* d_mask, int n, cudaStream_t s) {
    k_prepare<<<kPrepBlocks, 256, 0, s>>>(d_x, mlp->x, (long long)n * mlp->din, d_mask, (long long)n * mlp->dout,
                                          mlp->counts);
}

// Whether kernels of the current device can work on a caller's array where it
// is: its own and managed memory.  Memory of another device, which a kernel
// reaches only with peer access, and pinned host memory go through `side` in
// copies of the runtime.  Pageable memory is refused.
int in_place(const float* p, bool* direct) {
    cudaPointerAttributes at;
    int dev = 0;
    if (!p) return mfail(BINE_ERR_ARG, "null output, targets or mask");
    MLP_TRY(cudaPointerGetAttributes(&at, p));
    MLP_TRY(cudaGetDevice(&dev));
    if (at.type == cudaMemoryTypeUnregistered)
        return mfail(BINE_ERR_ARG, "output, targets and mask must be device arrays");
    *direct = at.type == cudaMemoryTypeManaged || (at.type == cudaMemoryTypeDevice && at.device == dev);
    return BINE_SUCCESS;
}

int check_batch(bine_mlp_t mlp, const float* d_x, int n) {
    if (!mlp || !d_x || n <= 0 || n > mlp->max_batch || n % 16)
        return mfail(BINE_ERR_ARG, "batch must be a multiple of 16 within max_batch");
    return BINE_SUCCESS;
}

// Targets and mask as the kernels read them: *t and *mask are replaced by
// their copies where needed.
int place_targets(bine_mlp_t mlp, const float** t, const float** mask, int n, cudaStream_t s) {
    bool direct[2];
    int rc = in_place(*t, &direct[0]);
    if (rc == BINE_SUCCESS) rc = in_place(*mask, &direct[1]);
    if (rc) return rc;
    const float** arr[2] = {t, mask};
    for (int i = 0; i < 2; i++) {
        if (direct[i]) continue;
        float* own = mlp->side + (size_t)i * mlp->max_batch * mlp->dout;
        MLP_TRY(cudaMemcpyAsync(own, *arr[i], sizeof(float) * (size_t)n * mlp->dout, cudaMemcpyDefault, s));
        *arr[i] = own;
    }
    return BINE_SUCCESS;
}

// Forward pass of the `n` prepared rows: to d_y, or with targets to the
// output gradient and the loss partials.
void forward(bine_mlp_t mlp, int n, float* d_y, const float* d_t, const float* d_mask, cudaStream_t s) {
    for (int l = 0; l < mlp->nlayer; l++) {
        const bool hidden = l + 1 < mlp->nlayer;
        ForwardArgs a{};
        a.in = l == 0 ? mlp->x : mlp->act[l - 1];
        a.w = mlp->wb + mlp->woff[l];
        a.bias = mlp->w + mlp->boff[l];
        a.M = n;
        a.N = mlp->out_dim[l];
        a.K = mlp->in_dim[l];
        if (hidden) {
            a.pre = mlp->pre[l];
            a.act = mlp->act[l];
        } else {
            a.y = d_y;
            a.t = d_t;
            a.mask = d_mask;
            a.counts = mlp->counts;
            a.losses = mlp->losses;
            a.grad = mlp->dpre[l & 1];
        }
        // One row of the grid: a batch may have more rows of tiles than a
        // grid has rows (65,535).
        a.nx = tiles(a.N);
        k_forward<<<(unsigned)(a.nx * tiles(n)), kGemmThreads, 0, s>>>(a);
    }
}

// Backward pass: fills mlp->g with the gradients of every weight and bias
// and *mlp->loss.
void backward(bine_mlp_t mlp, int n, cudaStream_t s) {
    for (int l = mlp->nlayer - 1; l >= 0; l--) {
        BackwardArgs a{};
        a.n = n;
        a.N = mlp->out_dim[l];
        a.K = mlp->in_dim[l];
        a.g = mlp->dpre[l & 1];
        a.w = mlp->wb + mlp->woff[l];
        a.in = l == 0 ? mlp->x : mlp->act[l - 1];
        a.dw = mlp->g + mlp->woff[l];
        a.db = mlp->g + mlp->boff[l];
        if (l > 0) {
            a.pre = mlp->pre[l - 1];
            a.below = mlp->dpre[(l - 1) & 1];
            a.nx = tiles(a.K);
            a.ny = tiles(n);
        }
        if (l == mlp->nlayer - 1) {
            a.losses = mlp->losses;
            a.nlosses = tiles(mlp->dout) * tiles(n);
            a.loss = mlp->loss;
        }
        k_backward<<<a.nx * a.ny + tiles(a.N) * tiles(a.K), kGemmThreads, 0, s>>>(a);
    }
}

}  // namespace

extern "C" {

const char* bine_mlp_last_error(void) { return g_mlp_err.c_str(); }

int bine_mlp_create(int in_dim, int hidden, int out_dim, int max_batch, unsigned long long seed, bine_mlp_t* out) {
    if (!out || in_dim <= 0 || hidden <= 0 || out_dim <= 0 || max_batch <= 0 || in_dim % 16 || hidden % 16 ||
        out_dim % 16 || max_batch % 16)
        return mfail(BINE_ERR_ARG, "dimensions must be positive multiples of 16");
    *out = nullptr;
    auto m = std::unique_ptr<bine_mlp_s>(new bine_mlp_s());
    m->din = in_dim;
    m->h = hidden;
    m->dout = out_dim;
    m->max_batch = max_batch;
    const int dims[5] = {in_dim, hidden, hidden, hidden, out_dim};
    size_t off = 0;
    for (int l = 0; l < 4; l++) {
        m->in_dim[l] = dims[l];
        m->out_dim[l] = dims[l + 1];
        m->woff[l] = off;
        off += (size_t)dims[l] * dims[l + 1];
        off = (off + 15) / 16 * 16;
        m->boff[l] = off;
        off += (size_t)dims[l + 1];
        off = (off + 15) / 16 * 16;
    }
    m->nparams = off;
    // He-style initialisation from a seeded generator; biases zero.
    std::vector<float> hw(off, 0.f);
    std::mt19937_64 rng(seed);
    for (int l = 0; l < 4; l++) {
        std::normal_distribution<float> nd(0.f, std::sqrt(2.0f / dims[l]) * (l == 3 ? 0.5f : 1.0f));
        for (size_t i = 0; i < (size_t)dims[l] * dims[l + 1]; i++) hw[m->woff[l] + i] = nd(rng);
    }
    MLP_TRY(cudaMalloc(&m->w, off * sizeof(float)));
    MLP_TRY(cudaMalloc(&m->g, off * sizeof(float)));
    MLP_TRY(cudaMalloc(&m->m, off * sizeof(float)));
    MLP_TRY(cudaMalloc(&m->v, off * sizeof(float)));
    MLP_TRY(cudaMalloc(&m->wb, off * sizeof(bf16)));
    MLP_TRY(cudaMemcpy(m->w, hw.data(), off * sizeof(float), cudaMemcpyHostToDevice));
    MLP_TRY(cudaMemset(m->g, 0, off * sizeof(float)));
    MLP_TRY(cudaMemset(m->m, 0, off * sizeof(float)));
    MLP_TRY(cudaMemset(m->v, 0, off * sizeof(float)));
    k_to_bf16<<<grid1(off), 256>>>(m->w, m->wb, (long long)off);
    MLP_TRY(cudaMalloc(&m->x, (size_t)max_batch * in_dim * sizeof(bf16)));
    for (int l = 0; l < 3; l++) {
        MLP_TRY(cudaMalloc(&m->pre[l], (size_t)max_batch * hidden * sizeof(float)));
        MLP_TRY(cudaMalloc(&m->act[l], (size_t)max_batch * hidden * sizeof(bf16)));
    }
    for (int l = 0; l < 2; l++)
        MLP_TRY(cudaMalloc(&m->dpre[l], (size_t)max_batch * std::max(hidden, out_dim) * sizeof(bf16)));
    MLP_TRY(cudaMalloc(&m->counts, kPrepBlocks * sizeof(int)));
    const size_t nlosses = (size_t)tiles(max_batch) * tiles(out_dim);
    const size_t aside = (nlosses + 1 + 3) / 4 * 4;  // a 16-byte boundary
    MLP_TRY(cudaMalloc(&m->losses, (aside + 2 * (size_t)max_batch * out_dim) * sizeof(float)));
    m->loss = m->losses + nlosses;
    m->side = m->losses + aside;
    MLP_TRY(cudaMallocHost(&m->staged, (off + 1) * sizeof(float)));
    MLP_TRY(cudaEventCreateWithFlags(&m->inputs_read, cudaEventDisableTiming));
    MLP_TRY(cudaDeviceSynchronize());
    *out = m.release();
    return BINE_SUCCESS;
}

int bine_mlp_destroy(bine_mlp_t mlp) {
    delete mlp;
    return BINE_SUCCESS;
}

int bine_mlp_num_params(bine_mlp_t mlp, size_t* n) {
    if (!mlp || !n) return mfail(BINE_ERR_ARG, "null argument");
    *n = mlp->nparams;
    return BINE_SUCCESS;
}

int bine_mlp_get_params(bine_mlp_t mlp, float* host) {
    if (!mlp || !host) return mfail(BINE_ERR_ARG, "null argument");
    MLP_TRY(cudaMemcpy(host, mlp->w, mlp->nparams * sizeof(float), cudaMemcpyDeviceToHost));
    return BINE_SUCCESS;
}

int bine_mlp_set_params(bine_mlp_t mlp, const float* host) {
    if (!mlp || !host) return mfail(BINE_ERR_ARG, "null argument");
    MLP_TRY(cudaMemcpy(mlp->w, host, mlp->nparams * sizeof(float), cudaMemcpyHostToDevice));
    k_to_bf16<<<grid1(mlp->nparams), 256>>>(mlp->w, mlp->wb, (long long)mlp->nparams);
    MLP_TRY(cudaDeviceSynchronize());
    return BINE_SUCCESS;
}

int bine_mlp_forward(bine_mlp_t mlp, const float* d_x, int n, float* d_y, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    bool direct;
    int rc = check_batch(mlp, d_x, n);
    if (rc == BINE_SUCCESS) rc = in_place(d_y, &direct);
    if (rc) return rc;
    prepare_batch(mlp, d_x, nullptr, n, s);
    forward(mlp, n, direct ? d_y : mlp->side, nullptr, nullptr, s);
    if (!direct)
        MLP_TRY(cudaMemcpyAsync(d_y, mlp->side, sizeof(float) * (size_t)n * mlp->dout, cudaMemcpyDefault, s));
    MLP_TRY(cudaGetLastError());
    return BINE_SUCCESS;
}

int bine_mlp_gradients(bine_mlp_t mlp, const float* d_x, const float* d_t, const float* d_mask, int n, float* host_grads,
                       float* loss) {
    cudaStream_t s = 0;
    int rc = check_batch(mlp, d_x, n);
    if (rc == BINE_SUCCESS) rc = place_targets(mlp, &d_t, &d_mask, n, s);
    if (rc) return rc;
    prepare_batch(mlp, d_x, d_mask, n, s);
    forward(mlp, n, nullptr, d_t, d_mask, s);
    backward(mlp, n, s);
    MLP_TRY(cudaGetLastError());
    // Through pinned memory: straight into the caller's pageable arrays the
    // driver stages the copies itself, one after the other.
    if (host_grads)
        MLP_TRY(cudaMemcpyAsync(mlp->staged, mlp->g, mlp->nparams * sizeof(float), cudaMemcpyDeviceToHost, s));
    MLP_TRY(cudaMemcpyAsync(mlp->staged + mlp->nparams, mlp->loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    MLP_TRY(cudaStreamSynchronize(s));
    if (host_grads) std::memcpy(host_grads, mlp->staged, mlp->nparams * sizeof(float));
    if (loss) *loss = mlp->staged[mlp->nparams];
    return BINE_SUCCESS;
}

int bine_mlp_train_step(bine_mlp_t mlp, const float* d_x, const float* d_t, const float* d_mask, int n, float lr,
                        void* stream, float* loss) {
    cudaStream_t s = (cudaStream_t)stream;
    int rc = check_batch(mlp, d_x, n);
    if (rc == BINE_SUCCESS) rc = place_targets(mlp, &d_t, &d_mask, n, s);
    if (rc) return rc;
    prepare_batch(mlp, d_x, d_mask, n, s);
    forward(mlp, n, nullptr, d_t, d_mask, s);
    // The caller may refill or free its arrays on return, and only the stages
    // up to here read them.
    if (!loss) MLP_TRY(cudaEventRecord(mlp->inputs_read, s));
    backward(mlp, n, s);
    mlp->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)mlp->step), c2 = 1.f - std::pow(b2, (float)mlp->step);
    k_adam<<<grid1(mlp->nparams), 256, 0, s>>>(mlp->w, mlp->g, mlp->m, mlp->v, mlp->wb, (long long)mlp->nparams, lr, b1,
                                               b2, 1e-8f, c1, c2);
    if (loss) {
        MLP_TRY(cudaMemcpyAsync(mlp->staged + mlp->nparams, mlp->loss, sizeof(float), cudaMemcpyDeviceToHost, s));
        MLP_TRY(cudaStreamSynchronize(s));
        *loss = mlp->staged[mlp->nparams];
    } else {
        MLP_TRY(cudaEventSynchronize(mlp->inputs_read));
    }
    MLP_TRY(cudaGetLastError());
    return BINE_SUCCESS;
}

struct bine_mlp_ensemble_s {
    std::vector<bine_mlp_t> models;
};

int bine_mlp_ensemble_create(const bine_mlp_t* models, int nmodels, bine_mlp_ensemble_t* out) {
    if (!out || !models || nmodels < 1 || nmodels > kEnsMaxModels)
        return mfail(BINE_ERR_ARG, "an ensemble holds 1 to 8 models");
    *out = nullptr;
    const bine_mlp_t m0 = models[0];
    if (!m0) return mfail(BINE_ERR_ARG, "null model");
    if (m0->h != kEnsH || m0->din > kEnsH || m0->dout > kEnsMaxOut)
        return mfail(BINE_ERR_ARG, "the fused forward takes hidden width 256, input and output widths up to 256");
    for (int i = 1; i < nmodels; i++)
        if (!models[i] || models[i]->din != m0->din || models[i]->h != m0->h || models[i]->dout != m0->dout)
            return mfail(BINE_ERR_ARG, "the models of an ensemble must have the same shape");
    auto e = new bine_mlp_ensemble_s();
    e->models.assign(models, models + nmodels);
    *out = e;
    return BINE_SUCCESS;
}

int bine_mlp_ensemble_destroy(bine_mlp_ensemble_t e) {
    delete e;
    return BINE_SUCCESS;
}

int bine_mlp_ensemble_forward(bine_mlp_ensemble_t e, const float* d_x, int n, float* d_y, void* stream) {
    if (!e || !d_x || !d_y || n <= 0 || n % 16) return mfail(BINE_ERR_ARG, "batch must be a positive multiple of 16");
    if (n / 16 > 65535) return mfail(BINE_ERR_ARG, "batch too large for one launch");
    EnsArgs a{};
    const bine_mlp_t m0 = e->models[0];
    for (int l = 0; l < 4; l++) {
        a.woff[l] = (long long)m0->woff[l];
        a.boff[l] = (long long)m0->boff[l];
    }
    a.nmodels = (int)e->models.size();
    for (int i = 0; i < a.nmodels; i++) a.m[i] = EnsModel{e->models[i]->wb, e->models[i]->w};
    a.din = m0->din;
    a.dout = m0->dout;
    a.x = d_x;
    a.y = d_y;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)a.nmodels, (unsigned)(n / 16), 1);
    cfg.blockDim = dim3(kEnsThreads, 1, 1);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)a.nmodels;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MLP_TRY(cudaLaunchKernelEx(&cfg, k_mlp_ensemble, a));
    return BINE_SUCCESS;
}

}  // extern "C"
