// Message-passing network that proposes a start subspace for the Lanczos
// iteration of a finite-volume diffusion operator (the learned warm start).
//
//   h0   = tanh(W0 x + b0)                          x: F node features
//   h_l  = tanh(W_l [h_{l-1}, A h_{l-1}] + b_l)     l = 1..L, A the normalised
//                                                   adjacency of the operator
//   Y    = W_o h_L + b_o                            P outputs per node
//
// Activations are stored in BF16, weights are used in BF16 and kept in FP32
// for the optimiser; every product accumulates in FP32.  Training minimises
// the subspace loss 1 - trace(U^T P_Y U) / k, P_Y the orthogonal projector
// onto span(Y) and U the k eigenvectors the solver computed for the same
// operator; its gradient is dL/dY = -(2/k) (U - Y C) C^T with
// C = (Y^T Y)^{-1} Y^T U.  Adam updates the FP32 weights.
#include "../chain.cuh"
#include "../common.cuh"
#include "../counters.h"
#include "../../../include/speigs_b200.h"

#include <cub/device/device_scan.cuh>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

namespace spx {
const char *set_last_error_text(const char *msg);
cudaMemPool_t device_pool(int dev);
}

namespace {

using bf16 = __nv_bfloat16;
constexpr int kRows = 64;       // nodes per block in the dense layers
constexpr int kThreads = 256;
constexpr int kHid = 64;        // hidden width (the only one create accepts)

SPX_DEV float to_f(bf16 v) { return __bfloat162float(v); }
SPX_DEV float to_f(float v) { return v; }
template <class T> SPX_DEV T from_f(float v);
template <> SPX_DEV bf16 from_f<bf16>(float v) { return __float2bfloat16(v); }
template <> SPX_DEV float from_f<float>(float v) { return v; }

// ---- message passing of the layers that stay off the tensor cores: out =
// A in, one warp per node, 2 features a lane
__global__ void spmm_kernel(int n, int hid, const int32_t *__restrict__ rp,
                            const int32_t *__restrict__ ci, const float *__restrict__ w,
                            const bf16 *__restrict__ in, bf16 *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= n) return;
    for (int f0 = 0; f0 < hid; f0 += 64) {
        float a0 = 0.f, a1 = 0.f;
        const int f = f0 + 2 * lane;
        for (int q = rp[row]; q < rp[row + 1]; q++) {
            const float wq = w[q];
            const bf16 *src = in + (size_t)ci[q] * hid;
            if (f < hid) a0 += wq * to_f(src[f]);
            if (f + 1 < hid) a1 += wq * to_f(src[f + 1]);
        }
        bf16 *dst = out + (size_t)row * hid;
        if (f < hid) dst[f] = from_f<bf16>(a0);
        if (f + 1 < hid) dst[f + 1] = from_f<bf16>(a1);
    }
}

// ---- the messages' gradient: out += A in, FP32, 64 features a node.
// Bound by L2 latency: 16 lanes take a node (a float4 each, one 256-byte row
// a gather), read the indices and weights of eight edges at once and then
// have eight gathers in flight.  32^3 nodes: 10.6 -> 7.0 us against one
// warp per node with one edge in flight.
__global__ void __launch_bounds__(kThreads)
spmm_add_kernel(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                const float *__restrict__ w, const float *__restrict__ in, float *__restrict__ out) {
    const int lane = threadIdx.x & 31, f = lane & 15, g0 = lane & 16;
    spx::chain_begin();
    const int row = blockIdx.x * (kThreads / 16) + (threadIdx.x >> 4);
    int q = row < n ? rp[row] : 0;
    const int q1 = row < n ? rp[row + 1] : 0;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (; __any_sync(~0u, q < q1); q += 8) {
        const bool mine = f < 8 && q + f < q1;
        const int c = mine ? ci[q + f] : -1;
        const float wv = mine ? w[q + f] : 0.f;
        float4 v[8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const int cc = __shfl_sync(~0u, c, g0 + t);
            v[t] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (cc >= 0) v[t] = *reinterpret_cast<const float4 *>(in + (size_t)cc * kHid + 4 * f);
        }
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const float ww = __shfl_sync(~0u, wv, g0 + t);
            acc.x += ww * v[t].x;
            acc.y += ww * v[t].y;
            acc.z += ww * v[t].z;
            acc.w += ww * v[t].w;
        }
    }
    if (row >= n) return;
    float4 *dst = reinterpret_cast<float4 *>(out + (size_t)row * kHid + 4 * f);
    float4 o = *dst;
    o.x += acc.x;
    o.y += acc.y;
    o.z += acc.z;
    o.w += acc.w;
    *dst = o;
}

// ---- input layer: out[i, :] = tanh(W x_i + b), FP32 features (F <= 64) to 64
// BF16 outputs.  Bound by tanhf and the 128-byte rows it writes; a thread
// takes 4 rows x 8 outputs so that F FMAs an output cost few shared-memory
// reads.  48^3 nodes, F = 9: 33.4 -> 11.7 us against one output a thread at a
// time.
constexpr int kInRows = 128;
__global__ void __launch_bounds__(kThreads)
input_fwd_kernel(int n, int F, const float *__restrict__ X, const bf16 *__restrict__ W,
                 const float *__restrict__ b, bf16 *__restrict__ out) {
    extern __shared__ float4 in_sm[];
    spx::chain_begin();
    float *Ws = reinterpret_cast<float *>(in_sm);   // F x 64: W transposed
    float *Xs = Ws + F * kHid;                      // kInRows x (F + 1)
    const int r0 = blockIdx.x * kInRows;
    const int rows = min(kInRows, n - r0);
    for (int t = threadIdx.x; t < kHid * F; t += kThreads) Ws[(t % F) * kHid + t / F] = to_f(W[t]);
    for (int t = threadIdx.x; t < kInRows * F; t += kThreads)
        Xs[(t / F) * (F + 1) + t % F] = t < rows * F ? X[(size_t)r0 * F + t] : 0.f;
    __syncthreads();
    const int og = threadIdx.x & 7, rg = threadIdx.x >> 3;   // outputs 4 og + {0..3, 32..35}
    float acc[4][8];
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int e = 0; e < 8; e++) acc[j][e] = b[(e & 4) * 8 + 4 * og + (e & 3)];
    for (int k = 0; k < F; k++) {
        const float4 w0 = *reinterpret_cast<const float4 *>(Ws + k * kHid + 4 * og);
        const float4 w1 = *reinterpret_cast<const float4 *>(Ws + k * kHid + 32 + 4 * og);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float x = Xs[(rg + 32 * j) * (F + 1) + k];
            acc[j][0] += x * w0.x;
            acc[j][1] += x * w0.y;
            acc[j][2] += x * w0.z;
            acc[j][3] += x * w0.w;
            acc[j][4] += x * w1.x;
            acc[j][5] += x * w1.y;
            acc[j][6] += x * w1.z;
            acc[j][7] += x * w1.w;
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int r = rg + 32 * j;
        if (r >= rows) break;
        __align__(16) bf16 v[8];
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = __float2bfloat16(tanhf(acc[j][e]));
        bf16 *dst = out + (size_t)(r0 + r) * kHid + 4 * og;
        *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(v);
        *reinterpret_cast<uint2 *>(dst + 32) = *reinterpret_cast<const uint2 *>(v + 4);
    }
}

// ---- dense layer forward: out[i, o] = act(b[o] + sum_k W[o, k] x[i, k]),
// x = [X1[i, 0:K1], X2[i, 0:K2]] (X2 may be absent).  act: 0 identity, 1 tanh.
template <class TO>
__global__ void __launch_bounds__(kThreads)
dense_fwd_kernel(int n, int K1, const bf16 *__restrict__ X1, int K2, const bf16 *__restrict__ X2,
                 int N, const bf16 *__restrict__ W, const float *__restrict__ b, int act,
                 TO *__restrict__ out) {
    extern __shared__ float sm[];
    const int K = K1 + K2;
    float *Xs = sm;                       // kRows x (K + 1)
    float *Ws = Xs + kRows * (K + 1);     // N x (K + 1)
    const int r0 = blockIdx.x * kRows;
    for (int t = threadIdx.x; t < kRows * K; t += blockDim.x) {
        const int r = t / K, k = t % K, i = r0 + r;
        float v = 0.f;
        if (i < n) v = (k < K1) ? to_f(X1[(size_t)i * K1 + k]) : to_f(X2[(size_t)i * K2 + (k - K1)]);
        Xs[r * (K + 1) + k] = v;
    }
    for (int t = threadIdx.x; t < N * K; t += blockDim.x) Ws[(t / K) * (K + 1) + t % K] = to_f(W[t]);
    __syncthreads();
    for (int t = threadIdx.x; t < kRows * N; t += blockDim.x) {
        const int r = t / N, o = t % N, i = r0 + r;
        if (i >= n) continue;
        float acc = b[o];
        const float *xr = Xs + r * (K + 1), *wr = Ws + o * (K + 1);
        for (int k = 0; k < K; k++) acc += xr[k] * wr[k];
        out[(size_t)i * N + o] = from_f<TO>(act ? tanhf(acc) : acc);
    }
}

// ---- dense layer backward.  dZ = dOut * act'(y); dX1, dX2 = the columns of
// dZ W (FP32, 64 each); dW += dZ^T x; db += column sums of dZ.  x is 128 wide
// (K = 128: two BF16 halves) or up to 64 wide (K = 64: F columns of BF16 or
// FP32, the rest zero; dX1 is then 64 wide or not wanted).
//
// Both products stay in FP32 on the FMA pipe (dZ is an FP32 gradient), so a
// tile of 64 rows costs at least 2 x 64 x 64 x K FMAs: 15 us a hidden layer at
// 32^3 nodes.  What bounds the rest is the shared-memory reads, so a thread
// keeps a 4 x 8 piece of the product in registers (2 x 8 for K = 64) and reads
// 16 bytes at a time, and a block keeps its share of dW in registers over all
// its tiles: one 16-byte atomic a thread and row at the end.  Hidden layer:
// 210 -> 40 us, output layer of 24: 46 -> 17, input layer of 9: 21 -> 23
// us against one element a thread at a time and dW added up once a tile.
constexpr int kZs = kHid + 4;
template <int K>
constexpr size_t bwd_smem() { return sizeof(float) * ((size_t)kHid * K + (size_t)kRows * K + (size_t)kRows * kZs); }

template <int K, class TX>
__global__ void __launch_bounds__(kThreads, 2)
dense_bwd_kernel(int n, int F, const TX *__restrict__ X1, const bf16 *__restrict__ X2, int N,
                 const bf16 *__restrict__ W, const bf16 *__restrict__ y,
                 const float *__restrict__ dout, float *__restrict__ dX1, float *__restrict__ dX2,
                 float *__restrict__ dW, float *__restrict__ db) {
    constexpr int CG = K / 8;               // thread columns: 4 cg + {0..3} and K / 2 + the same
    constexpr int TR = kRows * CG / kThreads;   // thread rows
    extern __shared__ float4 bwd_sm[];
    spx::chain_begin();
    float *Ws = reinterpret_cast<float *>(bwd_sm);   // 64 x K, rows >= N zero
    float *Xs = Ws + kHid * K;                       // kRows x K
    float *Zs = Xs + kRows * K;                      // kRows x kZs, columns >= N zero
    const int tid = threadIdx.x, cg = tid % CG, rg = tid / CG;
    const int KW = K == 128 ? 128 : F;               // columns that exist
    for (int t = tid; t < kHid * K; t += kThreads) {
        const int o = t / K, k = t % K;
        Ws[t] = o < N && k < KW ? to_f(W[(size_t)o * KW + k]) : 0.f;
    }
    float aw[TR][8], ab = 0.f;
#pragma unroll
    for (int j = 0; j < TR; j++)
#pragma unroll
        for (int e = 0; e < 8; e++) aw[j][e] = 0.f;
    for (int64_t r0 = (int64_t)blockIdx.x * kRows; r0 < n; r0 += (int64_t)gridDim.x * kRows) {
        __syncthreads();                             // the tile before is read
        if constexpr (K == 128) {
            for (int t = tid; t < kRows * 16; t += kThreads) {
                const int r = t >> 4, c = t & 15;
                const int64_t i = r0 + r;
                __align__(16) bf16 v[8];
                *reinterpret_cast<uint4 *>(v) = make_uint4(0u, 0u, 0u, 0u);
                if (i < n)
                    *reinterpret_cast<uint4 *>(v) = *reinterpret_cast<const uint4 *>(
                        (c < 8 ? X1 : X2) + i * kHid + (c & 7) * 8);
                float4 *dst = reinterpret_cast<float4 *>(Xs + r * K + c * 8);
                dst[0] = make_float4(to_f(v[0]), to_f(v[1]), to_f(v[2]), to_f(v[3]));
                dst[1] = make_float4(to_f(v[4]), to_f(v[5]), to_f(v[6]), to_f(v[7]));
            }
        } else {
            for (int t = tid; t < kRows * K; t += kThreads) {
                const int r = t / K, k = t % K;
                Xs[t] = r0 + r < n && k < F ? to_f(X1[(r0 + r) * F + k]) : 0.f;
            }
        }
        if (N == kHid && y) {
            for (int t = tid; t < kRows * 16; t += kThreads) {
                const int r = t >> 4, o = (t & 15) * 4;
                const int64_t i = r0 + r;
                float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                if (i < n) {
                    z = *reinterpret_cast<const float4 *>(dout + i * kHid + o);
                    __align__(8) bf16 v[4];
                    *reinterpret_cast<uint2 *>(v) = *reinterpret_cast<const uint2 *>(y + i * kHid + o);
                    const float y0 = to_f(v[0]), y1 = to_f(v[1]), y2 = to_f(v[2]), y3 = to_f(v[3]);
                    z.x *= 1.f - y0 * y0;
                    z.y *= 1.f - y1 * y1;
                    z.z *= 1.f - y2 * y2;
                    z.w *= 1.f - y3 * y3;
                }
                *reinterpret_cast<float4 *>(Zs + r * kZs + o) = z;
            }
        } else {
            for (int t = tid; t < kRows * kHid; t += kThreads) {
                const int r = t / kHid, o = t % kHid;
                Zs[r * kZs + o] = r0 + r < n && o < N ? dout[(r0 + r) * N + o] : 0.f;
            }
        }
        __syncthreads();
        if (dX1) {                                   // dX = dZ W
            float ax[TR][8];
#pragma unroll
            for (int j = 0; j < TR; j++)
#pragma unroll
                for (int e = 0; e < 8; e++) ax[j][e] = 0.f;
            for (int o = 0; o < N; o += 4) {
                float z[TR][4];
#pragma unroll
                for (int j = 0; j < TR; j++)
                    *reinterpret_cast<float4 *>(z[j]) =
                        *reinterpret_cast<const float4 *>(Zs + (rg * TR + j) * kZs + o);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    float wv[8];
                    *reinterpret_cast<float4 *>(wv) =
                        *reinterpret_cast<const float4 *>(Ws + (o + u) * K + 4 * cg);
                    *reinterpret_cast<float4 *>(wv + 4) =
                        *reinterpret_cast<const float4 *>(Ws + (o + u) * K + K / 2 + 4 * cg);
#pragma unroll
                    for (int j = 0; j < TR; j++)
#pragma unroll
                        for (int e = 0; e < 8; e++) ax[j][e] += z[j][u] * wv[e];
                }
            }
#pragma unroll
            for (int j = 0; j < TR; j++) {
                const int64_t i = r0 + rg * TR + j;
                if (i >= n) break;
                float *d0 = dX1 + i * kHid + 4 * cg;
                float *d1 = K == 128 ? dX2 + i * kHid + 4 * cg : d0 + 32;
                *reinterpret_cast<float4 *>(d0) = make_float4(ax[j][0], ax[j][1], ax[j][2], ax[j][3]);
                *reinterpret_cast<float4 *>(d1) = make_float4(ax[j][4], ax[j][5], ax[j][6], ax[j][7]);
            }
        }
        if (rg * TR < N)                             // dW += dZ^T x
#pragma unroll 4
            for (int r = 0; r < kRows; r++) {
                float z[TR], x[8];
                if constexpr (TR == 4)
                    *reinterpret_cast<float4 *>(z) =
                        *reinterpret_cast<const float4 *>(Zs + r * kZs + rg * TR);
                else
                    *reinterpret_cast<float2 *>(z) =
                        *reinterpret_cast<const float2 *>(Zs + r * kZs + rg * TR);
                *reinterpret_cast<float4 *>(x) =
                    *reinterpret_cast<const float4 *>(Xs + r * K + 4 * cg);
                *reinterpret_cast<float4 *>(x + 4) =
                    *reinterpret_cast<const float4 *>(Xs + r * K + K / 2 + 4 * cg);
#pragma unroll
                for (int j = 0; j < TR; j++)
#pragma unroll
                    for (int e = 0; e < 8; e++) aw[j][e] += z[j] * x[e];
            }
        for (int r = tid >> 6; r < kRows; r += kThreads >> 6) ab += Zs[r * kZs + (tid & 63)];
    }
    if ((tid & 63) < N) atomicAdd(db + (tid & 63), ab);
    if (KW == K) {
#pragma unroll
        for (int j = 0; j < TR; j++) {
            const int o = rg * TR + j;
            if (o >= N) break;
#pragma unroll
            for (int h = 0; h < 2; h++)
                atomicAdd(reinterpret_cast<float4 *>(dW + (size_t)o * K + h * (K / 2) + 4 * cg),
                          make_float4(aw[j][4 * h], aw[j][4 * h + 1], aw[j][4 * h + 2], aw[j][4 * h + 3]));
        }
        return;
    }
    // few columns: through shared memory, so that a warp's atomics are
    // consecutive (the same 128-byte lines for every block)
    __syncthreads();
#pragma unroll
    for (int j = 0; j < TR; j++)
#pragma unroll
        for (int e = 0; e < 8; e++)
            Ws[(rg * TR + j) * K + (e >> 2) * (K / 2) + 4 * cg + (e & 3)] = aw[j][e];
    __syncthreads();
    for (int t = tid; t < N * KW; t += kThreads) atomicAdd(dW + t, Ws[(t / KW) * K + t % KW]);
}

// ---- one message-passing layer on the tensor cores (tcgen05, TMEM
// accumulator), the messages gathered straight into the product's operand:
//   h'_i = tanh(b + W [h_i, sum_q w_q h_ci(q)]),   Y_i = bo + Wo h'_i (last layer)
// for 64 BF16 features a node.  With rp == nullptr only the output product is
// done, on h itself.
//
// One block of 8 warps takes 128 nodes:
//   * eight lanes take a node's row (16 bytes each).  They copy it into the
//     first half of A (128 x 64 BF16), read eight edges' indices and weights
//     at once, and with up to eight gathers in flight add the neighbours' rows
//     in FP32, in edge order; the sum, rounded to BF16, is the second half.
//     Rows of 128 bytes lie in the 128-byte swizzle (chunk c of row r at
//     c ^ (r & 7)), so that the eight lanes' stores take different banks.
//   * one thread issues 8 tcgen05.mma kind::f16 (M = 128, N = 64, K = 16) and
//     commits them to an mbarrier;
//   * each warp reads 32 TMEM lanes -- lane = node -- and 32 of the 64 columns,
//     applies bias and tanh, and puts the BF16 row back in the first half of
//     A, from where it is stored in whole rows and, in the last layer, is the
//     operand of the output product.
// The mbarrier wait is bounded: when it runs out, *err is set, the block
// waits (bounded) once more for its MMAs, frees its TMEM and stores nothing.
//
// What bounds it: the seven 128-byte rows a node reads from L2 (100 MB a layer
// at 48^3), then tanhf.  The messages and, where the caller does not train,
// the last activations never go to memory.  48^3 nodes: 27 us a layer
// against 29 for the messages and 32 for the dense part in launches of their
// own; the whole forward pass 301 -> 115 us.  Three blocks fit an SM (56 KB
// of shared memory each), enough for 24 warps of gathers while one block is
// in its epilogue.
constexpr int kTcRows = 128;
constexpr int kTcThreads = 256;
constexpr uint32_t kTcA = kTcRows * 128, kTcB = kHid * 128;   // bytes of a 64-column half
constexpr size_t kTcSmem = 1024 + 2 * kTcA + 3 * kTcB;        // + alignment of the base
constexpr long kTcSpin = 1L << 22;

SPX_DEV uint32_t sh_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor, K-major rows of 128 bytes in the 128-byte
// swizzle: start address and stride between 8-row groups (1024 bytes) in
// 16-byte units, descriptor version 1, swizzle mode 2; the leading offset is
// not used
SPX_DEV uint64_t umma_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}
// instruction descriptor of kind::f16: FP32 D (bits 4-5 = 1), BF16 A and B
// (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
constexpr uint32_t umma_idesc_bf16(int nn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nn >> 3) << 17) |
           ((uint32_t)(kTcRows >> 4) << 24);
}
SPX_DEV bool tc_bar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// byte offset of 16-byte chunk c of row r in a 64-column half
SPX_DEV uint32_t tc_off(int r, int c) {
    return (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u + (uint32_t)((c ^ (r & 7)) << 4);
}
// D (TMEM) = A B^T over `halves` pairs of 64-column halves, one thread
SPX_DEV void tc_mma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, int halves) {
    for (int j = 0; j < 4 * halves; j++) {
        const uint64_t da = umma_desc(a + (j >> 2) * kTcA + (j & 3) * 32u);
        const uint64_t db = umma_desc(b + (j >> 2) * kTcB + (j & 3) * 32u);
        const uint32_t acc = j > 0 ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
            ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
    }
}
SPX_DEV void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(bar) : "memory");
}
// shared-memory stores of all threads become visible to the tensor core
SPX_DEV void tc_operands_ready() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// bounded wait of the whole block; 0 when it ran out
SPX_DEV int tc_wait(uint32_t bar, uint32_t parity, volatile int *err) {
    bool done = false;
    for (long it = 0; it < kTcSpin && !done; it++) done = tc_bar_test(bar, parity);
    if (!done) {
        *err = 1;
        for (long it = 0; it < kTcSpin && !done; it++) done = tc_bar_test(bar, parity);
        done = false;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return __syncthreads_and(done ? 1 : 0);
}
// 16 columns of a warp's 32 TMEM lanes
SPX_DEV void tc_load16(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,"
        "%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
          "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(kTcThreads, 3)
layer_fwd_kernel(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                 const float *__restrict__ w, const bf16 *__restrict__ Hp, bf16 *__restrict__ M,
                 const bf16 *__restrict__ W, const float *__restrict__ b, bf16 *__restrict__ Hn,
                 int P, const bf16 *__restrict__ Wo, const float *__restrict__ bo,
                 float *__restrict__ Y, volatile int *err) {
    extern __shared__ unsigned char tc_sm[];
    spx::chain_begin();
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ float s_b[kHid], s_bo[kHid];
    unsigned char *sA = tc_sm + ((1024u - (sh_addr(tc_sm) & 1023u)) & 1023u);
    unsigned char *sB = sA + 2 * kTcA, *sBo = sB + 2 * kTcB;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NP = (P + 15) & ~15;
    const uint32_t ncols = Y ? 128u : 64u;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(sh_addr(&s_tmem)), "r"(ncols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sh_addr(&s_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    if (rp) {
        for (int t = tid; t < kHid * 16; t += kTcThreads) {
            const int o = t >> 4, c = t & 15;
            *reinterpret_cast<uint4 *>(sB + (c >> 3) * kTcB + tc_off(o, c & 7)) =
                *reinterpret_cast<const uint4 *>(W + o * 128 + c * 8);
        }
        if (tid < kHid) s_b[tid] = b[tid];
    }
    if (Y) {
        for (int t = tid; t < NP * 8; t += kTcThreads) {
            const int o = t >> 3, c = t & 7;
            *reinterpret_cast<uint4 *>(sBo + tc_off(o, c)) =
                o < P ? *reinterpret_cast<const uint4 *>(Wo + o * kHid + c * 8) : zero;
        }
        if (tid < P) s_bo[tid] = bo[tid];
    }
    const int64_t row0 = (int64_t)blockIdx.x * kTcRows;
    const int c = lane & 7, g0 = lane & 24;
    for (int p = 0; p < 4; p++) {
        const int r = warp * 16 + p * 4 + (lane >> 3);
        const int64_t i = row0 + r;
        const uint4 own = i < n ? *reinterpret_cast<const uint4 *>(Hp + i * kHid + c * 8) : zero;
        if (rp) {
            int q = i < n ? rp[i] : 0;
            const int q1 = i < n ? rp[i + 1] : 0;
            float acc[8];
#pragma unroll
            for (int e = 0; e < 8; e++) acc[e] = 0.f;
            for (; __any_sync(~0u, q < q1); q += 8) {
                const bool mine = q + c < q1;
                const int cq = mine ? ci[q + c] : -1;
                const float wq = mine ? w[q + c] : 0.f;
                uint4 v[8];
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    const int cc = __shfl_sync(~0u, cq, g0 + t);
                    v[t] = zero;
                    if (cc >= 0)
                        v[t] = *reinterpret_cast<const uint4 *>(Hp + (size_t)cc * kHid + c * 8);
                }
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    const float ww = __shfl_sync(~0u, wq, g0 + t);
                    const uint32_t u[4] = {v[t].x, v[t].y, v[t].z, v[t].w};
#pragma unroll
                    for (int e = 0; e < 4; e++) {   // BF16 is the upper half of FP32
                        acc[2 * e] += ww * __uint_as_float(u[e] << 16);
                        acc[2 * e + 1] += ww * __uint_as_float(u[e] & 0xFFFF0000u);
                    }
                }
            }
            __align__(16) bf16 m[8];
#pragma unroll
            for (int e = 0; e < 8; e++) m[e] = __float2bfloat16(acc[e]);
            const uint4 mv = *reinterpret_cast<const uint4 *>(m);
            *reinterpret_cast<uint4 *>(sA + kTcA + tc_off(r, c)) = mv;
            if (M && i < n) *reinterpret_cast<uint4 *>(M + i * kHid + c * 8) = mv;
        }
        *reinterpret_cast<uint4 *>(sA + tc_off(r, c)) = own;
    }
    tc_operands_ready();
    const uint32_t tmem = s_tmem, bar = sh_addr(&s_bar);
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int r = (warp & 3) * 32 + lane, half = warp >> 2;
    int ok = 1;
    uint32_t parity = 0;
    if (rp) {
        if (tid == 0) {
            tc_mma(tmem, sh_addr(sA), sh_addr(sB), umma_idesc_bf16(kHid), 2);
            tc_commit(bar);
        }
        ok = tc_wait(bar, parity, err);
        parity = 1;
        if (ok) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int c0 = half * 32 + h * 16;
                uint32_t d[16];
                tc_load16(lanes + (uint32_t)c0, d);
                __align__(16) bf16 v[16];
#pragma unroll
                for (int e = 0; e < 16; e++)
                    v[e] = __float2bfloat16(tanhf(__uint_as_float(d[e]) + s_b[c0 + e]));
#pragma unroll
                for (int u = 0; u < 2; u++)
                    *reinterpret_cast<uint4 *>(sA + tc_off(r, (c0 >> 3) + u)) =
                        *reinterpret_cast<const uint4 *>(v + 8 * u);
            }
            tc_operands_ready();
            if (Hn)
                for (int t = tid; t < kTcRows * 8; t += kTcThreads) {
                    const int64_t i = row0 + (t >> 3);
                    if (i < n)
                        *reinterpret_cast<uint4 *>(Hn + i * kHid + (t & 7) * 8) =
                            *reinterpret_cast<const uint4 *>(sA + tc_off(t >> 3, t & 7));
                }
        }
    }
    if (Y && ok) {
        if (tid == 0) {
            tc_mma(tmem + kHid, sh_addr(sA), sh_addr(sBo), umma_idesc_bf16(NP), 1);
            tc_commit(bar);
        }
        if (tc_wait(bar, parity, err)) {
            float *yrow = Y + (row0 + r) * P;
            for (int c0 = half * 16; c0 < NP; c0 += 32) {
                uint32_t d[16];
                tc_load16(lanes + (uint32_t)(kHid + c0), d);
                if (row0 + r >= n) continue;
#pragma unroll
                for (int h = 0; h < 4; h++) {       // P is a multiple of 4
                    const int o = c0 + 4 * h;
                    if (o >= P) break;
                    float4 v;
                    v.x = __uint_as_float(d[4 * h + 0]) + s_bo[o + 0];
                    v.y = __uint_as_float(d[4 * h + 1]) + s_bo[o + 1];
                    v.z = __uint_as_float(d[4 * h + 2]) + s_bo[o + 2];
                    v.w = __uint_as_float(d[4 * h + 3]) + s_bo[o + 3];
                    *reinterpret_cast<float4 *>(yrow + o) = v;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols)
                     : "memory");
}

// ---- the network's input graph on the device ---------------------------
// The normalised adjacency of the N^3 finite-volume operator from the cell
// conductivities kap (node i = (a0 N + a1) N + a2): the neighbours of i are
// i - N^2, i - N, i - 1, i + 1, i + N, i + N^2 (slots 0..5, ascending) where
// they lie in the grid; a face between a lower cell a and an upper cell b
// has t = 2 k_a k_b / (k_a + k_b); s_i = t_0 + ... + t_5 in slot order
// (absent slots 0); w_ij = t_ij / sqrt(s_i s_j) rounded to FP32.  These are
// the operations, in the same order, of the host construction, so the CSR
// is the same to the bit.
__global__ void grid_faces_kernel(int N, const double *__restrict__ kap, double *__restrict__ T,
                                  double *__restrict__ s, int32_t *__restrict__ deg) {
    const int64_t n = (int64_t)N * N * N;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int a0 = (int)(i / ((int64_t)N * N)), a1 = (int)((i / N) % N), a2 = (int)(i % N);
    const int64_t step[6] = {-(int64_t)N * N, -(int64_t)N, -1, 1, N, (int64_t)N * N};
    const bool in[6] = {a0 > 0, a1 > 0, a2 > 0, a2 < N - 1, a1 < N - 1, a0 < N - 1};
    const double ki = kap[i];
    double acc = 0.0;
    int d = 0;
#pragma unroll
    for (int j = 0; j < 6; j++) {
        double t = 0.0;
        if (in[j]) {
            const double kj = kap[i + step[j]];
            // slots 0-2: the neighbour is the lower cell; 3-5: this cell is
            t = j < 3 ? 2.0 * kj * ki / (kj + ki) : 2.0 * ki * kj / (ki + kj);
        }
        T[i * 6 + j] = t;
        acc += t;
        d += t > 0.0;
    }
    s[i] = acc;
    deg[i] = d;
}

__global__ void grid_fill_kernel(int N, const double *__restrict__ T, const double *__restrict__ s,
                                 const int32_t *__restrict__ rowptr, int32_t *__restrict__ col,
                                 float *__restrict__ w) {
    const int64_t n = (int64_t)N * N * N;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t step[6] = {-(int64_t)N * N, -(int64_t)N, -1, 1, N, (int64_t)N * N};
    int32_t q = rowptr[i];
    const double si = s[i];
#pragma unroll
    for (int j = 0; j < 6; j++) {
        const double t = T[i * 6 + j];
        if (t > 0.0) {
            const int64_t c = i + step[j];
            col[q] = (int32_t)c;
            w[q] = (float)(t / sqrt(si * s[c]));
            q++;
        }
    }
}

// ---- loss: G = Y^T Y (P x P, upper triangle), B = Y^T U (P x k), FP64 sums.
// The rows are converted once, on the way to shared memory (the conversions
// cost more than the FP64 FMAs when every product makes its own), and a
// thread sums a 2 x 2 piece.  32^3 nodes, P = 24, k = 16: 47.7 -> 21 us.
constexpr int kGramRows = 128;
__global__ void __launch_bounds__(kThreads)
gram_kernel(int n, int P, const float *__restrict__ Y, int k, const float *__restrict__ U,
            double *G, double *B) {
    extern __shared__ double2 gram_sm[];
    spx::chain_begin();
    double *S = reinterpret_cast<double *>(gram_sm);    // kGramRows x ld: [Y, U, 0]
    const int Q = P + k, ld = (Q + 1) & ~1;
    const int64_t r0 = (int64_t)blockIdx.x * kGramRows;
    for (int t = threadIdx.x; t < kGramRows * ld; t += kThreads) {
        const int r = t / ld, c = t - r * ld;
        double v = 0.0;
        if (r0 + r < n && c < Q) v = c < P ? Y[(r0 + r) * P + c] : U[(r0 + r) * k + (c - P)];
        S[t] = v;
    }
    __syncthreads();
    const int pa = (P + 1) >> 1, pc = ld >> 1;
    for (int t = threadIdx.x; t < pa * pc; t += kThreads) {
        const int ta = t / pc, tc = t - ta * pc;
        if (tc < ta) continue;                          // symmetric: upper part
        double s00 = 0.0, s01 = 0.0, s10 = 0.0, s11 = 0.0;
#pragma unroll 4
        for (int r = 0; r < kGramRows; r++) {
            const double2 x = *reinterpret_cast<const double2 *>(S + r * ld + 2 * ta);
            const double2 z = *reinterpret_cast<const double2 *>(S + r * ld + 2 * tc);
            s00 += x.x * z.x;
            s01 += x.x * z.y;
            s10 += x.y * z.x;
            s11 += x.y * z.y;
        }
        const double s[4] = {s00, s01, s10, s11};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int a = 2 * ta + (e >> 1), c = 2 * tc + (e & 1);
            if (a >= P || c >= Q || c < a) continue;
            atomicAdd(c < P ? G + a * P + c : B + a * k + (c - P), s[e]);
        }
    }
}

// C = (G + eps tr(G)/P I)^{-1} B by Cholesky in one block (P <= 64);
// loss = 1 - trace(B^T C) / k.  G holds its upper triangle.  A chain of P
// steps each way: the block updates the trailing part of a step together, and
// a warp takes a right-hand side with its entries in registers.  P = 24,
// k = 16: 367 -> 19 us against one thread.
constexpr int kSolveThreads = 512;
__global__ void __launch_bounds__(kSolveThreads)
small_solve_kernel(int P, int k, const double *__restrict__ G, const double *__restrict__ B,
                   float *__restrict__ C, double *loss) {
    constexpr int LD = 65;
    spx::chain_begin();
    __shared__ double L[64 * LD], s_inv[64];
    __shared__ double s_tr;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int t = tid; t < P * P; t += kSolveThreads) {
        const int c = t / P, a = t - c * P;             // a >= c: G(c, a) is stored
        if (a >= c) L[a * LD + c] = G[t];
    }
    if (tid == 0) s_tr = 0.0;
    __syncthreads();
    double tr = 0.0;
    for (int a = 0; a < P; a++) tr += L[a * LD + a];
    const double eps = 1e-8 * tr / P + 1e-300;
    __syncthreads();
    if (tid < P) L[tid * LD + tid] += eps;
    const int ti = tid >> 4, tj = tid & 15;             // 32 x 16 threads over the trailing part
    for (int j = 0; j < P; j++) {
        __syncthreads();
        const double d = L[j * LD + j];
        const double inv = 1.0 / sqrt(d > 0.0 ? d : 1e-300);
        if (tid == 0) s_inv[j] = inv;
        // the column is scaled on the fly (and for good by the row's thread)
        for (int a = j + 1 + ti; a < P; a += 32) {
            const double la = L[a * LD + j] * inv;
            for (int c = j + 1 + tj; c <= a; c += 16) L[a * LD + c] -= la * (L[c * LD + j] * inv);
        }
        __syncthreads();
        if (tid > j && tid < P) L[tid * LD + j] *= inv;
    }
    __syncthreads();
    for (int b = warp; b < k; b += kSolveThreads / 32) {
        const double b0 = lane < P ? B[lane * k + b] : 0.0;
        const double b1 = lane + 32 < P ? B[(lane + 32) * k + b] : 0.0;
        double s0 = b0, s1 = b1;
        for (int t = 0; t < P; t++) {
            const double z = __shfl_sync(~0u, t < 32 ? s0 : s1, t & 31) * s_inv[t];
            if (lane == t) s0 = z;
            else if (lane > t && lane < P) s0 -= L[lane * LD + t] * z;
            if (lane + 32 == t) s1 = z;
            else if (lane + 32 > t && lane + 32 < P) s1 -= L[(lane + 32) * LD + t] * z;
        }
        for (int t = P - 1; t >= 0; t--) {
            const double x = __shfl_sync(~0u, t < 32 ? s0 : s1, t & 31) * s_inv[t];
            if (lane == t) s0 = x;
            else if (lane < t) s0 -= L[t * LD + lane] * x;
            if (lane + 32 == t) s1 = x;
            else if (lane + 32 < t) s1 -= L[t * LD + lane + 32] * x;
        }
        if (lane < P) C[lane * k + b] = (float)s0;
        if (lane + 32 < P) C[(lane + 32) * k + b] = (float)s1;
        double v = lane < P ? b0 * s0 : 0.0;
        if (lane + 32 < P) v += b1 * s1;
        for (int o = 16; o; o >>= 1) v += __shfl_down_sync(~0u, v, o);
        if (lane == 0) atomicAdd(&s_tr, v);
    }
    __syncthreads();
    if (tid == 0) *loss = 1.0 - s_tr / k;
}

// dY[i, a] = -(2/k) sum_b (U[i, b] - sum_c Y[i, c] C[c, b]) C[a, b].  64 rows a
// block, one entry of the residual and then of dY a thread at a time, all of
// it in shared memory (with a thread a row its 64 residuals live in local
// memory and its reads are P floats apart).  32^3 nodes, P = 24, k = 16: 26
// -> 11.6 us.
__global__ void __launch_bounds__(kThreads)
dy_kernel(int n, int P, int k, const float *__restrict__ Y, const float *__restrict__ U,
          const float *__restrict__ C, float *__restrict__ dY) {
    extern __shared__ float dy_sm[];
    spx::chain_begin();
    const int lp = P | 1, lk = k | 1;
    float *Cs = dy_sm, *Ys = Cs + P * lk, *Es = Ys + kRows * lp;
    const int64_t r0 = (int64_t)blockIdx.x * kRows;
    const int rows = (int)min((int64_t)kRows, n - r0);
    for (int t = threadIdx.x; t < P * k; t += kThreads) Cs[(t / k) * lk + t % k] = C[t];
    for (int t = threadIdx.x; t < rows * P; t += kThreads) Ys[(t / P) * lp + t % P] = Y[r0 * P + t];
    __syncthreads();
    for (int t = threadIdx.x; t < rows * k; t += kThreads) {
        const int r = t / k, b = t - r * k;
        float s = U[r0 * k + t];
        for (int c = 0; c < P; c++) s -= Ys[r * lp + c] * Cs[c * lk + b];
        Es[r * lk + b] = s;
    }
    __syncthreads();
    const float sc = -2.f / k;
    for (int t = threadIdx.x; t < rows * P; t += kThreads) {
        const int r = t / P, a = t - r * P;
        float s = 0.f;
        for (int b = 0; b < k; b++) s += Es[r * lk + b] * Cs[a * lk + b];
        dY[r0 * P + t] = sc * s;
    }
}
size_t dy_smem(int P, int k) { return sizeof(float) * ((size_t)P * (k | 1) + (size_t)kRows * ((P | 1) + (k | 1))); }

// Adam on the FP32 weights, refreshing their BF16 copies
__global__ void adam_kernel(int64_t cnt, float *p, const float *g, float *m, float *v, float lr,
                            float b1, float b2, float c1, float c2, float eps, bf16 *pb) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cnt;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        p[i] = pi;
        pb[i] = __float2bfloat16(pi);
    }
}

__global__ void to_bf16_kernel(int64_t cnt, const float *src, bf16 *dst) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cnt;
         i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = __float2bfloat16(src[i]);
}

template <class T>
T *dalloc(size_t cnt) {
    void *p = nullptr;
    if (cudaMalloc(&p, (cnt ? cnt : 1) * sizeof(T)) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return (T *)p;
}

}  // namespace

struct speigs_mpnn_s {
    int F = 0, H = 64, L = 4, P = 0;
    int64_t nparam = 0;
    std::vector<int64_t> woff, boff;   // per layer (0 = input, 1..L, L+1 = output)
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
    bf16 *pb = nullptr;
    int64_t step = 0;
    int64_t ncap = 0;
    bf16 *Hs = nullptr, *Ms = nullptr;   // (L+1) x n x H, L x n x H
    float *Y = nullptr, *dY = nullptr, *dH = nullptr, *dH2 = nullptr, *dM = nullptr;
    double *G = nullptr, *loss = nullptr;
    float *C = nullptr;
    int kcap = 0;
    // dense layers of the forward pass on the tensor cores (tcgen05) where
    // their shapes allow it; 0 selects the FP32-FMA kernels throughout
    int tensor_cores = 1;
    // set by a tensor-core wait that ran out; mapped page-locked memory, so
    // the host reads it without synchronising the stream
    int *err_h = nullptr, *err_d = nullptr;
    // scratch of the device grid graph: face values (6 a node), node sums,
    // degrees and the scan's temporary storage
    double *gT = nullptr, *gs = nullptr;
    int32_t *gdeg = nullptr;
    void *gscan = nullptr;
    size_t gscan_bytes = 0;
    int64_t gcap = 0;
    ~speigs_mpnn_s() {
        void *ptrs[] = {p, g, m, v, pb, Hs, Ms, Y, dY, dH, dH2, dM, G, loss, C, gT, gs, gdeg, gscan};
        for (void *q : ptrs)
            if (q) cudaFree(q);
        if (err_h) cudaFreeHost(err_h);
    }
    int layer_in(int l) const { return l == 0 ? F : (l <= L ? 2 * H : H); }
    int layer_out(int l) const { return l <= L ? H : P; }
    int reserve(int64_t n, int k) {
        if (n <= ncap && k <= kcap) return 0;
        void *ptrs[] = {Hs, Ms, Y, dY, dH, dH2, dM, G, loss, C};
        for (void *q : ptrs)
            if (q) cudaFree(q);
        ncap = std::max(n, ncap);
        kcap = std::max(k, kcap);
        Hs = dalloc<bf16>((size_t)(L + 1) * ncap * H);
        Ms = dalloc<bf16>((size_t)L * ncap * H);
        Y = dalloc<float>((size_t)ncap * P);
        dY = dalloc<float>((size_t)ncap * P);
        dH = dalloc<float>((size_t)ncap * H);
        dH2 = dalloc<float>((size_t)ncap * H);
        dM = dalloc<float>((size_t)ncap * H);
        G = dalloc<double>((size_t)P * (P + std::max(kcap, 1)));   // [G, B]
        loss = dalloc<double>(1);
        C = dalloc<float>((size_t)P * std::max(kcap, 1));
        if (!Hs || !Ms || !Y || !dY || !dH || !dH2 || !dM || !G || !loss || !C)
            return SPEIGS_ERR_MEM;
        return 0;
    }
};

namespace {

size_t dense_smem(int K, int N) {
    return ((size_t)kRows * (K + 1) + (size_t)N * (K + 1)) * sizeof(float);
}
size_t input_smem(int F) { return sizeof(float) * ((size_t)F * kHid + (size_t)kInRows * (F + 1)); }

void set_smem_limits() {
    const auto a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const int big = 200 * 1024;
    cudaFuncSetAttribute(gram_kernel, a, big);
    cudaFuncSetAttribute(dy_kernel, a, big);
    cudaFuncSetAttribute(input_fwd_kernel, a, (int)input_smem(64));
    cudaFuncSetAttribute(dense_fwd_kernel<bf16>, a, big);
    cudaFuncSetAttribute(dense_fwd_kernel<float>, a, big);
    cudaFuncSetAttribute(dense_bwd_kernel<128, bf16>, a, (int)bwd_smem<128>());
    cudaFuncSetAttribute(dense_bwd_kernel<64, bf16>, a, (int)bwd_smem<64>());
    cudaFuncSetAttribute(dense_bwd_kernel<64, float>, a, (int)bwd_smem<64>());
    cudaFuncSetAttribute(layer_fwd_kernel, a, (int)kTcSmem);
}

bool aligned16(const void *q) { return ((uintptr_t)q & 15u) == 0; }

// forward pass; Y (FP32) in net->Y or, where it fits, straight into Yout.
// `keep` keeps what the backward pass reads: every layer's activations and
// messages.  The layers run on the tensor cores when the network allows it;
// the output layer where its rows are whole 16-byte pieces (P a multiple of
// 4), and then in the last layer's kernel.  Returns where Y is.
float *forward(speigs_mpnn_s *net, int n, const int32_t *rp, const int32_t *ci, const float *w,
               const float *X, float *Yout, bool keep, cudaStream_t st) {
    const int H = net->H, L = net->L, P = net->P;
    const int nb = (n + kRows - 1) / kRows, tb = (n + kTcRows - 1) / kTcRows;
    const bool tc = net->tensor_cores != 0, tco = tc && P % 4 == 0;
    float *Y = tco && !keep && aligned16(Yout) ? Yout : net->Y;
    const bf16 *Wo = net->pb + net->woff[L + 1];
    const float *bo = net->p + net->boff[L + 1];
    spx::launch_chained(input_fwd_kernel, (n + kInRows - 1) / kInRows, kThreads,
                        input_smem(net->F), st, n, net->F, X, net->pb + net->woff[0], net->p +
                        net->boff[0], net->Hs);
    for (int l = 1; l <= L; l++) {
        bf16 *Hp = net->Hs + (size_t)(l - 1) * n * H, *Hn = net->Hs + (size_t)l * n * H;
        bf16 *Ml = net->Ms + (size_t)(l - 1) * n * H;
        const bf16 *W = net->pb + net->woff[l];
        const float *b = net->p + net->boff[l];
        if (tc) {
            const bool last = l == L && tco;
            spx::launch_chained(layer_fwd_kernel, tb, kTcThreads, kTcSmem, st, n, rp, ci, w, Hp,
                                keep ? Ml : nullptr, W, b, last && !keep ? nullptr : Hn, P, Wo, bo,
                                last ? Y : nullptr, net->err_d);
        } else {
            spmm_kernel<<<(n + 7) / 8, 256, 0, st>>>(n, H, rp, ci, w, Hp, Ml);
            dense_fwd_kernel<bf16><<<nb, kThreads, dense_smem(2 * H, H), st>>>(n, H, Hp, H, Ml, H,
                                                                               W, b, 1, Hn);
            spx::note_launch(2);
        }
    }
    const bf16 *HL = net->Hs + (size_t)L * n * H;
    if (!tco)
        dense_fwd_kernel<float><<<nb, kThreads, dense_smem(H, P), st>>>(n, H, HL, 0, nullptr, P, Wo,
                                                                        bo, 0, Y);
    else if (L == 0)
        spx::launch_chained(layer_fwd_kernel, tb, kTcThreads, kTcSmem, st, n, nullptr, nullptr,
                            nullptr, HL, nullptr, nullptr, nullptr, nullptr, P, Wo, bo, Y,
                            net->err_d);
    if (!tco) spx::note_launch();
    return Y;
}

}  // namespace

extern "C" {

int speigs_b200_mpnn_create(int nfeat, int hidden, int layers, int nout, uint64_t seed,
                            speigs_mpnn *out) {
    if (!out || nfeat < 1 || nfeat > 64 || hidden != 64 || layers < 0 || layers > 8 || nout < 1 ||
        nout > 64)
        return SPEIGS_ERR_ARG;
    *out = nullptr;
    speigs_mpnn_s *net = new (std::nothrow) speigs_mpnn_s;
    if (!net) return SPEIGS_ERR_MEM;
    net->F = nfeat;
    net->H = hidden;
    net->L = layers;
    net->P = nout;
    int64_t off = 0;
    for (int l = 0; l <= layers + 1; l++) {
        net->woff.push_back(off);
        off += (int64_t)net->layer_out(l) * net->layer_in(l);
        net->boff.push_back(off);
        off += net->layer_out(l);
    }
    net->nparam = off;
    // Xavier-uniform weights from a seeded xorshift64* stream, zero biases
    std::vector<float> hp(off, 0.f);
    uint64_t s = seed ? seed : 88172645463325252ULL;
    auto uni = [&]() {
        s ^= s >> 12; s ^= s << 25; s ^= s >> 27;
        return (double)((s * 0x2545F4914F6CDD1DULL) >> 11) / 9007199254740992.0;
    };
    for (int l = 0; l <= layers + 1; l++) {
        const int fi = net->layer_in(l), fo = net->layer_out(l);
        const double a = std::sqrt(6.0 / (fi + fo)) * (l == layers + 1 ? 0.1 : 1.0);
        for (int64_t t = 0; t < (int64_t)fi * fo; t++) hp[net->woff[l] + t] = (float)((2.0 * uni() - 1.0) * a);
    }
    net->p = dalloc<float>(off);
    net->g = dalloc<float>(off);
    net->m = dalloc<float>(off);
    net->v = dalloc<float>(off);
    net->pb = dalloc<bf16>(off);
    if (!net->p || !net->g || !net->m || !net->v || !net->pb) { delete net; return SPEIGS_ERR_MEM; }
    cudaMemcpy(net->p, hp.data(), sizeof(float) * off, cudaMemcpyHostToDevice);
    cudaMemset(net->m, 0, sizeof(float) * off);
    cudaMemset(net->v, 0, sizeof(float) * off);
    cudaMemset(net->g, 0, sizeof(float) * off);
    to_bf16_kernel<<<64, 256>>>(off, net->p, net->pb);
    spx::note_launch();
    if (cudaHostAlloc((void **)&net->err_h, sizeof(int), cudaHostAllocMapped) != cudaSuccess ||
        cudaHostGetDevicePointer((void **)&net->err_d, net->err_h, 0) != cudaSuccess) {
        cudaGetLastError();
        delete net;
        return SPEIGS_ERR_MEM;
    }
    *net->err_h = 0;
    set_smem_limits();
    if (cudaDeviceSynchronize() != cudaSuccess) { cudaGetLastError(); delete net; return SPEIGS_ERR_INTERNAL; }
    *out = net;
    return SPEIGS_OK;
}

void speigs_b200_mpnn_destroy(speigs_mpnn net) { delete net; }

int speigs_b200_mpnn_grid_graph(speigs_mpnn net, int N, const double *kap, int32_t *rowptr,
                                int32_t *col, float *w, void *stream) {
    if (!net || N < 1 || (int64_t)N * N * N > INT32_MAX / 6 || !kap || !rowptr || !col || !w)
        return SPEIGS_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t n = (int64_t)N * N * N;
    if (n > net->gcap) {
        void *old[] = {net->gT, net->gs, net->gdeg, net->gscan};
        for (void *q : old)
            if (q) cudaFree(q);
        net->gT = dalloc<double>((size_t)n * 6);
        net->gs = dalloc<double>((size_t)n);
        net->gdeg = dalloc<int32_t>((size_t)n);
        net->gscan_bytes = 0;
        cub::DeviceScan::InclusiveSum(nullptr, net->gscan_bytes, net->gdeg, rowptr + 1, (int)n, st);
        net->gscan = net->gscan_bytes ? (void *)dalloc<unsigned char>(net->gscan_bytes) : nullptr;
        net->gcap = (net->gT && net->gs && net->gdeg && (net->gscan || !net->gscan_bytes)) ? n : 0;
        if (!net->gcap) return SPEIGS_ERR_MEM;
    }
    const int tb = 256, nb = (int)((n + tb - 1) / tb);
    grid_faces_kernel<<<nb, tb, 0, st>>>(N, kap, net->gT, net->gs, net->gdeg);
    cudaMemsetAsync(rowptr, 0, sizeof(int32_t), st);
    size_t tmp = net->gscan_bytes;
    cub::DeviceScan::InclusiveSum(net->gscan, tmp, net->gdeg, rowptr + 1, (int)n, st);
    grid_fill_kernel<<<nb, tb, 0, st>>>(N, net->gT, net->gs, rowptr, col, w);
    spx::note_launch(3);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { spx::set_last_error_text(cudaGetErrorString(e)); return SPEIGS_ERR_INTERNAL; }
    return SPEIGS_OK;
}

int speigs_b200_mpnn_tensor_cores(speigs_mpnn net, int on) {
    if (!net) return SPEIGS_ERR_ARG;
    const int was = net->tensor_cores;
    if (on >= 0) net->tensor_cores = on ? 1 : 0;
    return was;
}

int speigs_b200_mpnn_params(speigs_mpnn net, float *host, int64_t *count, int set) {
    if (!net || !count) return SPEIGS_ERR_ARG;
    if (!host) { *count = net->nparam; return SPEIGS_OK; }
    if (*count < net->nparam) return SPEIGS_ERR_ARG;
    if (set) {
        cudaMemcpy(net->p, host, sizeof(float) * net->nparam, cudaMemcpyHostToDevice);
        to_bf16_kernel<<<64, 256>>>(net->nparam, net->p, net->pb);
        spx::note_launch();
    } else {
        cudaMemcpy(host, net->p, sizeof(float) * net->nparam, cudaMemcpyDeviceToHost);
    }
    *count = net->nparam;
    return cudaDeviceSynchronize() == cudaSuccess ? SPEIGS_OK : SPEIGS_ERR_INTERNAL;
}

int speigs_b200_mpnn_grads(speigs_mpnn net, float *host) {
    if (!net || !host) return SPEIGS_ERR_ARG;
    cudaMemcpy(host, net->g, sizeof(float) * net->nparam, cudaMemcpyDeviceToHost);
    return cudaDeviceSynchronize() == cudaSuccess ? SPEIGS_OK : SPEIGS_ERR_INTERNAL;
}

int speigs_b200_mpnn_forward(speigs_mpnn net, int64_t n, const int32_t *rowptr, const int32_t *col,
                             const float *w, const float *X, float *Y, void *stream) {
    if (!net || n <= 0 || n > INT32_MAX || !rowptr || !col || !w || !X || !Y) return SPEIGS_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (*(volatile int *)net->err_h) {
        spx::set_last_error_text("mpnn: a tensor-core wait of an earlier call ran out");
        return SPEIGS_ERR_INTERNAL;
    }
    if (net->reserve(n, 1)) return SPEIGS_ERR_MEM;
    const float *at = forward(net, (int)n, rowptr, col, w, X, Y, false, st);
    if (at != Y)
        cudaMemcpyAsync(Y, at, sizeof(float) * (size_t)n * net->P, cudaMemcpyDeviceToDevice, st);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { spx::set_last_error_text(cudaGetErrorString(e)); return SPEIGS_ERR_INTERNAL; }
    return SPEIGS_OK;
}

int speigs_b200_mpnn_train_step(speigs_mpnn net, int64_t n, const int32_t *rowptr,
                                const int32_t *col, const float *w, const float *X,
                                const float *U, int k, float lr, double *loss, void *stream) {
    if (!net || n <= 0 || n > INT32_MAX || !rowptr || !col || !w || !X || !U || k < 1 || k > 64)
        return SPEIGS_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (net->reserve(n, k)) return SPEIGS_ERR_MEM;
    const int H = net->H, L = net->L, P = net->P, nn = (int)n;
    const int nb = (nn + kRows - 1) / kRows, sb = (nn + kThreads / 16 - 1) / (kThreads / 16);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int bb = std::min(nb, 2 * sms);               // two blocks fit an SM
    forward(net, nn, rowptr, col, w, X, nullptr, true, st);
    // loss and dL/dY
    double *G = net->G, *B = G + (size_t)P * P;
    cudaMemsetAsync(G, 0, sizeof(double) * (size_t)P * (P + k), st);
    spx::launch_chained(gram_kernel, (nn + kGramRows - 1) / kGramRows, kThreads, sizeof(double) *
                        kGramRows * ((P + k + 1) & ~1), st, nn, P, net->Y, k, U, G, B);
    spx::launch_chained(small_solve_kernel, 1, kSolveThreads, 0, st, P, k, G, B, net->C,
                        net->loss);
    spx::launch_chained(dy_kernel, nb, kThreads, dy_smem(P, k), st, nn, P, k, net->Y, U, net->C,
                        net->dY);
    // backward
    cudaMemsetAsync(net->g, 0, sizeof(float) * net->nparam, st);
    spx::launch_chained(dense_bwd_kernel<64, bf16>, bb, kThreads, bwd_smem<64>(), st, nn, H,
                        net->Hs + (size_t)L * nn * H, nullptr, P, net->pb + net->woff[L + 1],
                        nullptr, net->dY, net->dH, nullptr, net->g + net->woff[L + 1], net->g +
                        net->boff[L + 1]);
    for (int l = L; l >= 1; l--) {
        bf16 *Hp = net->Hs + (size_t)(l - 1) * nn * H, *Hn = net->Hs + (size_t)l * nn * H;
        bf16 *Ml = net->Ms + (size_t)(l - 1) * nn * H;
        // dH holds dL/dh_l; produce dL/dh_{l-1} (direct part) and dL/dm_l
        spx::launch_chained(dense_bwd_kernel<128, bf16>, bb, kThreads, bwd_smem<128>(), st, nn, 2 *
                            H, Hp, Ml, H, net->pb + net->woff[l], Hn, net->dH, net->dH2, net->dM,
                            net->g + net->woff[l], net->g + net->boff[l]);
        // dL/dh_{l-1} = direct part + A^T dL/dm_l (A symmetric)
        spx::launch_chained(spmm_add_kernel, sb, kThreads, 0, st, nn, rowptr, col, w, net->dM,
                            net->dH2);
        std::swap(net->dH, net->dH2);
    }
    spx::launch_chained(dense_bwd_kernel<64, float>, bb, kThreads, bwd_smem<64>(), st, nn, net->F,
                        X, nullptr, H, net->pb + net->woff[0], net->Hs, net->dH, nullptr, nullptr,
                        net->g + net->woff[0], net->g + net->boff[0]);
    if (lr > 0.f) {
        net->step++;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.f - powf(b1, (float)net->step), c2 = 1.f - powf(b2, (float)net->step);
        adam_kernel<<<256, 256, 0, st>>>(net->nparam, net->p, net->g, net->m, net->v, lr, b1, b2, c1,
                                         c2, 1e-8f, net->pb);
        spx::note_launch();
    }
    double hl = 0.0;
    cudaMemcpyAsync(&hl, net->loss, sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { spx::set_last_error_text(cudaGetErrorString(e)); return SPEIGS_ERR_INTERNAL; }
    if (*(volatile int *)net->err_h) {
        spx::set_last_error_text("mpnn: a tensor-core wait ran out");
        return SPEIGS_ERR_INTERNAL;
    }
    if (loss) *loss = hl;
    return SPEIGS_OK;
}

}  // extern "C"
