// Krylov-side kernels: FP64 CSR SpMV, tall-skinny Gram-Schmidt passes with a
// deterministic grid reduction, Ritz vectors and true residuals, the
// xorshift64* start vector with exact jump-ahead, and the one-block Jacobi
// eigensolver for the projected matrix.
//
// These replace the BLAS-1/2 and LAPACK calls of the reference's Lanczos
// (src/speigs_core.c): cholmod_l_sdmult in op_multA (:75-83), dgemv T/N in
// orth_block (:122-132), dnrm2/dscal/ddot (:189-191, :209, :223, :251-257),
// dgemv N for Ritz vectors (:250, :278), dsyev (:236) and rand_vec (:49-54).
#include "krylov.cuh"
#include "../chain.cuh"
#include "../common.cuh"
#include "../counters.h"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>

namespace spx {

// ------------------------------------------------------------------ SpMV --
// One block per 128 consecutive rows.  When the block's nonzeros fit in
// shared memory the products are formed with fully coalesced vector loads --
// a pair of values (16 bytes) and a pair of column indices (8 bytes) per
// thread and step, after at most one leading entry that puts the pairs on
// their 16-byte boundary -- and each thread then sums its own row from
// shared memory (CSR-stream); otherwise a warp walks each row.  Bound by the
// matrix's bytes, if enough loads are in flight: 100^3 grid, 7 entries a row
// (104 MB), 39 us with one pair at a time, 31 with four.
constexpr int kSpmvRows = 128;
constexpr int kSpmvCap = 2048;

__global__ void __launch_bounds__(kSpmvRows)
spmv_kernel(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
            const double *__restrict__ va, const double *__restrict__ x,
            double *__restrict__ y) {
    __shared__ double prod[kSpmvCap];
    chain_begin();
    const int r0 = blockIdx.x * kSpmvRows;
    const int r1 = min(r0 + kSpmvRows, n);
    const int p0 = rp[r0], p1 = rp[r1];
    const int cnt = p1 - p0;
    if (cnt <= kSpmvCap) {
        // entries [p0, p1): an odd p0 is done alone, then aligned pairs, then
        // an odd last entry alone
        const int head = p0 & 1;
        const int npair = (cnt - head) >> 1;
        if (threadIdx.x == 0 && head && cnt > 0) prod[0] = va[p0] * __ldg(x + ci[p0]);
        const double2 *va2 = reinterpret_cast<const double2 *>(va + p0 + head);
        const int2 *ci2 = reinterpret_cast<const int2 *>(ci + p0 + head);
        // four pairs a step: the matrix's loads and then the eight gathers of
        // x are in flight together
        for (int t0 = threadIdx.x; t0 < npair; t0 += 4 * kSpmvRows) {
            double2 v[4];
            int2 c[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int t = t0 + u * kSpmvRows;
                c[u] = make_int2(-1, -1);
                if (t < npair) {
                    v[u] = va2[t];
                    c[u] = ci2[t];
                }
            }
            double xa[4], xb[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (c[u].x >= 0) {
                    xa[u] = __ldg(x + c[u].x);
                    xb[u] = __ldg(x + c[u].y);
                }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int t = t0 + u * kSpmvRows;
                if (t < npair) {
                    prod[head + 2 * t] = v[u].x * xa[u];
                    prod[head + 2 * t + 1] = v[u].y * xb[u];
                }
            }
        }
        const int last = head + 2 * npair;
        if (threadIdx.x == 0 && last < cnt) prod[last] = va[p0 + last] * __ldg(x + ci[p0 + last]);
        __syncthreads();
        const int r = r0 + threadIdx.x;
        if (r < r1) {
            const int a = rp[r] - p0, b = rp[r + 1] - p0;
            double s = 0.0;
            for (int q = a; q < b; q++) s += prod[q];
            y[r] = s;
        }
    } else {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        for (int r = r0 + wid; r < r1; r += blockDim.x >> 5) {
            double s = 0.0;
            for (int q = rp[r] + lane; q < rp[r + 1]; q += 32) s += va[q] * __ldg(x + ci[q]);
            s = warp_sum(s);
            if (lane == 0) y[r] = s;
        }
    }
}

void launch_spmv(int n, const int32_t *rowptr, const int32_t *col, const double *val,
                 const double *x, double *y, cudaStream_t st) {
    if (n <= 0) return;
    int nb = (n + kSpmvRows - 1) / kSpmvRows;
    launch_chained(spmv_kernel, nb, kSpmvRows, 0, st, n, rowptr, col, val, x, y);
}

// ---------------------------------------------------------- tall-skinny --
constexpr int kTsThreads = 256;
constexpr int kTsRows = 2;       // rows per thread
constexpr int kTsChunk = 8;      // vectors per register chunk
constexpr int kTsMaxBlocks = 4 * 148;

static int ts_blocks(int n) {
    int nb = (n + kTsThreads * kTsRows - 1) / (kTsThreads * kTsRows);
    return nb < 1 ? 1 : nb;
}

enum { TS_DOT = 0, TS_UPDATE_DOT = 1, TS_UPDATE_NORM = 2, TS_NORM = 3 };

struct TsParams {
    const double *V;
    int64_t ldv;
    int n, m;
    double *w;
    const double *hin;
    double *out;      // h (m) or nrm2 (1)
    double *hcol;     // optional projected-matrix column
    int hmode;        // 0 none, 1 assign, 2 add
    double *part;
    unsigned *counter;
};

// Shared memory beyond what a kernel may have unasked, 48 KB for its static
// part (16 and 272 bytes in the kernels below) and the dynamic one together.
// What may be asked for belongs to the kernel and the process, so every call
// raises it to the same size, all that a block can have: with sizes of their
// own, one thread's call could lower another's before its launch.
constexpr size_t kSmemUnasked = 47 * 1024, kSmemMost = 227 * 1024 - 512;
template <class... P>
static void allow_smem(void (*kernel)(P...), size_t smem) {
    if (smem > kSmemUnasked)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMost);
}

// Final cross-block reduction by the last block to arrive: column c of the
// partials (nb values in a row for each column) is summed by one warp in a
// fixed order, so results are reproducible run to run.  A chain of one L2
// latency and the shuffles; with 512 partial sums added up by one thread the
// reduction of a single column took 5 us.
SPX_DEV void last_block_reduce(double *part, unsigned *counter, int ncols, double *out,
                               double *hcol, int hmode) {
    __shared__ bool am_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = atomicAdd(counter, 1u);
        am_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!am_last) return;
    __threadfence();
    const int nb = gridDim.x, lane = threadIdx.x & 31;
    for (int c = threadIdx.x >> 5; c < ncols; c += blockDim.x >> 5) {
        const double *q = part + (size_t)c * nb;
        double acc = 0.0;
        for (int b0 = lane; b0 < nb; b0 += 32 * 10) {
            double x[10];
#pragma unroll
            for (int u = 0; u < 10; u++) x[u] = b0 + 32 * u < nb ? __ldcg(q + b0 + 32 * u) : 0.0;
#pragma unroll
            for (int u = 0; u < 10; u++) acc += x[u];
        }
        const double t = warp_sum(acc);
        if (lane == 0) {
            out[c] = t;
            if (hmode == 1) hcol[c] = t;
            else if (hmode == 2) hcol[c] += t;
        }
    }
    if (threadIdx.x == 0) *counter = 0u;
}

// A block takes a contiguous range of rows (at most two blocks an SM, at least
// 512 rows), in segments of kGsSeg rows of w that it keeps in shared memory:
//   * the update w -= V h gives a thread two adjacent rows and eight columns'
//     loads at a time; when the segment has fewer pairs of rows than half the
//     threads, groups of threads split the columns;
//   * the dot products give a warp one column of a share of the segment, so
//     that no barrier stands between the loads of V: the lanes' sums are added
//     once a column and share, into a slot of its own (a fixed order, so the
//     result is reproducible).
// VEC: V and w are 16-byte aligned and ldv is even, so a pair is one load.
//
// Bound by reading V (once a launch; the dot products after an update find
// their segment in L2), for small n by launch, two dependent passes and the
// reduction over blocks.  With a barrier for every eight columns of 512 rows:
// 100^3 rows and 14 columns on average, dot 33.8, update and dot 30.9, update
// and norm 35.7 us; 46^3 rows 11.2, 8.7, 8.3.  Now 20.2,
// 30.3, 17.3 and 7.7, 8.9, 6.2.
constexpr int kGsThreads = 512;
constexpr int kGsWarps = kGsThreads / 32;
constexpr int kGsSeg = 4096;
constexpr int kGsMaxBlocks = 2 * 148;

template <bool VEC>
__device__ __forceinline__ double2 ts_ld2(const double *q, bool both) {
    if (!both) return make_double2(*q, 0.0);
    if (VEC) return *reinterpret_cast<const double2 *>(q);
    return make_double2(q[0], q[1]);
}

// sum over c in [c0, c1) of V(i, c) h[c] for the pair of rows at v
template <bool VEC>
__device__ __forceinline__ double2 ts_cols(const double *v, int64_t ldv, const double *hs, int c0,
                                           int c1, bool both) {
    double2 s = make_double2(0.0, 0.0);
    v += (size_t)c0 * ldv;
    int c = c0;
    for (; c + 8 <= c1; c += 8) {
        double2 x[8];
#pragma unroll
        for (int q = 0; q < 8; q++, v += ldv) x[q] = ts_ld2<VEC>(v, both);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            s.x += x[q].x * hs[c + q];
            s.y += x[q].y * hs[c + q];
        }
    }
    if (c + 4 <= c1) {
        double2 x[4];
#pragma unroll
        for (int q = 0; q < 4; q++, v += ldv) x[q] = ts_ld2<VEC>(v, both);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            s.x += x[q].x * hs[c + q];
            s.y += x[q].y * hs[c + q];
        }
        c += 4;
    }
    if (c < c1) {
        double2 x[3];
#pragma unroll
        for (int q = 0; q < 3; q++, v += ldv)
            x[q] = c + q < c1 ? ts_ld2<VEC>(v, both) : make_double2(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < 3; q++)
            if (c + q < c1) {
                s.x += x[q].x * hs[c + q];
                s.y += x[q].y * hs[c + q];
            }
    }
    return s;
}

// shares of a segment's rows for the dot products: enough items for the
// warps, at least 256 rows an item
__host__ __device__ inline int ts_shares(int m, int per) {
    const int q = (per < kGsSeg ? per : kGsSeg) / 256;
    return m > 64 ? 1 : (q < 1 ? 1 : (q > 4 ? 4 : q));
}

template <int MODE, bool VEC>
__global__ void __launch_bounds__(kGsThreads, 2) ts_kernel(TsParams p, int per) {
    extern __shared__ double2 ts_sm[];
    constexpr bool UPD = MODE == TS_UPDATE_DOT || MODE == TS_UPDATE_NORM;
    constexpr bool DOT = MODE == TS_DOT || MODE == TS_UPDATE_DOT;
    const int m = p.m, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ncols = DOT ? m : 1, shares = DOT ? ts_shares(m, per) : 1;
    double *ws = reinterpret_cast<double *>(ts_sm);     // kGsSeg rows of w
    double *hs = ws + kGsSeg;                           // m coefficients
    double *slot = hs + ((m + 1) & ~1);                 // ncols x shares
    __shared__ double red[32];
    chain_begin();
    if (UPD)
        for (int c = tid; c < m; c += kGsThreads) hs[c] = p.hin[c];
    if (DOT)
        for (int c = tid; c < m * shares; c += kGsThreads) slot[c] = 0.0;
    double sq = 0.0;
    const int64_t lo = min((int64_t)p.n, (int64_t)blockIdx.x * per);
    const int64_t hi = min((int64_t)p.n, lo + per);
    for (int64_t s0 = lo; s0 < hi; s0 += kGsSeg) {
        const int len = (int)min((int64_t)kGsSeg, hi - s0), pairs = (len + 1) >> 1;
        const double *V = p.V + s0;
        double *w = p.w + s0;
        __syncthreads();                                // hs, slot; the segment before is read
        if (!UPD) {
            for (int t = tid; t < pairs; t += kGsThreads) {
                const double2 x = ts_ld2<VEC>(w + 2 * t, 2 * t + 1 < len);
                if (DOT) *reinterpret_cast<double2 *>(ws + 2 * t) = x;
                else sq += x.x * x.x + x.y * x.y;
            }
        } else {
            int groups = 1;                             // > 1: partial sums at ws + 1024
            while (groups < 8 && 2 * groups * pairs <= kGsThreads) groups *= 2;
            auto finish = [&](int t, double2 s) {
                const bool both = 2 * t + 1 < len;
                double2 x = ts_ld2<VEC>(w + 2 * t, both);
                x.x -= s.x;
                x.y -= s.y;
                if (VEC && both) {
                    *reinterpret_cast<double2 *>(w + 2 * t) = x;
                } else {
                    w[2 * t] = x.x;
                    if (both) w[2 * t + 1] = x.y;
                }
                if (DOT) *reinterpret_cast<double2 *>(ws + 2 * t) = x;
                else sq += x.x * x.x + x.y * x.y;
            };
            for (int k = tid; k < groups * pairs; k += kGsThreads) {
                const int g = groups > 1 ? k / pairs : 0, t = k - g * pairs;
                const double2 s = ts_cols<VEC>(V + 2 * t, p.ldv, hs, m * g / groups,
                                               m * (g + 1) / groups, 2 * t + 1 < len);
                if (groups > 1) *reinterpret_cast<double2 *>(ws + 1024 + 2 * k) = s;
                else finish(t, s);
            }
            if (groups > 1) {
                __syncthreads();
                if (tid < pairs) {
                    double2 s = make_double2(0.0, 0.0);
                    for (int g = 0; g < groups; g++) {
                        const double2 v =
                            *reinterpret_cast<const double2 *>(ws + 1024 + 2 * (g * pairs + tid));
                        s.x += v.x;
                        s.y += v.y;
                    }
                    finish(tid, s);
                }
            }
        }
        if (DOT) {
            __syncthreads();
            const int part = ((len + shares - 1) / shares + 63) & ~63;
            for (int it = warp; it < m * shares; it += kGsWarps) {
                const int sh = it / m, c = it - sh * m;
                const int b = min(len, (sh + 1) * part);
                const double *v = V + (size_t)c * p.ldv;
                double acc[4] = {0.0, 0.0, 0.0, 0.0};
                int r = sh * part + 2 * lane;
                for (; r + 64 * 7 + 1 < b; r += 512) {
                    double2 x[8];
#pragma unroll
                    for (int q = 0; q < 8; q++) x[q] = ts_ld2<VEC>(v + r + 64 * q, true);
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const double2 y = *reinterpret_cast<const double2 *>(ws + r + 64 * q);
                        acc[q & 3] += x[q].x * y.x;
                        acc[q & 3] += x[q].y * y.y;
                    }
                }
                for (; r < b; r += 256) {
                    double2 x[4];
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        x[q] = r + 64 * q < b ? ts_ld2<VEC>(v + r + 64 * q, r + 64 * q + 1 < b)
                                              : make_double2(0.0, 0.0);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (r + 64 * q < b) {
                            const double2 y = *reinterpret_cast<const double2 *>(ws + r + 64 * q);
                            acc[q] += x[q].x * y.x;
                            acc[q] += x[q].y * y.y;
                        }
                }
                const double t = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
                if (lane == 0) slot[it] += t;
            }
        }
    }
    __syncthreads();
    if (DOT) {
        for (int c = tid; c < m; c += kGsThreads) {
            double t = 0.0;
            for (int sh = 0; sh < shares; sh++) t += slot[sh * m + c];
            p.part[(size_t)c * gridDim.x + blockIdx.x] = t;
        }
    } else {
        sq = block_sum(sq, red);
        if (tid == 0) p.part[blockIdx.x] = sq;
    }
    last_block_reduce(p.part, p.counter, ncols, p.out, p.hcol, p.hmode);
}

// Update and dot products in one read of V, for up to M columns: a thread holds
// its row of V in registers between the two and the columns' sums over its
// rows, which are added over the block once at the end.  100^3 rows, 14 columns
// on average: 30.3 us when the products read V again out of L2, 24 now (a
// solve of 47 steps and 3 restarts 11.05 -> 10.1 ms); at 64^3 rows, V in L2, the
// two are equal.  M: powers of two, the default basis size (20), and the widest
// whose sums fit the registers; 20 and 40 spill a few (36 bytes) all the same.
constexpr int kUdThreads = 256;
// blocks an SM that the registers allow
__host__ __device__ constexpr int ud_blocks(int M) { return M <= 8 ? 3 : M <= 20 ? 2 : 1; }
template <int M>
__global__ void __launch_bounds__(kUdThreads, ud_blocks(M))
ts_update_dot_kernel(TsParams p) {
    __shared__ double hs[M], slot[kUdThreads / 32][M];
    const int m = p.m, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    chain_begin();
    for (int c = tid; c < m; c += kUdThreads) hs[c] = p.hin[c];
    __syncthreads();
    double acc[M];
#pragma unroll
    for (int c = 0; c < M; c++) acc[c] = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * kUdThreads + tid; i < p.n;
         i += (int64_t)gridDim.x * kUdThreads) {
        const double *v = p.V + i;
        double x[M];
#pragma unroll
        for (int c = 0; c < M; c++) x[c] = c < m ? v[(size_t)c * p.ldv] : 0.0;
        double w = p.w[i], s = 0.0;
#pragma unroll
        for (int c = 0; c < M; c++)
            if (c < m) s += x[c] * hs[c];
        w -= s;
        p.w[i] = w;
#pragma unroll
        for (int c = 0; c < M; c++) acc[c] += x[c] * w;
    }
#pragma unroll
    for (int c = 0; c < M; c++) {
        if (c >= m) break;
        const double t = warp_sum(acc[c]);
        if (lane == 0) slot[warp][c] = t;
    }
    __syncthreads();
    for (int c = tid; c < m; c += kUdThreads) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < kUdThreads / 32; q++) t += slot[q][c];
        p.part[(size_t)c * gridDim.x + blockIdx.x] = t;
    }
    last_block_reduce(p.part, p.counter, m, p.out, p.hcol, p.hmode);
}
constexpr int kUdCols = 40;          // wider: the sums no longer fit the registers

static void update_dot_launch(const TsParams &p, cudaStream_t st) {
    // at least two rows a thread, and as many blocks as run at once
    auto launch = [&](void (*kernel)(TsParams), int M) {
        launch_chained(kernel, std::min(ts_blocks(p.n), ud_blocks(M) * 148), kUdThreads, 0, st, p);
    };
    if (p.m <= 8) launch(ts_update_dot_kernel<8>, 8);
    else if (p.m <= 16) launch(ts_update_dot_kernel<16>, 16);
    else if (p.m <= 20) launch(ts_update_dot_kernel<20>, 20);
    else if (p.m <= 32) launch(ts_update_dot_kernel<32>, 32);
    else launch(ts_update_dot_kernel<kUdCols>, kUdCols);
}

template <int MODE>
static void ts_launch(const TsParams &p, cudaStream_t st) {
    const int nb = std::min(ts_blocks(p.n), kGsMaxBlocks);
    const int per = (((p.n + nb - 1) / nb) + 1) & ~1;
    const int slots = MODE == TS_DOT || MODE == TS_UPDATE_DOT ? p.m * ts_shares(p.m, per) : 0;
    const size_t smem = sizeof(double) * ((size_t)kGsSeg + ((p.m + 1) & ~1) + slots);
    const bool vec = (((uintptr_t)p.V | (uintptr_t)p.w) & 15u) == 0 && p.ldv % 2 == 0;
    const auto kernel = vec ? ts_kernel<MODE, true> : ts_kernel<MODE, false>;
    allow_smem(kernel, smem);                           // from about 960 columns on
    launch_chained(kernel, nb, kGsThreads, smem, st, p, per);
}

void launch_ts_dot(const double *V, int64_t ldv, int n, int m, const double *w, double *h,
                   double *hcol, int hmode, const ReduceScratch &rs, cudaStream_t st) {
    if (m <= 0) return;
    TsParams p{V, ldv, n, m, const_cast<double *>(w), nullptr, h, hcol, hmode, rs.part, rs.counter};
    ts_launch<TS_DOT>(p, st);
}
void launch_ts_update_dot(const double *V, int64_t ldv, int n, int m, double *w,
                          const double *hin, double *h, double *hcol, int hmode,
                          const ReduceScratch &rs, cudaStream_t st) {
    if (m <= 0) return;
    TsParams p{V, ldv, n, m, w, hin, h, hcol, hmode, rs.part, rs.counter};
    if (m <= kUdCols) update_dot_launch(p, st);
    else ts_launch<TS_UPDATE_DOT>(p, st);
}
void launch_ts_update_norm(const double *V, int64_t ldv, int n, int m, double *w,
                           const double *hin, double *nrm2, const ReduceScratch &rs,
                           cudaStream_t st) {
    TsParams p{V, ldv, n, m, w, hin, nrm2, nullptr, 0, rs.part, rs.counter};
    if (m <= 0) ts_launch<TS_NORM>(p, st);
    else ts_launch<TS_UPDATE_NORM>(p, st);
}
void launch_ts_norm(int n, const double *w, double *nrm2, const ReduceScratch &rs,
                    cudaStream_t st) {
    TsParams p{nullptr, 0, n, 0, const_cast<double *>(w), nullptr, nrm2, nullptr, 0, rs.part,
               rs.counter};
    ts_launch<TS_NORM>(p, st);
}

__global__ void scale_invnorm_kernel(int n, const double *src, const double *nrm2, double *dst) {
    chain_begin();
    const double s = 1.0 / sqrt(nrm2[0]);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        dst[i] = src[i] * s;
}
void launch_scale_by_invnorm(int n, const double *src, const double *nrm2, double *dst,
                             cudaStream_t st) {
    int nb = std::min(4096, (n + 255) / 256);
    launch_chained(scale_invnorm_kernel, std::max(nb, 1), 256, 0, st, n, src, nrm2, dst);
}

// ------------------------------------------------------ Ritz / residual --
struct RitzParams {
    const double *V;
    int64_t ldv;
    int n, m;
    const double *S;
    int lds;
    const int *idx;
    int idx_off, nvec;
    double *X;
    int64_t ldx;
    double *nrm2;
    double *part;
    unsigned *counter;
};

// A thread takes two adjacent rows and eight vectors at a time, with four
// columns' loads in flight; a block loops over 512-row segments (at most four
// blocks an SM) and adds its squared norms up per warp, with one barrier at
// the end.  Bound by reading V once for every eight vectors (out of L2 after
// the first).  20 columns, 6 vectors at 100^3 rows: 120 -> 56 us (two rows of
// separate loads, one column in flight and a barrier a vector before).
template <bool VEC>
__global__ void __launch_bounds__(kTsThreads) ritz_kernel(RitzParams p) {
    extern __shared__ double2 ritz_sm[];
    chain_begin();
    const int m = p.m, nv = p.nvec, nvp = (nv + kTsChunk - 1) & ~(kTsChunk - 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    double *Ss = reinterpret_cast<double *>(ritz_sm);  // m x nvp, a column's vectors adjacent
    double *slot = Ss + (size_t)m * nvp;               // warps x nvp
    for (int t = tid; t < m * nvp; t += kTsThreads) {
        const int c = t / nvp, v = t - c * nvp;
        Ss[t] = v < nv ? p.S[(size_t)p.idx[p.idx_off + v] * p.lds + c] : 0.0;
    }
    for (int t = tid; t < (kTsThreads / 32) * nvp; t += kTsThreads) slot[t] = 0.0;
    __syncthreads();
    constexpr int kSeg = kTsThreads * kTsRows;
    for (int64_t base = (int64_t)blockIdx.x * kSeg; base < p.n; base += (int64_t)gridDim.x * kSeg) {
        const int64_t i = base + 2 * tid;
        const bool any = i < p.n, both = i + 1 < p.n;
        const double *v0p = p.V + i;
        for (int v0 = 0; v0 < nv; v0 += kTsChunk) {
            double a0[kTsChunk], a1[kTsChunk];
#pragma unroll
            for (int q = 0; q < kTsChunk; q++) a0[q] = a1[q] = 0.0;
            if (any)
                for (int c0 = 0; c0 < m; c0 += 4) {
                    double2 x[4];
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (c0 + u < m) x[u] = ts_ld2<VEC>(v0p + (size_t)(c0 + u) * p.ldv, both);
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (c0 + u < m) {
                            const double *s = Ss + (size_t)(c0 + u) * nvp + v0;
#pragma unroll
                            for (int q = 0; q < kTsChunk; q += 2) {
                                const double2 sv = *reinterpret_cast<const double2 *>(s + q);
                                a0[q] += x[u].x * sv.x;
                                a1[q] += x[u].y * sv.x;
                                a0[q + 1] += x[u].x * sv.y;
                                a1[q + 1] += x[u].y * sv.y;
                            }
                        }
                }
#pragma unroll
            for (int q = 0; q < kTsChunk; q++) {
                if (v0 + q >= nv) break;
                if (any) {
                    double *x = p.X + (size_t)(v0 + q) * p.ldx + i;
                    if (VEC && both) {
                        *reinterpret_cast<double2 *>(x) = make_double2(a0[q], a1[q]);
                    } else {
                        x[0] = a0[q];
                        if (both) x[1] = a1[q];
                    }
                }
                double t = any ? a0[q] * a0[q] : 0.0;
                if (both) t += a1[q] * a1[q];
                t = warp_sum(t);
                if (lane == 0) slot[warp * nvp + v0 + q] += t;
            }
        }
    }
    __syncthreads();
    for (int v = tid; v < nv; v += kTsThreads) {
        double t = 0.0;
        for (int q = 0; q < kTsThreads / 32; q++) t += slot[q * nvp + v];
        p.part[(size_t)v * gridDim.x + blockIdx.x] = t;
    }
    last_block_reduce(p.part, p.counter, nv, p.nrm2, nullptr, 0);
}

void launch_ritz_vectors(const double *V, int64_t ldv, int n, int m, const double *S, int lds,
                         const int *idx, int idx_off, int nvec, double *X, int64_t ldx,
                         double *nrm2, const ReduceScratch &rs, cudaStream_t st) {
    if (nvec <= 0) return;
    // vectors per launch: the m x nv block of S and the warps' sums fit 48 KB
    // of shared memory, but at least one chunk of eight (opting in to more
    // where m is above 760)
    const int cap = std::max(kTsChunk, 6144 / (m + 8) / kTsChunk * kTsChunk);
    const bool vec = (((uintptr_t)V | (uintptr_t)X) & 15u) == 0 && ldv % 2 == 0 && ldx % 2 == 0;
    for (int v0 = 0; v0 < nvec; v0 += cap) {
        const int nv = std::min(cap, nvec - v0), nvp = (nv + kTsChunk - 1) & ~(kTsChunk - 1);
        RitzParams p{V, ldv, n, m, S, lds, idx, idx_off + v0, nv, X + (size_t)v0 * ldx, ldx,
                     nrm2 + v0, rs.part, rs.counter};
        const int nb = std::min(ts_blocks(n), kTsMaxBlocks);
        const size_t smem = sizeof(double) * (size_t)(m + kTsThreads / 32) * nvp;
        const auto kernel = vec ? ritz_kernel<true> : ritz_kernel<false>;
        allow_smem(kernel, smem);
        launch_chained(kernel, nb, kTsThreads, smem, st, p);
    }
}

__global__ void scale_cols_kernel(int n, int nvec, double *X, int64_t ldx, const double *nrm2) {
    chain_begin();
    const int v = blockIdx.y;
    const double q = nrm2[v];
    if (!(q > 0.0)) return;
    const double s = 1.0 / sqrt(q);
    double *x = X + (size_t)v * ldx;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x[i] *= s;
}
void launch_scale_cols(int n, int nvec, double *X, int64_t ldx, const double *nrm2,
                       cudaStream_t st) {
    if (nvec <= 0) return;
    int nb = std::max(1, std::min(1024, (n + 255) / 256));
    launch_chained(scale_cols_kernel, dim3(nb, nvec), 256, 0, st, n, nvec, X, ldx, nrm2);
}

struct RqParams {
    int n, nvec;
    const double *X;
    int64_t ldx;
    const double *AX;
    int64_t ldax;
    double *lam, *r2;
    int pass;
    double *part;
    unsigned *counter;
};

// Four rows a thread and vector in flight, blocks over all rows (at most four
// an SM), one barrier at the end.  Bound by reading X and AX.  6 vectors of
// 100^3 rows: 37 -> 21 us a pass (a barrier for every vector of 512 rows
// before).
__global__ void __launch_bounds__(kTsThreads) rq_kernel(RqParams p) {
    extern __shared__ double sh[];
    constexpr int kWarps = kTsThreads / 32;
    double *slot = sh;
    chain_begin();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t step = (int64_t)gridDim.x * kTsThreads;
    for (int v = 0; v < p.nvec; v++) {
        const double *x = p.X + (size_t)v * p.ldx, *ax = p.AX + (size_t)v * p.ldax;
        const double lam = (p.pass == 1) ? p.lam[v] : 0.0;
        double acc = 0.0;
        for (int64_t i0 = (int64_t)blockIdx.x * kTsThreads + threadIdx.x; i0 < p.n; i0 += 4 * step) {
            double a[4], b[4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int64_t i = i0 + r * step;
                a[r] = i < p.n ? x[i] : 0.0;
                b[r] = i < p.n ? ax[i] : 0.0;
            }
#pragma unroll
            for (int r = 0; r < 4; r++) {
                if (i0 + r * step >= p.n) break;
                if (p.pass == 0) acc += a[r] * b[r];
                else { const double d = b[r] - lam * a[r]; acc += d * d; }
            }
        }
        acc = warp_sum(acc);
        if (lane == 0) slot[v * kWarps + warp] = acc;
    }
    __syncthreads();
    for (int v = threadIdx.x; v < p.nvec; v += kTsThreads) {
        double t = 0.0;
        for (int q = 0; q < kWarps; q++) t += slot[v * kWarps + q];
        p.part[(size_t)v * gridDim.x + blockIdx.x] = t;
    }
    last_block_reduce(p.part, p.counter, p.nvec, p.pass == 0 ? p.lam : p.r2, nullptr, 0);
}

void launch_rayleigh_resid(int n, int nvec, const double *X, int64_t ldx, const double *AX,
                           int64_t ldax, double *lam, double *r2, const ReduceScratch &rs,
                           cudaStream_t st) {
    const int cap = 512;                 // vectors per launch: 32 KB of warps' sums
    for (int v0 = 0; v0 < nvec; v0 += cap) {
        const int nv = std::min(cap, nvec - v0);
        const int nb = std::min(ts_blocks(n), kTsMaxBlocks);
        const size_t smem = sizeof(double) * (size_t)nv * (kTsThreads / 32);
        for (int pass = 0; pass < 2; pass++) {
            RqParams p{n, nv, X + (size_t)v0 * ldx, ldx, AX + (size_t)v0 * ldax, ldax, lam + v0,
                       r2 + v0, pass, rs.part, rs.counter};
            launch_chained(rq_kernel, nb, kTsThreads, smem, st, p);
        }
    }
}

// ------------------------------------------------------- refinement ------
// One block per 128 rows (the SpMV layout above); per-block partial sums of
// ||r||^2, ||y||^2 and ||b||^2 are reduced by the last block to arrive, in a
// fixed order, which then takes the convergence decision.
__global__ void __launch_bounds__(kSpmvRows)
refine_residual_kernel(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                       const double *__restrict__ va, double shift, const double *__restrict__ b,
                       const double *__restrict__ y, double *__restrict__ r, double tol,
                       double anorm, int *flag, int *count, double *part, unsigned *counter) {
    __shared__ double red[32];
    __shared__ double fin[3 * kSpmvRows];
    __shared__ bool am_last;
    if (*(volatile const int *)flag) return;
    const int row = blockIdx.x * kSpmvRows + threadIdx.x;
    double r2 = 0.0, y2 = 0.0, b2 = 0.0;
    if (row < n) {
        double s = 0.0;
        for (int q = rp[row]; q < rp[row + 1]; q++) s += va[q] * __ldg(y + ci[q]);
        const double yi = y[row], bi = b[row];
        const double ri = bi - s - shift * yi;
        r[row] = ri;
        r2 = ri * ri;
        y2 = yi * yi;
        b2 = bi * bi;
    }
    r2 = block_sum(r2, red);
    y2 = block_sum(y2, red);
    b2 = block_sum(b2, red);
    if (threadIdx.x == 0) {
        part[(size_t)blockIdx.x * 3 + 0] = r2;
        part[(size_t)blockIdx.x * 3 + 1] = y2;
        part[(size_t)blockIdx.x * 3 + 2] = b2;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) am_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!am_last) return;
    __threadfence();
    // fixed-order reduction: thread t sums blocks t, t+128, ... per column
    for (int c = 0; c < 3; c++) {
        double acc = 0.0;
        for (int bk = threadIdx.x; bk < (int)gridDim.x; bk += blockDim.x)
            acc += ((volatile double *)part)[(size_t)bk * 3 + c];
        fin[c * kSpmvRows + threadIdx.x] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t[3] = {0.0, 0.0, 0.0};
        for (int c = 0; c < 3; c++)
            for (int i = 0; i < (int)blockDim.x; i++) t[c] += fin[c * kSpmvRows + i];
        if (sqrt(t[0]) <= tol * (anorm * sqrt(t[1]) + sqrt(t[2]))) *flag = 1;
        else *count += 1;
        *counter = 0u;
    }
}

void launch_refine_residual(int n, const int32_t *rowptr, const int32_t *col, const double *val,
                            double shift, const double *b, const double *y, double *r,
                            double tol, double anorm, int *flag, int *count,
                            const ReduceScratch &rs, cudaStream_t st) {
    const int nb = (n + kSpmvRows - 1) / kSpmvRows;
    refine_residual_kernel<<<nb, kSpmvRows, 0, st>>>(n, rowptr, col, val, shift, b, y, r, tol,
                                                     anorm, flag, count, rs.part, rs.counter);
    note_launch();
}

__global__ void axpy_unless_kernel(int n, double *y, const double *d, const int *flag) {
    if (*(volatile const int *)flag) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        y[i] += d[i];
}
void launch_axpy_unless(int n, double *y, const double *d, const int *flag, cudaStream_t st) {
    const int nb = std::max(1, std::min(4096, (n + 255) / 256));
    axpy_unless_kernel<<<nb, 256, 0, st>>>(n, y, d, flag);
    note_launch();
}

// ------------------------------------------------------------ RNG ------
// xorshift64* (reference src/speigs_core.c:49-54).  The state update is
// linear over GF(2), so the state after s steps is M^s applied to the seed;
// the 64 matrices M^(2^b) are tabulated once on the host.
struct JumpTable {
    uint64_t col[64][64];   // col[b][j] = M^(2^b) e_j
};

static uint64_t xs_step(uint64_t x) {
    x ^= x >> 12; x ^= x << 25; x ^= x >> 27;
    return x;
}
static uint64_t apply_mat(const uint64_t *col, uint64_t x) {
    uint64_t y = 0;
    for (int j = 0; j < 64; j++) if ((x >> j) & 1ull) y ^= col[j];
    return y;
}
static const JumpTable &jump_table() {
    static JumpTable T;
    static std::once_flag once;
    std::call_once(once, [] {
        for (int j = 0; j < 64; j++) T.col[0][j] = xs_step(1ull << j);
        for (int b = 1; b < 64; b++)
            for (int j = 0; j < 64; j++) T.col[b][j] = apply_mat(T.col[b - 1], T.col[b - 1][j]);
    });
    return T;
}

const uint64_t *rng_jump_table() { return &jump_table().col[0][0]; }

uint64_t rng_advance(uint64_t seed, uint64_t steps) {
    const JumpTable &T = jump_table();
    for (int b = 0; b < 64; b++)
        if ((steps >> b) & 1ull) seed = apply_mat(T.col[b], seed);
    return seed;
}

constexpr int kRngChunk = 64;

// memory pool of the device (engine.cu): allocations are cached across calls
cudaMemPool_t device_pool(int dev);

__global__ void rand_vec_kernel(int n, uint64_t seed, const uint64_t *__restrict__ jt,
                                double *v) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t first = (int64_t)g * kRngChunk;
    if (first >= n) return;
    uint64_t s = seed;
    uint64_t steps = (uint64_t)first;
    for (int b = 0; steps; b++, steps >>= 1) {
        if (!(steps & 1ull)) continue;
        const uint64_t *col = jt + (size_t)b * 64;
        uint64_t y = 0;
        for (int j = 0; j < 64; j++) y ^= col[j] & (0ull - ((s >> j) & 1ull));
        s = y;
    }
    const int64_t last = min((int64_t)n, first + kRngChunk);
    for (int64_t i = first; i < last; i++) {
        s ^= s >> 12; s ^= s << 25; s ^= s >> 27;
        const uint64_t out = s * 0x2545F4914F6CDD1DULL;
        v[i] = (double)(out >> 11) / 9007199254740992.0 - 0.5;
    }
}

void launch_rand_vec(int n, uint64_t seed, double *v, cudaStream_t st) {
    // the jump table travels with the launch as a small device copy that is
    // owned by this call (no global device state)
    const JumpTable &T = jump_table();
    // (from the library's pool, which keeps its memory: CUDA's default pool
    // returns freed memory to the driver at every synchronisation, and
    // mapping it again on the next call can take milliseconds)
    uint64_t *dj = nullptr;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaMemPool_t pool = device_pool(dev);
    cudaError_t ea = pool ? cudaMallocFromPoolAsync((void **)&dj, sizeof(T.col), pool, st)
                          : cudaMallocAsync((void **)&dj, sizeof(T.col), st);
    if (ea != cudaSuccess) { cudaGetLastError(); return; }
    cudaMemcpyAsync(dj, T.col, sizeof(T.col), cudaMemcpyHostToDevice, st);
    note_h2d(sizeof(T.col));
    int threads = (n + kRngChunk - 1) / kRngChunk;
    int nb = (threads + 127) / 128;
    rand_vec_kernel<<<std::max(nb, 1), 128, 0, st>>>(n, seed, dj, v);
    note_launch();
    cudaFreeAsync(dj, st);
}

// -------------------------------------------------- projected eigenproblem --
// Parallel cyclic Jacobi (round-robin pairing, m/2 rotations per round) on
// the symmetric matrix given by the upper triangle of H, in one block.
// Rotation angles follow Rutishauser's formulas; a pair is skipped when
// |a_pq| <= eps * sqrt(|a_pp| |a_qq|), which keeps small eigenvalues
// relatively accurate.  Finishes with eigenvalues ascending (the order dsyev
// returns) and an index list by |theta| descending, stable among ties.
constexpr int kJacThreads = 256;

__device__ void jacobi_body(int m, const double *__restrict__ H, int ldh, double *theta,
                            double *Sout, int *ord, double *gwork, int *status, int use_smem) {
    extern __shared__ double sm[];
    const int me = (m + 1) & ~1;              // even size (a dummy index when m is odd)
    const int half = me / 2;
    double *A, *V, *cs, *sn;
    int *pos;
    if (use_smem) {
        A = sm; V = A + (size_t)me * me;
        cs = V + (size_t)me * me;
    } else {
        A = gwork; V = gwork + (size_t)me * me;
        cs = sm;
    }
    sn = cs + half;
    pos = (int *)(sn + half);
    int *flags = pos + me;                    // [0]: rotated in this sweep
    for (int t = threadIdx.x; t < me * me; t += blockDim.x) {
        int i = t % me, j = t / me;
        double a = 0.0;
        if (i < m && j < m) a = (i <= j) ? H[i + (size_t)j * ldh] : H[j + (size_t)i * ldh];
        A[t] = a;
        V[t] = (i == j) ? 1.0 : 0.0;
    }
    __syncthreads();
    // round-robin pairing: index 0 stays, the others shift by one per round,
    // so in round r position t >= 1 holds 1 + ((t - 1 - r) mod (me - 1));
    // phase 1 of a round stores pair pi as (pos[pi], pos[half + pi]), p < q
    auto slot = [&](int t, int r) {
        if (t == 0) return 0;
        int x = t - 1 - r;             // in (-(me - 1), me - 1)
        if (x < 0) x += me - 1;
        return 1 + x;
    };
    int sweep = 0;
    const int max_sweeps = 60;
    for (; sweep < max_sweeps; sweep++) {
        if (threadIdx.x == 0) flags[0] = 0;
        __syncthreads();
        for (int round = 0; round < me - 1; round++) {
            // 1. rotation parameters for every disjoint pair
            for (int pi = threadIdx.x; pi < half; pi += blockDim.x) {
                int p = slot(pi, round), q = slot(me - 1 - pi, round);
                if (p > q) { int t = p; p = q; q = t; }
                pos[pi] = p;
                pos[half + pi] = q;
                double c = 1.0, s = 0.0;
                if (q < m) {
                    const double apq = A[p + (size_t)q * me];
                    const double app = A[p + (size_t)p * me], aqq = A[q + (size_t)q * me];
                    const double thr = DBL_EPSILON * 0.5 * sqrt(fabs(app)) * sqrt(fabs(aqq));
                    if (fabs(apq) > thr && apq != 0.0) {
                        const double th = (aqq - app) / (2.0 * apq);
                        double t;
                        if (fabs(th) > 1e150) t = 0.5 / th;
                        else t = (th >= 0.0 ? 1.0 : -1.0) / (fabs(th) + sqrt(1.0 + th * th));
                        c = 1.0 / sqrt(1.0 + t * t);
                        s = t * c;
                        flags[0] = 1;
                    }
                }
                cs[pi] = c; sn[pi] = s;
            }
            __syncthreads();
            // 2. A <- J^T A J as 2 x 2 blocks (row pair P, column pair Q; the
            // blocks are disjoint, and each is rotated by columns first, then
            // by rows), and V <- V J
            for (int t = threadIdx.x; t < half * half; t += blockDim.x) {
                const int P = t % half, Q = t / half;
                const double c1 = cs[P], s1 = sn[P], c2 = cs[Q], s2 = sn[Q];
                if (s1 == 0.0 && s2 == 0.0) continue;
                const int p1 = pos[P], q1 = pos[half + P], p2 = pos[Q], q2 = pos[half + Q];
                double *a11 = A + p1 + (size_t)p2 * me, *a12 = A + p1 + (size_t)q2 * me;
                double *a21 = A + q1 + (size_t)p2 * me, *a22 = A + q1 + (size_t)q2 * me;
                const double b11 = c2 * *a11 - s2 * *a12, b12 = s2 * *a11 + c2 * *a12;
                const double b21 = c2 * *a21 - s2 * *a22, b22 = s2 * *a21 + c2 * *a22;
                *a11 = c1 * b11 - s1 * b21;
                *a21 = s1 * b11 + c1 * b21;
                *a12 = c1 * b12 - s1 * b22;
                *a22 = s1 * b12 + c1 * b22;
                if (P == Q && s1 != 0.0) { *a12 = 0.0; *a21 = 0.0; }   // exactly decoupled
            }
            for (int t = threadIdx.x; t < half * me; t += blockDim.x) {
                const int Q = t / me, k = t % me;
                const double c = cs[Q], s = sn[Q];
                if (s == 0.0) continue;
                const int p = pos[Q], q = pos[half + Q];
                const double vkp = V[k + (size_t)p * me], vkq = V[k + (size_t)q * me];
                V[k + (size_t)p * me] = c * vkp - s * vkq;
                V[k + (size_t)q * me] = s * vkp + c * vkq;
            }
            __syncthreads();
        }
        int any = flags[0];
        __syncthreads();
        if (!any) break;
    }
    // sort: ascending theta (stable), then by |theta| descending (stable)
    if (threadIdx.x == 0) {
        for (int i = 0; i < m; i++) pos[i] = i;
        for (int i = 1; i < m; i++) {
            int key = pos[i];
            double kv = A[key + (size_t)key * me];
            int j = i - 1;
            while (j >= 0 && A[pos[j] + (size_t)pos[j] * me] > kv) { pos[j + 1] = pos[j]; j--; }
            pos[j + 1] = key;
        }
        for (int i = 0; i < m; i++) ord[i] = i;
        for (int i = 1; i < m; i++) {
            int key = ord[i];
            double kv = fabs(A[pos[key] + (size_t)pos[key] * me]);
            int j = i - 1;
            while (j >= 0 && fabs(A[pos[ord[j]] + (size_t)pos[ord[j]] * me]) < kv) {
                ord[j + 1] = ord[j]; j--;
            }
            ord[j + 1] = key;
        }
        status[0] = (sweep < max_sweeps) ? sweep + 1 : -sweep;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += blockDim.x) theta[i] = A[pos[i] + (size_t)pos[i] * me];
    for (int t = threadIdx.x; t < m * m; t += blockDim.x) {
        int r = t % m, c = t / m;
        Sout[t] = V[r + (size_t)pos[c] * me];
    }
}

__global__ void __launch_bounds__(kJacThreads)
jacobi_kernel(int m, const double *__restrict__ H, int ldh, double *theta, double *Sout,
              int *ord, double *gwork, int *status, int use_smem) {
    jacobi_body(m, H, ldh, theta, Sout, ord, gwork, status, use_smem);
}

// One problem per block: problem b (of order mvec[b] when mvec is given,
// else m) reads H + b * strideH and writes theta, S (ld its order), ord and
// status at b * m, b * m * m, b * m and b * 2; active[b] == 0 skips it.
__global__ void __launch_bounds__(kJacThreads)
jacobi_batched_kernel(int m, const int *mvec, const double *__restrict__ H, int ldh,
                      int64_t strideH, double *theta, double *Sout, int *ord, int *status,
                      const int *active) {
    const int b = blockIdx.x;
    if (active && !active[b]) return;
    const int mb = mvec ? mvec[b] : m;
    jacobi_body(mb, H + (size_t)b * strideH, ldh, theta + (size_t)b * m,
                Sout + (size_t)b * m * m, ord + (size_t)b * m, nullptr, status + 2 * b, 1);
}

static size_t jac_small_bytes(int m) {
    size_t me = (size_t)((m + 1) & ~1);
    return sizeof(double) * (2 * me * me + me) + sizeof(int) * (me + 2);
}

int syev_small_smem_limit() {
    int m = 2;
    while (jac_small_bytes(m + 2) <= 200 * 1024) m += 2;
    return m;
}

void launch_syev_small(int m, const double *H, int ldh, double *theta, double *S, int *ord,
                       double *work, int *status, cudaStream_t st) {
    if (m <= 0) return;
    int use_smem = (m <= syev_small_smem_limit()) ? 1 : 0;
    size_t me = (size_t)((m + 1) & ~1);
    size_t smem = use_smem ? jac_small_bytes(m) : sizeof(double) * me + sizeof(int) * (me + 2);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(jacobi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    jacobi_kernel<<<1, kJacThreads, smem, st>>>(m, H, ldh, theta, S, ord, work, status, use_smem);
    note_launch();
}

void launch_syev_batched(int nprob, int m, const int *mvec, const double *H, int ldh,
                         int64_t strideH, double *theta, double *S, int *ord, int *status,
                         const int *active, cudaStream_t st) {
    if (nprob <= 0 || m <= 0) return;
    const size_t smem = jac_small_bytes(m);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(jacobi_batched_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    jacobi_batched_kernel<<<nprob, kJacThreads, smem, st>>>(m, mvec, H, ldh, strideH, theta, S,
                                                            ord, status, active);
    note_launch();
}

void launch_syev_small_workspace(int m, const double *H, int ldh, double *theta, double *S,
                                 int *ord, double *work, int *status, cudaStream_t st) {
    if (m <= 0) return;
    const size_t me = (size_t)((m + 1) & ~1);
    const size_t smem = sizeof(double) * me + sizeof(int) * (me + 2);
    jacobi_kernel<<<1, kJacThreads, smem, st>>>(m, H, ldh, theta, S, ord, work, status, 0);
    note_launch();
}

__global__ void axpby_kernel(int64_t n, double a, const double *x, double b, double *y) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        y[i] = a * x[i] + b * y[i];
}
void launch_axpby(int64_t n, double a, const double *x, double b, double *y, cudaStream_t st) {
    if (n <= 0) return;
    const int nb = (int)std::max<int64_t>(1, std::min<int64_t>(4096, (n + 255) / 256));
    axpby_kernel<<<nb, 256, 0, st>>>(n, a, x, b, y);
    note_launch();
}

// ------------------------------------------------------------- helpers --
__global__ void set_diag_kernel(int ldh, int nd, const double *d, double *H) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ldh * ldh; t += gridDim.x * blockDim.x) {
        int i = t % ldh, j = t / ldh;
        H[t] = (i == j && i < nd) ? d[i] : 0.0;
    }
}
void launch_set_diag(int ldh, int nd, const double *d, double *H, cudaStream_t st) {
    int nb = std::max(1, std::min(256, (ldh * ldh + 255) / 256));
    set_diag_kernel<<<nb, 256, 0, st>>>(ldh, nd, d, H);
    note_launch();
}

__global__ void flag_if_below_kernel(const double *nrm2, double thr, int *flag) {
    chain_begin();
    if (!(nrm2[0] >= thr)) *flag = 1;
}
void launch_flag_if_below(const double *nrm2, double thr, int *flag, cudaStream_t st) {
    launch_chained(flag_if_below_kernel, 1, 1, 0, st, nrm2, thr, flag);
}

__global__ void set_beta_kernel(double *H, int ldh, int r, int c, const double *nrm2, int zero) {
    chain_begin();
    double b = zero ? 0.0 : sqrt(nrm2[0]);
    H[r + (size_t)c * ldh] = b;
    H[c + (size_t)r * ldh] = b;
}
void launch_set_beta(double *H, int ldh, int r, int c, const double *nrm2, int zero,
                     cudaStream_t st) {
    launch_chained(set_beta_kernel, 1, 1, 0, st, H, ldh, r, c, nrm2, zero);
}

__global__ void copy_kernel(int64_t n, const double *src, double *dst) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[i];
}
void launch_copy(int64_t n, const double *src, double *dst, cudaStream_t st) {
    if (n <= 0) return;
    int nb = (int)std::max<int64_t>(1, std::min<int64_t>(4096, (n + 255) / 256));
    copy_kernel<<<nb, 256, 0, st>>>(n, src, dst);
    note_launch();
}
__global__ void fill_kernel(int64_t n, double v, double *dst) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = v;
}
void launch_fill(int64_t n, double v, double *dst, cudaStream_t st) {
    if (n <= 0) return;
    int nb = (int)std::max<int64_t>(1, std::min<int64_t>(4096, (n + 255) / 256));
    fill_kernel<<<nb, 256, 0, st>>>(n, v, dst);
    note_launch();
}

}  // namespace spx

namespace spx {
Counters &counters() {
    static Counters c;
    return c;
}
// ------------------------------------------------------- new values ------
// Bound by the copy of the caller's values to the device; the host rebuilt the
// whole CSR for this before (7.8 ms at 48^3, 760,000 entries; 0.9 ms now).
__global__ void csc_map_kernel(int n, const int64_t *__restrict__ Ap, const int64_t *__restrict__ Ai,
                               const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                               int32_t *__restrict__ map, int *bad) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    // the place of column `col` in row `row`, or -1
    auto find = [&](int row, int col) {
        int lo = rp[row], hi = rp[row + 1];
        const int end = hi;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (ci[mid] < col) lo = mid + 1; else hi = mid;
        }
        return lo < end && ci[lo] == col ? lo : -1;
    };
    int64_t last = -1;
    bool ok = true;
    for (int64_t q = Ap[c]; q < Ap[c + 1]; q++) {
        const int64_t r = Ai[q];
        if (r <= last || r >= n) { ok = false; break; }
        last = r;
        if (r > c) continue;
        const int d = find((int)r, c), e = r < c ? find(c, (int)r) : d;
        if (d < 0 || e < 0) { ok = false; break; }
        map[d] = (int32_t)q;
        map[e] = (int32_t)q;
    }
    if (!ok) *bad = 1;
}
void launch_csc_map(int n, const int64_t *Ap, const int64_t *Ai, const int32_t *rp,
                    const int32_t *ci, int32_t *map, int *bad, cudaStream_t st) {
    csc_map_kernel<<<(n + 127) / 128, 128, 0, st>>>(n, Ap, Ai, rp, ci, map, bad);
    note_launch();
}

__global__ void csc_values_kernel(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ map,
                                  const double *__restrict__ ax, double *__restrict__ va,
                                  unsigned long long *norm_bits) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    double s = 0.0;
    if (r < n)
        for (int q = rp[r]; q < rp[r + 1]; q++) {
            const double v = ax[map[q]];
            va[q] = v;
            s += fabs(v);
        }
    // the maximum over rows, NaN rows left out; sums are not negative, so
    // their bits are ordered as they are
    unsigned long long b = s > 0.0 ? (unsigned long long)__double_as_longlong(s) : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, b, o);
        b = t > b ? t : b;
    }
    if ((threadIdx.x & 31) == 0 && b) atomicMax(norm_bits, b);
}
void launch_csc_values(int n, const int32_t *rp, const int32_t *map, const double *ax, double *va,
                       unsigned long long *norm_bits, cudaStream_t st) {
    csc_values_kernel<<<(n + 127) / 128, 128, 0, st>>>(n, rp, map, ax, va, norm_bits);
    note_launch();
}

}  // namespace spx
