// See dense_eig.cuh.
#include "dense_eig.cuh"
#include "../chain.cuh"
#include "../common.cuh"
#include "../counters.h"

#include <cooperative_groups.h>
#include <algorithm>
#include <cfloat>
#include <cmath>

namespace cg = cooperative_groups;

namespace spx {

namespace {

constexpr int kTriThreads = 512;
constexpr int kTriWarps = kTriThreads / 32;

// shared memory of a block: three copies of v and two of p, then (when they
// fit) the block's columns of the matrix
size_t tri_head(int n) { return sizeof(double) * (5 * (size_t)n + 2 * kTriWarps); }
size_t tri_smem(int n, int c) { return tri_head(n) + sizeof(double) * (size_t)n * ((n + c - 1) / c); }
constexpr size_t kTriMaxSmem = 226 * 1024;
// blocks of the cluster: 8 (portable) for small orders, where 16 gain nothing
// (n = 36: 0.50 and 0.49 ms a call) and callers on several streams share the
// SMs; else 16, or 8 where 16 are not to be had and the matrix fits
constexpr int kTriCluster = 16, kTriSmall = 128;

}  // namespace

bool dense_tridiag_work(int n) { return tri_smem(n, kTriCluster) > kTriMaxSmem; }

// One cluster, columns dealt out cyclically.  Step k starts with the reflector
// (v, beta) of column k in every block: every block forms p = beta A v on its
// columns and writes those entries into every block's shared memory, as the
// owner of column k + 1 does with that column; after the step's one cluster
// barrier every block applies A -= v w^T + w v^T to its columns, and to its
// copy of column k + 1, of which it makes the next reflector itself (the same
// operations on the same numbers everywhere, so the blocks agree to the bit).
// What is written remotely exists twice (p) or three times (v): a block may be
// one step ahead of another, not two.
//
// The barrier and the reductions' latency are what bounds it (3 us a step at
// n = 210, the products are 0.1 us), so the matrix stays in shared memory.  n =
// 210: 868 us with a second barrier a step (the owner made the reflector and
// distributed it) and 8 blocks, 696 with one barrier, 645 with 16 blocks.  The
// Jacobi solver took 95 ms, all of it on one SM and, from n = 110, out of
// global memory.
__global__ void __launch_bounds__(kTriThreads)
dense_tridiag_kernel(int n, const double *__restrict__ D, double *__restrict__ V,
                     double *__restrict__ beta, double *__restrict__ d, double *__restrict__ e,
                     double *work) {
    extern __shared__ double tsm[];
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), me = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double *vb = tsm, *pb = tsm + 3 * n, *red = tsm + 5 * n, *cols = red + 2 * kTriWarps;
    auto col = [&](int j) { return work ? work + (size_t)j * n : cols + (size_t)(j / C) * n; };
    for (int j = me + wid * C; j < n; j += kTriWarps * C)
        for (int i = lane; i < n; i += 32) col(j)[i] = D[(size_t)j * n + i];
    // The reflector of column k, whose entries i >= k are in x and whose squares
    // below the diagonal the threads have summed (sq): x becomes v.
    auto reflect = [&](int k, double *x, double sq) {
        double *r = red + (k & 1) * kTriWarps;
        sq = warp_sum(sq);
        if (lane == 0) r[wid] = sq;
        __syncthreads();
        sq = r[lane & (kTriWarps - 1)];
#pragma unroll
        for (int o = kTriWarps / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        const double x0 = x[k + 1], xn = sqrt(sq), alpha = x0 >= 0.0 ? -xn : xn;
        // 2 / v^T v = 1 / (|x|^2 + |x0| |x|), a sum of positive terms
        const double bt = sq > 0.0 ? 1.0 / (sq + fabs(x0) * xn) : 0.0;
        __syncthreads();                          // x0 is read
        if (tid == 0) x[k + 1] = x0 - alpha;
        if (k % C == me) {
            for (int i = k + 1 + tid; i < n; i += kTriThreads)
                V[(size_t)k * n + i] = i == k + 1 ? x0 - alpha : x[i];
            if (tid == 0) {
                beta[k] = bt;
                d[k] = x[k];
                e[k] = sq > 0.0 ? alpha : 0.0;
            }
        }
        __syncthreads();
        return bt;
    };
    double bt = 0.0;
    if (n > 2) {
        double sq = 0.0;
        for (int i = tid; i < n; i += kTriThreads) {
            const double x = D[i];
            vb[i] = x;
            if (i > 0) sq += x * x;
        }
        bt = reflect(0, vb, sq);
    }
    cl.sync();                                    // every block's shared memory is there
    for (int k = 0, at = 0; k + 2 < n; k++, at = at == 2 ? 0 : at + 1) {
        double *v = vb + at * n, *x = vb + (at == 2 ? 0 : at + 1) * n, *p = pb + (k & 1) * n;
        if ((k + 1) % C == me) {
            const double *a = col(k + 1);
            for (int i = k + 1 + tid; i < n; i += kTriThreads) {
                const double ai = a[i];
                for (int q = 0; q < C; q++) cl.map_shared_rank(x, q)[i] = ai;
            }
        }
        // first own column above k
        const int j0 = k + 1 + ((me - (k + 1)) % C + C) % C;
        if (bt != 0.0)                            // else column k is reduced already
            for (int j = j0 + wid * C; j < n; j += 2 * kTriWarps * C) {
                const int j2 = j + kTriWarps * C;     // two columns at a time, if there are two
                const double *a = col(j);
                double s = 0.0, s2 = 0.0;
                if (j2 < n) {
                    const double *a2 = col(j2);
                    for (int i = k + 1 + lane; i < n; i += 32) {
                        const double vi = v[i];
                        s += a[i] * vi;
                        s2 += a2[i] * vi;
                    }
                    s2 = bt * warp_sum(s2);
                    if (lane < C) cl.map_shared_rank(p, lane)[j2] = s2;
                } else {
                    for (int i = k + 1 + lane; i < n; i += 32) s += a[i] * v[i];
                }
                s = bt * warp_sum(s);
                if (lane < C) cl.map_shared_rank(p, lane)[j] = s;
            }
        cl.sync();
        double sq = 0.0;
        if (bt != 0.0) {
            double pv = 0.0;
            for (int i = k + 1 + lane; i < n; i += 32) pv += p[i] * v[i];
            const double K = 0.5 * bt * warp_sum(pv);
            const double v1 = v[k + 1], w1 = p[k + 1] - K * v1;
            for (int i = k + 1 + tid; i < n; i += kTriThreads) {
                const double xi = x[i] - (v[i] * w1 + (p[i] - K * v[i]) * v1);
                x[i] = xi;
                if (i > k + 1) sq += xi * xi;
            }
            for (int j = j0 + wid * C; j < n; j += kTriWarps * C) {
                double *a = col(j);
                const double vj = v[j], wj = p[j] - K * vj;
                for (int i = k + 1 + lane; i < n; i += 32) a[i] -= v[i] * wj + (p[i] - K * v[i]) * vj;
            }
        } else {
            for (int i = k + 2 + tid; i < n; i += kTriThreads) sq += x[i] * x[i];
        }
        if (k + 3 < n) bt = reflect(k + 1, x, sq);
    }
    __syncthreads();
    if (n >= 2 && (n - 2) % C == me && tid == 0) {
        d[n - 2] = col(n - 2)[n - 2];
        e[n - 2] = col(n - 2)[n - 1];
    }
    if ((n - 1) % C == me && tid == 0) d[n - 1] = col(n - 1)[n - 1];
    cl.sync();
}

cudaError_t launch_dense_tridiag(int n, const double *D, double *V, double *beta, double *d,
                                 double *e, double *work, cudaStream_t st) {
    const bool glob = dense_tridiag_work(n);
    cudaError_t err = cudaFuncSetAttribute(dense_tridiag_kernel,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTriMaxSmem);
    if (err == cudaSuccess)
        err = cudaFuncSetAttribute(dense_tridiag_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (err != cudaSuccess) return err;
    auto launch = [&](int c) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(kTriThreads);
        cfg.dynamicSmemBytes = glob ? tri_head(n) : tri_smem(n, c);
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = c;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        note_launch();
        return cudaLaunchKernelEx(&cfg, dense_tridiag_kernel, n, D, V, beta, d, e,
                                  glob ? work : (double *)nullptr);
    };
    err = launch(n <= kTriSmall ? 8 : kTriCluster);
    if (err != cudaSuccess && n > kTriSmall && (glob || tri_smem(n, 8) <= kTriMaxSmem)) {
        cudaGetLastError();
        err = launch(8);
    }
    return err;
}

// The kernels below hold one or two vectors in dynamic shared memory.  Up to
// 48 KB, static and dynamic part together (20.7 KB of the quotients' is
// static), need no asking; what is asked for is the largest order's size
// whatever n is, since it belongs to the kernel and the process: with the size
// of each call, one thread's call could lower another's before its launch.
template <class... P>
static cudaError_t allow_vectors(void (*kernel)(P...)) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(sizeof(double) * 2 * kDenseEigMax));
}

// ------------------------------------------------------------ bisection --
// eigenvalues of (d, e) below x (Sturm count of the LDL^T pivots)
SPX_DEV int sturm(int n, const double *d, const double *e2, double pivmin, double x) {
    double q = d[0] - x;
    if (fabs(q) < pivmin) q = -pivmin;
    int c = q < 0.0;
    for (int i = 1; i < n; i++) {
        q = d[i] - x - e2[i - 1] / q;
        if (fabs(q) < pivmin) q = -pivmin;
        c += q < 0.0;
    }
    return c;
}

// One block an eigenvalue: every round the threads count at 512 points inside
// the interval, which shrinks by 513; six rounds of n dependent divisions.
// More points a round are free as long as the warps' divisions hide behind one
// another's latency (16 warps do).  n = 210: 220 us with one warp (11 rounds),
// 172 with 16.
constexpr int kBisThreads = 512;
__global__ void __launch_bounds__(kBisThreads)
tri_bisect_kernel(int n, const double *__restrict__ gd, const double *__restrict__ ge, int k,
                  bool smallest, double *val, int *idx) {
    extern __shared__ double bsm[];
    __shared__ double part[3][kBisThreads / 32];
    double *d = bsm, *e2 = bsm + n;
    const int tid = threadIdx.x, w = blockIdx.x;
    double lo = DBL_MAX, hi = -DBL_MAX, emax = 0.0;
    for (int i = tid; i < n; i += kBisThreads) {
        const double el = i > 0 ? fabs(ge[i - 1]) : 0.0, er = i + 1 < n ? fabs(ge[i]) : 0.0;
        d[i] = gd[i];
        if (i + 1 < n) e2[i] = er * er;
        lo = fmin(lo, gd[i] - el - er);
        hi = fmax(hi, gd[i] + el + er);
        emax = fmax(emax, er);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
    }
    if ((tid & 31) == 0) {
        part[0][tid >> 5] = lo;
        part[1][tid >> 5] = hi;
        part[2][tid >> 5] = emax;
    }
    __syncthreads();
    for (int q = 0; q < kBisThreads / 32; q++) {
        lo = fmin(lo, part[0][q]);
        hi = fmax(hi, part[1][q]);
        emax = fmax(emax, part[2][q]);
    }
    const double pivmin = DBL_MIN * fmax(1.0, emax * emax), tn = fmax(fabs(lo), fabs(hi));
    lo -= 2.0 * DBL_EPSILON * tn * n + 2.0 * pivmin;
    hi += 2.0 * DBL_EPSILON * tn * n + 2.0 * pivmin;
    int at;
    if (smallest) at = sturm(n, d, e2, pivmin, 0.0) - k + w;
    else at = w < k ? w : n - 2 * k + w;
    bool there = at >= 0 && at < n;
    if (!smallest && 2 * k > n) {
        at = w;
        there = w < n;
    }
    if (!there) {
        if (tid == 0) idx[w] = -1;
        return;
    }
    for (int it = 0; it < 20; it++) {
        if (hi - lo <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi))) break;
        const double step = hi - lo;
        auto point = [&](int t) { return lo + step * ((t + 1) * (1.0 / (kBisThreads + 1))); };
        // the counts rise with the points: how many do not exceed `at`
        const int f = __syncthreads_count(sturm(n, d, e2, pivmin, point(tid)) <= at);
        const double nh = f < kBisThreads ? point(f) : hi, nl = f > 0 ? point(f - 1) : lo;
        if (nh == hi && nl == lo) break;
        hi = nh;
        lo = nl;
    }
    if (tid == 0) {
        val[w] = 0.5 * (lo + hi);
        idx[w] = at;
    }
}

cudaError_t launch_tri_bisect(int n, const double *d, const double *e, int k, bool smallest,
                              double *val, int *idx, cudaStream_t st) {
    if (cudaError_t err = allow_vectors(tri_bisect_kernel)) return err;
    return launch_plain(tri_bisect_kernel, 2 * k, kBisThreads, sizeof(double) * 2 * (size_t)n, st, n,
                        d, e, k, smallest, val, idx);
}

// ------------------------------------------------------- back-transform --
// One block a column, its entries in registers; reflector k is loaded while
// reflector k + 1 is applied.
template <int EPT>
__global__ void __launch_bounds__(128)
apply_reflectors_kernel(int n, const double *__restrict__ V, const double *__restrict__ beta,
                        double *__restrict__ Z) {
    __shared__ double red[2][4];
    double *z = Z + (size_t)blockIdx.x * n;
    const int tid = threadIdx.x;
    double x[EPT], v[EPT];
    auto load = [&](int k) {
#pragma unroll
        for (int q = 0; q < EPT; q++) {
            const int i = tid + 128 * q;
            v[q] = (k >= 0 && i > k && i < n) ? V[(size_t)k * n + i] : 0.0;
        }
    };
#pragma unroll
    for (int q = 0; q < EPT; q++) x[q] = tid + 128 * q < n ? z[tid + 128 * q] : 0.0;
    load(n - 3);
    for (int k = n - 3; k >= 0; k--) {
        const double b = beta[k];
        double u[EPT], s = 0.0;
#pragma unroll
        for (int q = 0; q < EPT; q++) {
            u[q] = b == 0.0 ? 0.0 : v[q];
            s += u[q] * x[q];
        }
        load(k - 1);
        s = warp_sum(s);
        if ((tid & 31) == 0) red[k & 1][tid >> 5] = s;
        __syncthreads();
        s = b * ((red[k & 1][0] + red[k & 1][1]) + (red[k & 1][2] + red[k & 1][3]));
#pragma unroll
        for (int q = 0; q < EPT; q++) x[q] -= s * u[q];
    }
#pragma unroll
    for (int q = 0; q < EPT; q++)
        if (tid + 128 * q < n) z[tid + 128 * q] = x[q];
}

cudaError_t launch_apply_reflectors(int n, const double *V, const double *beta, double *Z, int nc,
                                    cudaStream_t st) {
    if (n < 3 || nc <= 0) return cudaSuccess;
    const auto kernel = n <= 256 ? apply_reflectors_kernel<2>
                        : n <= 1024 ? apply_reflectors_kernel<8> : apply_reflectors_kernel<32>;
    return launch_plain(kernel, nc, 128, 0, st, n, V, beta, Z);
}

// ----------------------------------------- quotients in twice the precision --
struct DD { double h, l; };
SPX_DEV DD dd_add(DD a, DD b) {
    const double s = a.h + b.h, t = s - a.h;
    const double e = (a.h - (s - t)) + (b.h - t) + a.l + b.l;
    const double h = s + e;
    return {h, e - (h - s)};
}
SPX_DEV DD dd_fma(double a, double b, DD c) {          // a b + c
    const double p = a * b;
    return dd_add({p, fma(a, b, -p)}, c);
}
SPX_DEV DD dd_mul(DD a, double b) {
    const double p = a.h * b;
    const double e = fma(a.h, b, -p) + a.l * b, h = p + e;
    return {h, e - (h - p)};
}

// One block a vector: y = D x by rows (row i is column i, so the loads over i
// are contiguous), x^T y and x^T x summed over the threads.  256 rows at a
// time, each by four threads with a quarter of the columns (the chain of a
// row's sum in twice the precision is what it costs).  n = 210: 21 us with
// one thread a row, 13 with four.
constexpr int kRayParts = 4, kRayThreads = 256 * kRayParts;
__global__ void __launch_bounds__(kRayThreads)
rayleigh_dd_kernel(int n, const double *__restrict__ D, const double *__restrict__ X, double *lam,
                   double *res2) {
    extern __shared__ double qsm[];
    double *x = qsm, *y = qsm + n;
    __shared__ DD red[2][256], sums[kRayParts - 1][256];
    __shared__ double rs[32];
    const int t = threadIdx.x, tid = t & 255, part = t >> 8;
    for (int i = t; i < n; i += kRayThreads) x[i] = X[(size_t)blockIdx.x * n + i];
    __syncthreads();
    DD num = {0.0, 0.0}, den = {0.0, 0.0};
    const int j0 = (int)((int64_t)n * part / kRayParts), j1 = (int)((int64_t)n * (part + 1) / kRayParts);
    for (int i0 = 0; i0 < n; i0 += 256) {
        const int i = i0 + tid;
        DD a = {0.0, 0.0};
        if (i < n) {
            const double *row = D + i;
            int j = j0;
            for (; j + 8 <= j1; j += 8) {
                double v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = row[(size_t)(j + u) * n];
#pragma unroll
                for (int u = 0; u < 8; u++) a = dd_fma(v[u], x[j + u], a);
            }
            for (; j < j1; j++) a = dd_fma(row[(size_t)j * n], x[j], a);
        }
        __syncthreads();                               // the rows before are summed
        if (part > 0) sums[part - 1][tid] = a;
        __syncthreads();
        if (part == 0 && i < n) {
#pragma unroll
            for (int q = 0; q < kRayParts - 1; q++) a = dd_add(a, sums[q][tid]);
            y[i] = a.h;
            num = dd_add(num, dd_mul(a, x[i]));
            den = dd_fma(x[i], x[i], den);
        }
    }
    if (part == 0) {
        red[0][tid] = num;
        red[1][tid] = den;
    }
    for (int o = 128; o > 0; o >>= 1) {
        __syncthreads();
        if (t < o) {
            red[0][tid] = dd_add(red[0][tid], red[0][tid + o]);
            red[1][tid] = dd_add(red[1][tid], red[1][tid + o]);
        }
    }
    __syncthreads();
    // (num / den).h with one correction
    const DD nu = red[0][0], de = red[1][0];
    const double q0 = nu.h / de.h;
    const DD r = dd_add(nu, dd_mul(de, -q0));
    const double l = q0 + (r.h + r.l) / de.h;
    double s = 0.0;
    for (int i = t; i < n; i += kRayThreads) {
        const double v = y[i] - l * x[i];
        s += v * v;
    }
    s = block_sum(s, rs);
    if (t == 0) {
        lam[blockIdx.x] = l;
        res2[blockIdx.x] = s / de.h;
    }
}

cudaError_t launch_rayleigh_dd(int n, const double *D, const double *X, int nc, double *lam,
                               double *res2, cudaStream_t st) {
    if (cudaError_t err = allow_vectors(rayleigh_dd_kernel)) return err;
    return launch_plain(rayleigh_dd_kernel, nc, kRayThreads, sizeof(double) * 2 * (size_t)n, st, n, D,
                        X, lam, res2);
}

}  // namespace spx
