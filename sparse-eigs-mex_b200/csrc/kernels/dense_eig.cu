// See dense_eig.cuh.
#include "dense_eig.cuh"
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

// shared memory of a block: two copies each of v and p, then (when they fit)
// the block's columns of the matrix
size_t tri_head(int n) { return sizeof(double) * (4 * (size_t)n + 2 + kTriWarps); }
size_t tri_smem(int n, int c) { return tri_head(n) + sizeof(double) * (size_t)n * ((n + c - 1) / c); }
constexpr size_t kTriMaxSmem = 220 * 1024;
// blocks of the cluster: 8 (portable) while the matrix fits their shared
// memory, else 16
int tri_cluster(int n) { return tri_smem(n, 8) <= kTriMaxSmem ? 8 : 16; }

}  // namespace

bool dense_tridiag_work(int n) { return tri_smem(n, 16) > kTriMaxSmem; }

// One cluster, columns dealt out cyclically.  Step k: the owner of column k
// makes the reflector and writes it into every block's shared memory; every
// block forms p = beta A v on its columns and writes those entries everywhere;
// every block applies A -= v w^T + w v^T to its columns.  Two cluster barriers
// a step are what bounds it (about 2 us a step at n = 210; the products are
// 0.1 us), so the matrix stays in shared memory and 8 blocks are preferred to
// 16 while it fits.  The Jacobi solver took 95 ms at n = 210, all of it on one
// SM and, from n = 110, out of global memory.
__global__ void __launch_bounds__(kTriThreads)
dense_tridiag_kernel(int n, const double *__restrict__ D, double *__restrict__ V,
                     double *__restrict__ beta, double *__restrict__ d, double *__restrict__ e,
                     double *work) {
    extern __shared__ double tsm[];
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), me = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double *vb = tsm, *pb = tsm + 2 * n, *bb = tsm + 4 * n, *red = bb + 2, *cols = red + kTriWarps;
    auto col = [&](int j) { return work ? work + (size_t)j * n : cols + (size_t)(j / C) * n; };
    for (int j = me + wid * C; j < n; j += kTriWarps * C)
        for (int i = lane; i < n; i += 32) col(j)[i] = D[(size_t)j * n + i];
    __syncthreads();
    cl.sync();
    for (int k = 0; k + 2 < n; k++) {
        double *v = vb + (k & 1) * n, *p = pb + (k & 1) * n, *b = bb + (k & 1);
        if (k % C == me) {
            const double *x = col(k);
            double sq = 0.0;
            for (int i = k + 1 + tid; i < n; i += kTriThreads) sq += x[i] * x[i];
            sq = warp_sum(sq);
            if (lane == 0) red[wid] = sq;
            __syncthreads();
            sq = 0.0;
#pragma unroll
            for (int q = 0; q < kTriWarps; q++) sq += red[q];
            const double x0 = x[k + 1], xn = sqrt(sq), alpha = x0 >= 0.0 ? -xn : xn;
            // 2 / v^T v = 1 / (|x|^2 + |x0| |x|), a sum of positive terms
            const double bt = sq > 0.0 ? 1.0 / (sq + fabs(x0) * xn) : 0.0;
            for (int i = k + 1 + tid; i < n; i += kTriThreads) {
                const double vi = i == k + 1 ? x0 - alpha : x[i];
                for (int q = 0; q < C; q++) cl.map_shared_rank(v, q)[i] = vi;
                V[(size_t)k * n + i] = vi;
            }
            if (tid < C) *cl.map_shared_rank(b, tid) = bt;
            if (tid == 0) {
                beta[k] = bt;
                d[k] = x[k];
                e[k] = sq > 0.0 ? alpha : 0.0;
            }
        }
        cl.sync();
        const double bt = *b;
        if (bt == 0.0) continue;                  // column already reduced, the same in every block
        // first own column above k
        const int j0 = k + 1 + ((me - (k + 1)) % C + C) % C;
        for (int j = j0 + wid * C; j < n; j += kTriWarps * C) {
            const double *a = col(j);
            double s = 0.0;
            for (int i = k + 1 + lane; i < n; i += 32) s += a[i] * v[i];
            s = bt * warp_sum(s);
            if (lane < C) cl.map_shared_rank(p, lane)[j] = s;
        }
        cl.sync();
        double pv = 0.0;
        for (int i = k + 1 + lane; i < n; i += 32) pv += p[i] * v[i];
        const double K = 0.5 * bt * warp_sum(pv);
        for (int j = j0 + wid * C; j < n; j += kTriWarps * C) {
            double *a = col(j);
            const double vj = v[j], wj = p[j] - K * vj;
            for (int i = k + 1 + lane; i < n; i += 32) a[i] -= v[i] * wj + (p[i] - K * v[i]) * vj;
        }
        __syncthreads();
    }
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
    const int c = tri_cluster(n);
    const size_t smem = glob ? tri_head(n) : tri_smem(n, c);
    cudaError_t err = cudaFuncSetAttribute(dense_tridiag_kernel,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTriMaxSmem);
    if (err == cudaSuccess)
        err = cudaFuncSetAttribute(dense_tridiag_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (err != cudaSuccess) return err;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(kTriThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    err = cudaLaunchKernelEx(&cfg, dense_tridiag_kernel, n, D, V, beta, d, e, glob ? work : (double *)nullptr);
    note_launch();
    return err;
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

// One warp an eigenvalue: every round the lanes count at 32 points inside the
// interval, which shrinks by 33; about 11 rounds of n dependent divisions.
__global__ void __launch_bounds__(32)
tri_bisect_kernel(int n, const double *__restrict__ gd, const double *__restrict__ ge, int k,
                  bool smallest, double *val, int *idx) {
    extern __shared__ double bsm[];
    double *d = bsm, *e2 = bsm + n;
    const int lane = threadIdx.x, w = blockIdx.x;
    double lo = DBL_MAX, hi = -DBL_MAX, emax = 0.0;
    for (int i = lane; i < n; i += 32) {
        const double el = i > 0 ? fabs(ge[i - 1]) : 0.0, er = i + 1 < n ? fabs(ge[i]) : 0.0;
        d[i] = gd[i];
        if (i + 1 < n) e2[i] = er * er;
        lo = fmin(lo, gd[i] - el - er);
        hi = fmax(hi, gd[i] + el + er);
        emax = fmax(emax, er);
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
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
        if (lane == 0) idx[w] = -1;
        return;
    }
    for (int it = 0; it < 20; it++) {
        if (hi - lo <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi))) break;
        const double x = lo + (hi - lo) * ((lane + 1) * (1.0 / 33.0));
        const int c = sturm(n, d, e2, pivmin, x);
        const unsigned above = __ballot_sync(0xffffffffu, c > at);
        const int f = above ? __ffs(above) - 1 : 32;   // first point above the eigenvalue
        const double xh = __shfl_sync(0xffffffffu, x, f & 31), xl = __shfl_sync(0xffffffffu, x, (f - 1) & 31);
        const double nh = f < 32 ? xh : hi, nl = f > 0 ? xl : lo;
        if (nh == hi && nl == lo) break;
        hi = nh;
        lo = nl;
    }
    if (lane == 0) {
        val[w] = 0.5 * (lo + hi);
        idx[w] = at;
    }
}

void launch_tri_bisect(int n, const double *d, const double *e, int k, bool smallest, double *val,
                       int *idx, cudaStream_t st) {
    const size_t smem = sizeof(double) * 2 * (size_t)n;
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(tri_bisect_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    tri_bisect_kernel<<<2 * k, 32, smem, st>>>(n, d, e, k, smallest, val, idx);
    note_launch();
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

void launch_apply_reflectors(int n, const double *V, const double *beta, double *Z, int nc,
                             cudaStream_t st) {
    if (n < 3 || nc <= 0) return;
    if (n <= 256) apply_reflectors_kernel<2><<<nc, 128, 0, st>>>(n, V, beta, Z);
    else if (n <= 1024) apply_reflectors_kernel<8><<<nc, 128, 0, st>>>(n, V, beta, Z);
    else apply_reflectors_kernel<32><<<nc, 128, 0, st>>>(n, V, beta, Z);
    note_launch();
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
// are contiguous), x^T y and x^T x summed over the threads.
__global__ void __launch_bounds__(256)
rayleigh_dd_kernel(int n, const double *__restrict__ D, const double *__restrict__ X, double *lam,
                   double *res2) {
    extern __shared__ double qsm[];
    double *x = qsm, *y = qsm + n;
    __shared__ DD red[2][256];
    __shared__ double rs[32];
    const int tid = threadIdx.x;
    for (int i = tid; i < n; i += 256) x[i] = X[(size_t)blockIdx.x * n + i];
    __syncthreads();
    DD num = {0.0, 0.0}, den = {0.0, 0.0};
    for (int i = tid; i < n; i += 256) {
        DD a = {0.0, 0.0};
        for (int j = 0; j < n; j++) a = dd_fma(D[(size_t)j * n + i], x[j], a);
        y[i] = a.h;
        num = dd_add(num, dd_mul(a, x[i]));
        den = dd_fma(x[i], x[i], den);
    }
    red[0][tid] = num;
    red[1][tid] = den;
    for (int o = 128; o > 0; o >>= 1) {
        __syncthreads();
        if (tid < o) {
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
    for (int i = tid; i < n; i += 256) {
        const double t = y[i] - l * x[i];
        s += t * t;
    }
    s = block_sum(s, rs);
    if (tid == 0) {
        lam[blockIdx.x] = l;
        res2[blockIdx.x] = s / de.h;
    }
}

void launch_rayleigh_dd(int n, const double *D, const double *X, int nc, double *lam, double *res2,
                        cudaStream_t st) {
    const size_t smem = sizeof(double) * 2 * (size_t)n;
    if (smem > 32 * 1024)
        cudaFuncSetAttribute(rayleigh_dd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    rayleigh_dd_kernel<<<nc, 256, smem, st>>>(n, D, X, lam, res2);
    note_launch();
}

}  // namespace spx
