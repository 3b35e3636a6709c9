// Device multifrontal supernodal Cholesky (FP64) and the task-queue
// shift-invert solve.  See multifrontal.cuh for the storage scheme.
//
// The factorization is one persistent kernel over 64 x 64 tile tasks
// (mf_factor.cuh); the solve pair is another over panel tiles (below).  A
// pivot that is not positive records the failing column in a device status
// word (never a trap); the tasks after it do no work.
#include "multifrontal.cuh"
#include "../common.cuh"
#include "../counters.h"
#include "../host/parallel.h"

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

#include <algorithm>
#include <cstring>
#include <new>

#include <type_traits>

#include "../../../include/speigs.h"

// Storage type of the fronts and panels; this file is compiled once for
// double (plain FP64 operator) and once for float (mixed precision).
#ifndef SPX_REAL
#define SPX_REAL double
#endif

namespace spx {

using Real = SPX_REAL;
// G panels: leading dimension and offsets in multiples of 16 bytes, the
// granularity of the bulk copies that stage them in the solve
constexpr int kLdgA = (int)(16 / sizeof(Real));

// memory pool of the device (engine.cu): allocations are cached across calls
cudaMemPool_t device_pool(int dev);

namespace {

// ---------------------------------------------------------------- solve --
// The whole solve pair is one persistent kernel that pulls tasks from an
// atomic queue in a topological order (forward tasks leaves -> root, then
// backward tasks root -> leaves) and waits only for the tasks it depends on:
// a forward task for supernode s waits until all children of s are done, a
// backward task until its parent is done.  There is no grid-wide barrier, so
// independent subtrees overlap.  Every task first loads what does not depend
// on other tasks (its panel tile, index lists, b) and only then waits.
// Waits are bounded: a wait that runs out records an error word and returns.
// Deadlock cannot occur: a task waits only on tasks earlier in the queue,
// which are held by running blocks.
//
// Tasks: up to 8 small supernodes (c <= 32, r <= 128) as a bundle, one per
// warp; a larger supernode as 64 x 64 tiles of its panel G, one block task
// per tile that can hold a nonzero.  A tile writes its partial products to
// scratch; the last tile of a row chunk (forward) or column chunk
// (backward), found with an atomic counter, adds the partials in a fixed
// order, so results are the same on every run.
//
// Forward, supernode s:  f = b(pivots) + children's update vectors (host-built
// gather list per front row, children in a fixed order);
// [x1; r2] = G f(0:c);  yf(pivots) = x1;  u_s = f(c:r) - r2.
// Backward:  x1 = G^T [yf(pivots); -x(rows below)].
constexpr int kSThreads = 256;
constexpr int kSWarps = kSThreads / 32;
constexpr int kST = 64;          // rows per forward task, columns per backward task
constexpr int kStrip = 128;      // columns per forward task, rows per backward task
constexpr int kWarpMaxC = 16;    // warp tasks: c <= 16 ...
constexpr int kWarpMaxR = 128;   // ... and r <= 128
constexpr int kGW = 6;           // gather entries per row staged in shared memory
constexpr int kTinyR = 24;       // thread tasks: leaves with r <= 24 ...
constexpr int kTinyC = 6;        // ... and c <= 6
constexpr long kSpinLimit = 1L << 22;

enum { ST_FWD_BUNDLE = 0, ST_FWD_TILE = 1, ST_BWD_BUNDLE = 2, ST_BWD_TILE = 3, ST_FWD_THREADS = 4,
       ST_BWD_THREADS = 5 };

struct SNode {          // per-supernode solve metadata (64 bytes)
    int4 a;             // first, c, r, ldg
    int4 b;             // parent, completions expected from the children
                        // (forward), row chunks, column chunks
    longlong2 p;        // panel offset, row-list offset
    long long uptr;
    int bwd_expect;     // completions of the parent's backward (of its own
                        // forward, for a root) that the backward waits for
    int nchild;
};

struct STask {
    int4 a;             // kind, s, I, J
    int4 b;             // chunk, bundle offset, bundle size, 0
};

struct SolveArgs {
    const SNode *meta;
    const STask *tasks;
    int ntasks, ns;
    const int32_t *bundle, *perm, *rows, *cptr, *cidx;
    const Real *G;
    double *u, *yf, *x;
    const int32_t *fc_base, *fc_n, *bc_base, *bc_n;
    double *fpart, *bpart;
    int *fcnt, *bcnt;
    int *sync;          // block queue | forward arrivals per parent [ns] | forward warp
                        // queue, then unused [ns] | backward arrivals [ns] | root forward
                        // arrivals [ns] | backward warp queue, then unused [ns] | err
    const STask *wtasks;    // warp tasks: nfw forward, then nbw backward
    int nfw, nbw;
    const double *b;
    double *out;
    const int *skip;    // when set and nonzero: nothing to do
};

// relaxed-free publish: a release atomic orders every write that precedes it
// in causality order -- the caller's own, and those of threads that reached a
// block or warp barrier before it -- ahead of the increment
SPX_DEV void add_release(int *p, int v) {
    asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

SPX_DEV int ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Bounded wait for *p >= target; gives up (and flags *err) after about a
// second, or at once when another wait has already given up.
SPX_DEV void wait_at_least(const int *p, int target, int *err) {
    if (ld_acquire(p) >= target) return;
    for (long it = 0; it < kSpinLimit; it++) {
        __nanosleep(100);
        if (ld_acquire(p) >= target) return;
        if ((it & 255) == 0 && *(volatile int *)err) return;
    }
    atomicExch(err, 1);
}

// Stage the gather list of front row g: count in *n, first kGW indices in
// idx[0..), the list start in *e0 (for entries past kGW).
SPX_DEV void stage_list(const SolveArgs &a, int64_t g, int *idx, int *n, int *e0) {
    const int b0 = a.cptr[g], b1 = a.cptr[g + 1];
    *n = b1 - b0;
    *e0 = b0;
    const int m = min(b1 - b0, kGW);
    for (int e = 0; e < m; e++) idx[e] = a.cidx[b0 + e];
}
SPX_DEV double sum_list(const SolveArgs &a, const int *idx, int n, int e0) {
    double acc = 0.0;
    const int m = min(n, kGW);
    for (int e = 0; e < m; e++) acc += __ldcg(a.u + idx[e]);
    for (int e = kGW; e < n; e++) acc += __ldcg(a.u + a.cidx[e0 + e]);
    return acc;
}

// true in every thread of the block that holds the chunk's last arrival
SPX_DEV bool last_arrival(int *cnt, int n, int *flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        int old;
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(cnt) : "memory");
        *flag = (old == n - 1);
        if (*flag) *cnt = 0;          // every arrival for this solve is in
    }
    __syncthreads();
    return *flag;
}

// shared memory of one solve block.  gbuf holds one panel strip, staged by
// bulk asynchronous copies (one per panel column) that complete on `bar`.
struct SolveShared {
    Real gbuf[kStrip * kST];          // forward: 128 cols x 64 rows; backward: 64 x 128
    double part[4][kST];
    double vec[kStrip];               // f segment (forward) or v segment (backward)
    double colsum[kST];
    int idx[kStrip][kGW];             // gather lists of the strip's pivot columns
    int cnt[kStrip], e0[kStrip];
    int idx2[kST][kGW];               // gather lists of the chunk's rows below the pivots
    int cnt2[kST], e02[kST];
    int rowv[kStrip];
    int permv[kST];
    double bsum[kST];
};
struct WarpShared {           // per warp in a bundle: gather lists of <= 128 rows
    int idx[kWarpMaxR][kGW];
    int cnt[kWarpMaxR], e0[kWarpMaxR];
};

// Sum p[j] over the 32 lanes for every j < 16 at once: four exchange steps
// (8 + 4 + 2 + 1 shuffles) leave lanes L and L ^ 16 each holding the half
// sum for j = L & 15; one more exchange completes it.
SPX_DEV double transpose_reduce16(double (&p)[16], int lane) {
#pragma unroll
    for (int m = 0; m < 8; m++) {
        const bool hi = lane & 8;
        const double send = hi ? p[m] : p[m + 8];
        const double keep = hi ? p[m + 8] : p[m];
        p[m] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const bool hi = lane & 4;
        const double send = hi ? p[m] : p[m + 4];
        const double keep = hi ? p[m + 4] : p[m];
        p[m] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
#pragma unroll
    for (int m = 0; m < 2; m++) {
        const bool hi = lane & 2;
        const double send = hi ? p[m] : p[m + 2];
        const double keep = hi ? p[m + 2] : p[m];
        p[m] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    {
        const bool hi = lane & 1;
        const double send = hi ? p[0] : p[1];
        const double keep = hi ? p[1] : p[0];
        p[0] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
    }
    return p[0] + __shfl_xor_sync(0xffffffffu, p[0], 16);
}

// ---- bulk asynchronous copies into shared memory, tracked by an mbarrier
SPX_DEV uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
SPX_DEV void mbar_init(unsigned long long *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
SPX_DEV void mbar_expect(unsigned long long *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes) : "memory");
}
// copy `bytes` (a multiple of 16, both addresses 16-byte aligned) global -> shared
SPX_DEV void bulk_load(void *dst, const void *src, uint32_t bytes, unsigned long long *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}
SPX_DEV bool mbar_test(unsigned long long *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// bounded wait for the copies of the current phase; a wait that runs out
// flags *err and then waits again (bounded) for the copies still in flight
SPX_DEV void mbar_wait(unsigned long long *bar, uint32_t parity, int *err) {
    for (long it = 0; it < kSpinLimit; it++)
        if (mbar_test(bar, parity)) return;
    atomicExch(err, 1);
    for (long it = 0; it < kSpinLimit; it++)
        if (mbar_test(bar, parity)) return;
}
SPX_DEV void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Stage columns [j0, j0+ncols) x rows [i0, i0+nrows) of a panel (leading
// dimension ldg, column-major) into buf (column stride `stride` doubles):
// one bulk copy per column, issued by the lanes of warp 0.  nrows is even.
SPX_DEV void stage_panel(Real *buf, int stride, const Real *panel, int ldg, int i0, int nrows,
                         int j0, int ncols, unsigned long long *bar) {
    if (threadIdx.x >= 32) return;
    if (threadIdx.x == 0) mbar_expect(bar, (uint32_t)(ncols * nrows * sizeof(Real)));
    __syncwarp();
    for (int jj = threadIdx.x; jj < ncols; jj += 32)
        bulk_load(buf + (size_t)jj * stride, panel + (int64_t)i0 + (int64_t)(j0 + jj) * ldg,
                  (uint32_t)(nrows * sizeof(Real)), bar);
}

// ---- forward, one tiny leaf supernode (r <= 24, c <= 6) per thread.  A
// leaf has no children, so f is b(pivots); the row and column loops are
// unrolled with predication so all of the thread's loads are in flight at once.
SPX_DEV void fwd_thread(const SolveArgs &a, int s) {
    int *const fcd = a.sync + 1, *const fchk = fcd + 3 * a.ns;
    const SNode m = a.meta[s];
    const int first = m.a.x, c = m.a.y, r = m.a.z, ldg = m.a.w, parent = m.b.x;
    const Real *Gs = a.G + m.p.x;
    double f[kTinyC];
#pragma unroll
    for (int j = 0; j < kTinyC; j++) f[j] = (j < c) ? a.b[a.perm[first + j]] : 0.0;
#pragma unroll
    for (int i = 0; i < kTinyR; i++) {
        if (i < r) {
            double acc = 0.0;
#pragma unroll
            for (int j = 0; j < kTinyC; j++)
                if (j < c) acc += Gs[(int64_t)i + (int64_t)j * ldg] * f[j];
            if (i < c) a.yf[first + i] = acc;
            else a.u[m.uptr + (i - c)] = -acc;
        }
    }
    add_release(parent >= 0 ? fcd + parent : fchk + s, 1);
}

// ---- backward, one tiny leaf supernode per thread
SPX_DEV void bwd_thread(const SolveArgs &a, int s) {
    int *const bdone = a.sync + 1 + 2 * a.ns, *const fchk = bdone + a.ns,
              *const err = a.sync + 1 + 5 * a.ns;
    const SNode m = a.meta[s];
    const int first = m.a.x, c = m.a.y, r = m.a.z, ldg = m.a.w, parent = m.b.x;
    const int32_t *rows = a.rows + m.p.y;
    const Real *Gs = a.G + m.p.x;
    int ri[kTinyR];
#pragma unroll
    for (int i = 0; i < kTinyR; i++) ri[i] = (i >= c && i < r) ? rows[i] : 0;
    wait_at_least(parent >= 0 ? bdone + parent : fchk + s, m.bwd_expect, err);
    double v[kTinyR];
#pragma unroll
    for (int i = 0; i < kTinyR; i++)
        v[i] = (i < r) ? ((i < c) ? __ldcg(a.yf + first + i) : -__ldcg(a.x + ri[i])) : 0.0;
#pragma unroll
    for (int j = 0; j < kTinyC; j++) {
        if (j < c) {
            double acc = 0.0;
#pragma unroll
            for (int i = 0; i < kTinyR; i++)
                if (i < r) acc += Gs[(int64_t)i + (int64_t)j * ldg] * v[i];
            a.x[first + j] = acc;
            a.out[a.perm[first + j]] = acc;
        }
    }
    add_release(bdone + s, 1);
}

// ---- forward, one small supernode per warp.  Row i lives in lane i % 32
// (q = i / 32); the panel values of a lane's rows are read in blocks of 4
// columns before they are used, so loads are not serialised behind the
// column loop.
SPX_DEV void fwd_warp(const SolveArgs &a, int s, WarpShared &w) {
    int *const fcd = a.sync + 1, *const fchk = fcd + 3 * a.ns, *const err = a.sync + 1 + 5 * a.ns;
    const SNode m = a.meta[s];
    const int first = m.a.x, c = m.a.y, r = m.a.z, ldg = m.a.w;
    const int parent = m.b.x, nchild = m.nchild, expect = m.b.y;
    const int64_t g0 = m.p.y;
    const Real *Gs = a.G + m.p.x;
    const int lane = threadIdx.x & 31;
    const int nq = (r + 31) >> 5;
    double bv = 0.0;
    if (lane < c) bv = a.b[a.perm[first + lane]];
    // tiny panels (r <= 32, c <= 8) are read completely before the wait
    double gt[8];
    const bool tiny = (r <= 32 && c <= 8);
    if (tiny) {
#pragma unroll
        for (int j = 0; j < 8; j++)
            gt[j] = (j < c && lane < r) ? Gs[(int64_t)lane + (int64_t)j * ldg] : 0.0;
    }
    if (nchild > 0)
        for (int i = lane; i < r; i += 32) stage_list(a, g0 + i, w.idx[i], &w.cnt[i], &w.e0[i]);
    __syncwarp();
    if (nchild > 0) {
        if (lane == 0) wait_at_least(fcd + s, expect, err);
        __syncwarp();
    }
    double fj = 0.0;
    if (lane < c) fj = bv + (nchild > 0 ? sum_list(a, w.idx[lane], w.cnt[lane], w.e0[lane]) : 0.0);
    double acc[kWarpMaxR / 32];
#pragma unroll
    for (int q = 0; q < kWarpMaxR / 32; q++) acc[q] = 0.0;
    if (tiny) {
#pragma unroll
        for (int j = 0; j < 8; j++) acc[0] += gt[j] * __shfl_sync(0xffffffffu, fj, j);
    } else {
#pragma unroll
        for (int j = 0; j < kWarpMaxC; j++) {
            const double fb = __shfl_sync(0xffffffffu, fj, j);
#pragma unroll
            for (int q = 0; q < kWarpMaxR / 32; q++) {
                const int i = lane + 32 * q;
                if (j < c && q < nq && i < r) acc[q] += Gs[(int64_t)i + (int64_t)j * ldg] * fb;
            }
        }
    }
    // (the panel is zero above the diagonal of its pivot block, so the
    // products above need no masking)
#pragma unroll
    for (int q = 0; q < kWarpMaxR / 32; q++) {
        const int i = lane + 32 * q;
        if (i >= r) continue;
        if (i < c) a.yf[first + i] = acc[q];
        else a.u[m.uptr + (i - c)] =
            (nchild > 0 ? sum_list(a, w.idx[i], w.cnt[i], w.e0[i]) : 0.0) - acc[q];
    }
    __syncwarp();
    if (lane == 0) add_release(parent >= 0 ? fcd + parent : fchk + s, 1);
}

// ---- forward, rows [64 I, 64 I + 64) x a 128-column strip S of a large
// supernode's panel.  The strip is staged into shared memory before the
// dependency wait.
SPX_DEV void fwd_tile(const SolveArgs &a, int s, int I, int S, int chunk, SolveShared &sh,
                      unsigned long long *bar, uint32_t &phase, int *flag) {
    int *const fcd = a.sync + 1, *const fchk = fcd + 3 * a.ns, *const err = a.sync + 1 + 5 * a.ns;
    const SNode m = a.meta[s];
    const int first = m.a.x, c = m.a.y, r = m.a.z, ldg = m.a.w;
    const int parent = m.b.x, nchild = m.nchild, expect = m.b.y;
    const int64_t g0 = m.p.y;
    const int i0 = I * kST, j0 = S * kStrip;
    const int jn = min(kStrip, c - j0);
    // a multiple of 16 bytes: ldg is, and i0 is a multiple of 64
    const int hcopy = min(kST, ldg - i0);
    stage_panel(sh.gbuf, kST, a.G + m.p.x, ldg, i0, hcopy, j0, jn, bar);
    const int t = threadIdx.x;
    double bv = 0.0;
    if (t < jn) {
        bv = a.b[a.perm[first + j0 + t]];
        if (nchild > 0) stage_list(a, g0 + j0 + t, sh.idx[t], &sh.cnt[t], &sh.e0[t]);
    }
    if (t >= kStrip && t < kStrip + kST) {
        const int tt = t - kStrip, ii = i0 + tt;
        if (nchild > 0 && ii >= c && ii < r) stage_list(a, g0 + ii, sh.idx2[tt], &sh.cnt2[tt], &sh.e02[tt]);
    }
    if (nchild > 0 && t == 0) wait_at_least(fcd + s, expect, err);
    __syncthreads();
    if (t < kStrip) {
        sh.vec[t] = (t < jn) ? bv + (nchild > 0 ? sum_list(a, sh.idx[t], sh.cnt[t], sh.e0[t]) : 0.0)
                             : 0.0;
    } else if (t < kStrip + kST) {
        // the children's contributions to the chunk's rows below the pivots,
        // needed by whichever strip finishes the chunk
        const int tt = t - kStrip, ii = i0 + tt;
        sh.bsum[tt] = (nchild > 0 && ii >= c && ii < r)
                          ? sum_list(a, sh.idx2[tt], sh.cnt2[tt], sh.e02[tt]) : 0.0;
    }
    mbar_wait(bar, phase, err);
    phase ^= 1u;
    __syncthreads();
    const int row = t & (kST - 1), grp = t >> 6;
    double acc = 0.0;
    if (row < hcopy)
        for (int jj = grp; jj < jn; jj += 4) acc += sh.gbuf[jj * kST + row] * sh.vec[jj];
    sh.part[grp][row] = acc;
    __syncthreads();
    const int nt = a.fc_n[chunk];
    double own = 0.0;
    if (t < kST) {
        own = (sh.part[0][t] + sh.part[1][t]) + (sh.part[2][t] + sh.part[3][t]);
        if (nt > 1) a.fpart[(int64_t)(a.fc_base[chunk] + S) * kST + t] = own;
    }
    // a row chunk held by one strip needs no cross-block sum
    if (nt == 1 || last_arrival(a.fcnt + chunk, nt, flag)) {
        const int ii = i0 + t;
        if (t < kST && ii < r) {
            double rr = own;
            if (nt > 1) {
                const double *p0 = a.fpart + (int64_t)a.fc_base[chunk] * kST + t;
                rr = 0.0;
                for (int q = 0; q < nt; q++) rr += __ldcg(p0 + (int64_t)q * kST);
            }
            if (ii < c) a.yf[first + ii] = rr;
            else a.u[m.uptr + (ii - c)] = sh.bsum[t] - rr;
        }
        __syncthreads();
        // one completed row chunk: the parent counts every chunk of every child
        if (t == 0) add_release(parent >= 0 ? fcd + parent : fchk + s, 1);
    }
    __syncthreads();
}

// ---- backward, one small supernode per warp: column sums x1_j = sum_i
// G(i, j) v_i, with the panel values of blocks of 4 columns loaded before
// their reductions.
SPX_DEV void bwd_warp(const SolveArgs &a, int s) {
    int *const bdone = a.sync + 1 + 2 * a.ns, *const fchk = bdone + a.ns,
              *const err = a.sync + 1 + 5 * a.ns;
    const SNode m = a.meta[s];
    const int first = m.a.x, c = m.a.y, r = m.a.z, ldg = m.a.w, parent = m.b.x;
    const int32_t *rows = a.rows + m.p.y;
    const Real *Gs = a.G + m.p.x;
    const int lane = threadIdx.x & 31;
    const int nq = (r + 31) >> 5;
    int rv[kWarpMaxR / 32];
#pragma unroll
    for (int q = 0; q < kWarpMaxR / 32; q++) {
        const int i = lane + 32 * q;
        rv[q] = (i >= c && i < r) ? rows[i] : 0;
    }
    const int pj = (lane < c) ? a.perm[first + lane] : 0;
    double gt[8];
    const bool tiny = (r <= 32 && c <= 8);
    if (tiny) {
#pragma unroll
        for (int j = 0; j < 8; j++)
            gt[j] = (j < c && lane < r) ? Gs[(int64_t)lane + (int64_t)j * ldg] : 0.0;
    }
    if (lane == 0) wait_at_least(parent >= 0 ? bdone + parent : fchk + s, m.bwd_expect, err);
    __syncwarp();
    double v[kWarpMaxR / 32];
#pragma unroll
    for (int q = 0; q < kWarpMaxR / 32; q++) {
        const int i = lane + 32 * q;
        v[q] = (i < r) ? ((i < c) ? __ldcg(a.yf + first + i) : -__ldcg(a.x + rv[q])) : 0.0;
    }
    // every lane accumulates its rows' products for all 16 columns, then one
    // transposing reduction leaves column j's sum in lanes j and j + 16
    double p[kWarpMaxC];
#pragma unroll
    for (int j = 0; j < kWarpMaxC; j++) p[j] = 0.0;
    if (tiny) {
#pragma unroll
        for (int j = 0; j < 8; j++) p[j] = gt[j] * v[0];
    } else {
#pragma unroll
        for (int q = 0; q < kWarpMaxR / 32; q++) {
            const int i = lane + 32 * q;
            if (q < nq && i < r) {
#pragma unroll
                for (int j = 0; j < kWarpMaxC; j++)
                    if (j < c) p[j] += Gs[(int64_t)i + (int64_t)j * ldg] * v[q];
            }
        }
    }
    const double mine = transpose_reduce16(p, lane);
    if (lane < c) {
        a.x[first + lane] = mine;
        a.out[pj] = mine;
    }
    __syncwarp();
    if (lane == 0) add_release(bdone + s, 1);
}

// ---- backward, columns [64 J, 64 J + 64) x a 128-row strip S of a large
// supernode's panel, staged into shared memory before the dependency wait.
SPX_DEV void bwd_tile(const SolveArgs &a, int s, int J, int S, int chunk, SolveShared &sh,
                      unsigned long long *bar, uint32_t &phase, int *flag) {
    int *const bdone = a.sync + 1 + 2 * a.ns, *const fchk = bdone + a.ns,
              *const err = a.sync + 1 + 5 * a.ns;
    const SNode m = a.meta[s];
    const int first = m.a.x, c = m.a.y, r = m.a.z, ldg = m.a.w, parent = m.b.x;
    const int32_t *rows = a.rows + m.p.y;
    const int i0 = S * kStrip, j0 = J * kST;
    const int in = min(kStrip, r - i0), jn = min(kST, c - j0);
    const int hcopy = min(kStrip, ldg - i0);
    stage_panel(sh.gbuf, kStrip, a.G + m.p.x, ldg, i0, hcopy, j0, jn, bar);
    const int t = threadIdx.x;
    if (t < kStrip) {
        const int ii = i0 + t;
        sh.rowv[t] = (t < in && ii >= c) ? rows[ii] : 0;
    } else if (t < kStrip + kST) {
        const int tt = t - kStrip;
        sh.permv[tt] = (tt < jn) ? a.perm[first + j0 + tt] : 0;
    }
    if (t == 0) wait_at_least(parent >= 0 ? bdone + parent : fchk + s, m.bwd_expect, err);
    __syncthreads();
    if (t < kStrip) {
        const int ii = i0 + t;
        sh.vec[t] = (t < in) ? ((ii < c) ? __ldcg(a.yf + first + ii) : -__ldcg(a.x + sh.rowv[t]))
                             : 0.0;
    }
    mbar_wait(bar, phase, err);
    phase ^= 1u;
    __syncthreads();
    const int lane = t & 31, wid = t >> 5;
    const int nt = a.bc_n[chunk];
    {
        // warp wid owns columns wid + 8k, k < 8; lanes own rows lane + 32q
        double p[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int jj = wid + kSWarps * k;
            double acc = 0.0;
#pragma unroll
            for (int q = 0; q < kStrip / 32; q++) {
                const int ii = lane + 32 * q;
                if (jj < jn && ii < hcopy) acc += sh.gbuf[jj * kStrip + ii] * sh.vec[ii];
            }
            p[k] = acc;
        }
        // halve the 8 partial columns across lane bits 2, 1, 0, then finish
        // the sums over lane bits 3 and 4: lane L ends with column k = L & 7
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const bool hi = lane & 4;
            const double send = hi ? p[m] : p[m + 4];
            const double keep = hi ? p[m + 4] : p[m];
            p[m] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
        }
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const bool hi = lane & 2;
            const double send = hi ? p[m] : p[m + 2];
            const double keep = hi ? p[m + 2] : p[m];
            p[m] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
        }
        {
            const bool hi = lane & 1;
            const double send = hi ? p[0] : p[1];
            const double keep = hi ? p[1] : p[0];
            p[0] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
        }
        double col = p[0] + __shfl_xor_sync(0xffffffffu, p[0], 8);
        col += __shfl_xor_sync(0xffffffffu, col, 16);
        if (lane < 8) {
            const int jj = wid + kSWarps * lane;
            if (jj < jn) {
                if (nt > 1) a.bpart[(int64_t)(a.bc_base[chunk] + (S - (j0 / kStrip))) * kST + jj] = col;
                else sh.colsum[jj] = col;
            }
        }
    }
    if (nt == 1) __syncthreads();
    // a column chunk held by one strip needs no cross-block sum
    if (nt == 1 || last_arrival(a.bcnt + chunk, nt, flag)) {
        const int jj = t;
        if (jj < jn) {
            double rr = sh.colsum[jj];
            if (nt > 1) {
                const double *p0 = a.bpart + (int64_t)a.bc_base[chunk] * kST + jj;
                rr = 0.0;
                for (int q = 0; q < nt; q++) rr += __ldcg(p0 + (int64_t)q * kST);
            }
            a.x[first + j0 + jj] = rr;
            a.out[sh.permv[jj]] = rr;
        }
        __syncthreads();
        // one completed column chunk: the children count every chunk
        if (t == 0) add_release(bdone + s, 1);
    }
    __syncthreads();
}

// Warp tasks of one phase: each warp takes the next task from the phase's
// own counter.  A task is one small supernode (ST_*_BUNDLE with one entry)
// or up to 32 tiny leaves, one per lane (ST_*_THREADS).
SPX_DEV void solve_warp_tasks(const SolveArgs &a, const STask *tq, int nt, int *ctr,
                              WarpShared &w) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(ctr, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= nt) break;
        const STask tk = tq[t];
        switch (tk.a.x) {
            case ST_FWD_BUNDLE: fwd_warp(a, a.bundle[tk.b.y], w); break;
            case ST_BWD_BUNDLE: bwd_warp(a, a.bundle[tk.b.y]); break;
            case ST_FWD_THREADS:
                if (lane < tk.b.z) fwd_thread(a, a.bundle[tk.b.y + lane]);
                break;
            default:
                if (lane < tk.b.z) bwd_thread(a, a.bundle[tk.b.y + lane]);
                break;
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kSThreads, 2) mf_solve_sf(SolveArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int s_task, s_flag;
    __shared__ __align__(8) unsigned long long s_bar;
    SolveShared &sh = *reinterpret_cast<SolveShared *>(smem_raw);
    WarpShared *ws = reinterpret_cast<WarpShared *>(smem_raw);
    if (a.skip && *(volatile const int *)a.skip) return;
    const int wid = threadIdx.x >> 5;
    uint32_t phase = 0;
    if (threadIdx.x == 0) mbar_init(&s_bar);
    // forward warp tasks (the small subtrees), every warp on its own
    solve_warp_tasks(a, a.wtasks, a.nfw, a.sync + 1 + a.ns, ws[wid]);
    __syncthreads();
    fence_proxy_async();
    for (;;) {
        if (threadIdx.x == 0) s_task = atomicAdd(a.sync, 1);
        __syncthreads();
        const int t = s_task;
        __syncthreads();
        if (t >= a.ntasks) break;
        const STask tk = a.tasks[t];
        switch (tk.a.x) {
            case ST_FWD_BUNDLE:
                if (wid < tk.b.z) fwd_warp(a, a.bundle[tk.b.y + wid], ws[wid]);
                break;
            case ST_FWD_TILE:
                fwd_tile(a, tk.a.y, tk.a.z, tk.a.w, tk.b.x, sh, &s_bar, phase, &s_flag);
                break;
            case ST_BWD_BUNDLE:
                if (wid < tk.b.z) bwd_warp(a, a.bundle[tk.b.y + wid]);
                break;
            case ST_FWD_THREADS:
                if ((int)threadIdx.x < tk.b.z) fwd_thread(a, a.bundle[tk.b.y + threadIdx.x]);
                break;
            case ST_BWD_THREADS:
                if ((int)threadIdx.x < tk.b.z) bwd_thread(a, a.bundle[tk.b.y + threadIdx.x]);
                break;
            default:
                bwd_tile(a, tk.a.y, tk.a.z, tk.a.w, tk.b.x, sh, &s_bar, phase, &s_flag);
                break;
        }
        __syncthreads();
        // shared memory read by this task may be refilled by the async
        // proxy in the next one
        fence_proxy_async();
    }
    // backward warp tasks
    solve_warp_tasks(a, a.wtasks + a.nfw, a.nbw, a.sync + 1 + 4 * a.ns, ws[wid]);
}

#include "mf_factor.cuh"
#include "mf_block_solve.cuh"

static size_t solve_smem_bytes() {
    return std::max(sizeof(SolveShared), sizeof(WarpShared) * kSWarps);
}

// host mirrors of SNode / STask
struct SNodeH {
    int first, c, r, ldg, parent, fwd_expect, nrc, ncc;
    long long gptr, g0, uptr;
    int bwd_expect, nchild;
};
struct STaskH {
    int kind, s, I, J, chunk, boff, bn, pad;
};

struct FNodeH {
    int first, c, r, ldg, parent, nchild, child0, expect;
    long long fptr, uptr, gptr, g0;
    int flag0, nkb, nt, unused, pad[4];
};
struct FChildH {
    long long uptr, relmap;
    int cbnd, nb, pad[2];
};
struct FTaskH { int kind, s, I, J; };
static_assert(sizeof(FNodeH) == sizeof(FNode), "factor node layout");
static_assert(sizeof(FChildH) == sizeof(FChild), "factor child layout");
static_assert(sizeof(FTaskH) == sizeof(FTask), "factor task layout");

// The factor's nodes, tile storage (in Reals) and task queue.
//
// A task's key is an estimate (us) of the path from it to the end of the
// root: a column block of a front's diagonal chain costs kStep, and a front
// kFront for its assembly and hand-over.  Tasks run in decreasing key order,
// equal keys in the order they were made, which puts every task after the
// ones it waits for: a front starts below its children's update tiles, a
// column block below the one before it, rows below their diagonal tile.
// Inverse tiles follow two column blocks behind the chain; W tiles, which no
// factor task waits for, fill the middle of the parent's chain.
static void plan_factor_tasks(const spx_symbolic &S, const int64_t *gptr,
                              std::vector<FNodeH> &node, std::vector<FChildH> &child,
                              std::vector<int32_t> &cbnd, std::vector<FTaskH> &tasks,
                              int64_t *storage, int64_t *nflags) {
    constexpr int kStep = 15, kFront = 12, kRes = 4;
    const int32_t ns = S.nsuper;
    int64_t off = 0, nfl = 0;
    std::vector<int32_t> start(ns, 0);           // key of a front's first task
    auto r4 = [](int64_t v) { return (v + 3) & ~(int64_t)3; };
    auto is_small = [&](int32_t s) { return node[s].nkb == 1 && node[s].nt <= 2; };
    for (int32_t s = 0; s < ns; s++) {
        FNodeH &m = node[s];
        m = FNodeH();
        m.first = S.sfirst[s];
        m.c = S.sfirst[s + 1] - S.sfirst[s];
        m.r = (int)(S.rowptr[s + 1] - S.rowptr[s]);
        m.ldg = (m.r + kLdgA - 1) & ~(kLdgA - 1);
        m.parent = S.sparent[s];
        m.nchild = S.child_ptr[s + 1] - S.child_ptr[s];
        m.child0 = S.child_ptr[s];
        m.gptr = gptr[s];
        m.g0 = S.rowptr[s];
        m.nkb = (m.c + FT - 1) / FT;
        const int64_t nb = m.r - m.c, nu = (nb + FT - 1) / FT, nkb = m.nkb;
        m.nt = (int)(nkb + nu);
        const int64_t wc4 = r4(m.c - (nkb - 1) * FT);
        m.fptr = off;
        if (!is_small(s)) {
            // lower pivot tiles, then the transposed inverse's tiles
            off += (int64_t)FT * FT * ((nkb - 1) * m.nt - (nkb - 1) * (nkb - 2) / 2) + FT * wc4 * (nu + 1);
            off += (int64_t)FT * FT * (nkb * (nkb - 1) / 2) + FT * wc4 * nkb;
            m.flag0 = (int)nfl;
            nfl += nkb * m.nt + nkb * nkb;
        }
        m.uptr = off;
        if (nu > 0) {
            const int64_t wl4 = r4(nb - (nu - 1) * FT);
            off += (int64_t)FT * FT * ((nu - 1) * nu - (nu - 1) * (nu - 2) / 2) + FT * wl4;
        }
    }
    for (int32_t s = ns - 1; s >= 0; s--) {
        const FNodeH &m = node[s];
        start[s] = kRes * (kFront + kStep * m.nkb) + (m.parent < 0 ? 0 : start[m.parent]);
    }
    int64_t ntask = 0, nbnd = 0;
    for (int32_t s = 0; s < ns; s++) {
        const FNodeH &m = node[s];
        const int64_t nu = m.nt - m.nkb, nkb = m.nkb;
        ntask += is_small(s) ? 1 : (int64_t)m.nt * (m.nt + 1) / 2 + nkb * (nkb - 1) / 2 + nu * nkb;
        if (m.parent >= 0) {
            node[m.parent].expect += is_small(s) ? nu : nu * (nu + 1) / 2;
            nbnd += node[m.parent].nt + 1;
        }
    }
    // the children's records and their bounds per 64-row tile of the parent
    cbnd.reserve(nbnd);
    for (int32_t p = 0; p < ns; p++)
        for (int32_t q = S.child_ptr[p]; q < S.child_ptr[p + 1]; q++) {
            const int32_t ch = S.child_list[q];
            FChildH &c = child[q];
            c = FChildH();
            c.uptr = node[ch].uptr;
            c.relmap = S.rowptr[ch] + node[ch].c;
            c.nb = node[ch].r - node[ch].c;
            c.cbnd = (int)cbnd.size();
            const int32_t *rm = S.relmap + c.relmap;
            const FNodeH &m = node[p];
            int32_t at = 0;
            for (int I = 0; I <= m.nt; I++) {
                const int row = I == m.nt ? m.r : I < m.nkb ? I * FT : m.c + (I - m.nkb) * FT;
                at = (int32_t)(std::lower_bound(rm + at, rm + c.nb, row) - rm);
                cbnd.push_back(at);
            }
        }
    std::vector<FTaskH> t;
    std::vector<int32_t> key;
    t.reserve(ntask);
    key.reserve(ntask);
    int32_t kmin = 0, kmax = 0;
    auto emit = [&](int kind, int s, int I, int J, int k) {
        t.push_back({kind, s, I, J});
        key.push_back(k);
        kmin = std::min(kmin, k);
        kmax = std::max(kmax, k);
    };
    for (int32_t s = 0; s < ns; s++) {
        const FNodeH &m = node[s];
        if (is_small(s)) {
            emit(FK_SMALL, s, 0, 0, start[s]);
            continue;
        }
        const int up = m.parent < 0 ? 0 : start[m.parent];
        const int tp = m.parent < 0 ? 0 : kRes * (kFront + kStep * node[m.parent].nkb);
        for (int J = 0; J < m.nkb; J++) {
            emit(FK_DIAG, s, J, J, start[s] - kRes * kStep * J);
            for (int I = J + 1; I < m.nt; I++) emit(FK_ROWS, s, I, J, start[s] - kRes * (kStep * J + 4));
        }
        for (int J = m.nkb; J < m.nt; J++)
            for (int I = J; I < m.nt; I++) emit(FK_SCHUR, s, I, J, up + kRes * 8);
        for (int i = 1; i < m.nkb; i++)
            for (int j = 0; j < i; j++) emit(FK_INV, s, i, j, start[s] - kRes * (kStep * i + 20));
        for (int J = 0; J < m.nkb; J++)
            for (int I = m.nkb; I < m.nt; I++) emit(FK_WMUL, s, I, J, up - kRes * 2 - tp / 2);
    }
    const int64_t range = (int64_t)kmax - kmin + 1;
    tasks.resize(t.size());
    if (range <= 4 * (int64_t)t.size() + 65536) {
        std::vector<int32_t> cnt(range + 1, 0);
        for (int32_t k : key) cnt[kmax - k + 1]++;
        for (int64_t q = 0; q < range; q++) cnt[q + 1] += cnt[q];
        for (size_t i = 0; i < t.size(); i++) tasks[cnt[kmax - key[i]]++] = t[i];
    } else {
        std::vector<int32_t> ord(t.size());
        for (size_t i = 0; i < t.size(); i++) ord[i] = (int32_t)i;
        std::stable_sort(ord.begin(), ord.end(), [&](int32_t x, int32_t y) { return key[x] > key[y]; });
        for (size_t i = 0; i < t.size(); i++) tasks[i] = t[ord[i]];
    }
    *storage = off;
    *nflags = nfl;
}

template <class Tp>
static int dmalloc(Tp **p, size_t cnt, cudaStream_t st) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaMemPool_t pool = device_pool(dev);
    const size_t bytes = (cnt ? cnt : 1) * sizeof(Tp);
    cudaError_t e = pool ? cudaMallocFromPoolAsync((void **)p, bytes, pool, st)
                         : cudaMallocAsync((void **)p, bytes, st);
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return SPEIGS_ERR_MEM;
    }
    return 0;
}
template <class Tp>
static int dupload(Tp **p, const Tp *h, size_t cnt, cudaStream_t st) {
    int rc = dmalloc(p, cnt, st);
    if (rc) return rc;
    if (cnt) {
        cudaMemcpyAsync(*p, h, cnt * sizeof(Tp), cudaMemcpyHostToDevice, st);
        note_h2d((long long)(cnt * sizeof(Tp)));
    }
    return 0;
}

}  // namespace

template <> MultifrontalPlanT<Real>::~MultifrontalPlanT() { release(0); }

template <> void MultifrontalPlanT<Real>::release(cudaStream_t st) {
    void **ptrs[] = {(void **)&d_params_, (void **)&d_perm_, (void **)&d_rows_, (void **)&d_relmap_,
                     (void **)&d_cbnd_, (void **)&d_fnode_, (void **)&d_fchild_, (void **)&d_ftask_,
                     (void **)&d_fsync_, (void **)&d_acolptr_, (void **)&d_atpos_, (void **)&d_asrc_,
                     (void **)&d_front_, (void **)&d_G_, (void **)&d_u_, (void **)&d_yf_,
                     (void **)&d_x_, (void **)&d_meta_, (void **)&d_stask_, (void **)&d_bundle_,
                     (void **)&d_cptr_, (void **)&d_cidx_, (void **)&d_chunks_, (void **)&d_fpart_,
                     (void **)&d_bpart_, (void **)&d_cnt_, (void **)&d_sync_, (void **)&d_byf_,
                     (void **)&d_bx_, (void **)&d_bu_, (void **)&d_bfp_, (void **)&d_bbp_};
    for (void **p : ptrs)
        if (*p) {
            cudaFreeAsync(*p, st);
            *p = nullptr;
        }
    bw_ = 0;
}

template <> int64_t MultifrontalPlanT<Real>::solve_bytes() const {
    // G read once forward and once backward (lower triangle of the pivot
    // block plus the rows below), the row lists read twice, and the
    // right-hand side, the intermediate and the result vectors.
    return 2 * ((int64_t)sizeof(Real) * g_total_ + 4 * nrows_total_) + 24 * (int64_t)n_;
}

template <> int MultifrontalPlanT<Real>::init(const spx_symbolic &S, const int64_t *rowptr, const int32_t *col,
                           cudaStream_t st) {
    n_ = S.n;
    ns_ = S.nsuper;
    nlevels_ = S.nlevels;
    flops_ = S.flops;
    nrows_total_ = S.rowptr[ns_];
    const int32_t n = n_, ns = ns_;
    try {
        std::vector<int64_t> gptr(ns + 1, 0), uptr(ns + 1, 0);
        int64_t gtri = 0;
        for (int32_t s = 0; s < ns; s++) {
            int64_t r = S.rowptr[s + 1] - S.rowptr[s], c = S.sfirst[s + 1] - S.sfirst[s];
            gptr[s + 1] = gptr[s] + ((r + kLdgA - 1) & ~(int64_t)(kLdgA - 1)) * c;
            uptr[s + 1] = uptr[s] + (r - c);
            gtri += c * (c + 1) / 2 + (r - c) * c;
        }
        g_total_ = gtri;
        u_total_ = uptr[ns];
        // The assembly entries, the solve gather lists and the child tile
        // bounds are independent of the task lists: they are built on side
        // threads while this thread builds the factor and solve task lists.
        std::vector<int32_t> acolptr(n + 1, 0);
        std::vector<int32_t> atpos, asrc;
        std::vector<int32_t> cptr(nrows_total_ + 1, 0), cidx;
        std::vector<int32_t> cbnd;
        std::vector<FNodeH> fnode(ns);
        std::vector<FChildH> fchild(S.child_ptr[ns]);
        std::vector<FTaskH> ftask;
        TaskGroup side(rowptr[n] >= (1 << 17));
        side.run([&] {
            // assembly entries: for new column j, the entries of A's column
            // perm[j] with new row index >= j, as (row position in the front,
            // index into the CSR values), sorted by row position
            // (counted per column first, so that ranges of supernodes fill
            // their own columns' slices in parallel)
            parallel_ranges(n, 16384, [&](int64_t lo, int64_t hi) {
                for (int64_t j = lo; j < hi; j++) {
                    const int32_t o = S.perm[j];
                    int32_t c = 0;
                    for (int64_t p = rowptr[o]; p < rowptr[o + 1]; p++) c += S.iperm[col[p]] >= j;
                    acolptr[j + 1] = c;
                }
            });
            for (int32_t j = 0; j < n; j++) acolptr[j + 1] += acolptr[j];
            atpos.resize(acolptr[n]);
            asrc.resize(acolptr[n]);
            parallel_ranges(ns, 128, [&](int64_t lo, int64_t hi) {
                std::vector<int32_t> pos(n, -1);
                std::vector<std::pair<int32_t, int32_t>> tmp;
                for (int64_t s = lo; s < hi; s++) {
                    const int64_t r0 = S.rowptr[s], r1 = S.rowptr[s + 1];
                    for (int64_t t = r0; t < r1; t++) pos[S.rows[t]] = (int32_t)(t - r0);
                    for (int32_t j = S.sfirst[s]; j < S.sfirst[s + 1]; j++) {
                        const int32_t o = S.perm[j];
                        tmp.clear();
                        for (int64_t p = rowptr[o]; p < rowptr[o + 1]; p++) {
                            const int32_t i = S.iperm[col[p]];
                            if (i < j) continue;
                            tmp.emplace_back(pos[i], (int32_t)p);
                        }
                        std::sort(tmp.begin(), tmp.end());
                        int32_t d = acolptr[j];
                        for (auto &e : tmp) { atpos[d] = e.first; asrc[d] = e.second; d++; }
                    }
                    for (int64_t t = r0; t < r1; t++) pos[S.rows[t]] = -1;
                }
            });
        });
        side.run([&] {
            // gather lists: for every front row (global row-list index g) the
            // update-vector entries of the children that land on it, children in
            // their fixed order
            for (int32_t par = 0; par < ns; par++)
                for (int32_t q = S.child_ptr[par]; q < S.child_ptr[par + 1]; q++) {
                    const int ch = S.child_list[q];
                    const int cc = S.sfirst[ch + 1] - S.sfirst[ch];
                    for (int64_t t = S.rowptr[ch] + cc; t < S.rowptr[ch + 1]; t++)
                        cptr[S.rowptr[par] + S.relmap[t] + 1]++;
                }
            for (int64_t g = 0; g < nrows_total_; g++) cptr[g + 1] += cptr[g];
            cidx.assign(cptr[nrows_total_], 0);
            {
                std::vector<int32_t> fill(cptr.begin(), cptr.end() - 1);
                for (int32_t par = 0; par < ns; par++)
                    for (int32_t q = S.child_ptr[par]; q < S.child_ptr[par + 1]; q++) {
                        const int ch = S.child_list[q];
                        const int cc = S.sfirst[ch + 1] - S.sfirst[ch];
                        for (int64_t t = S.rowptr[ch] + cc; t < S.rowptr[ch + 1]; t++)
                            cidx[fill[S.rowptr[par] + S.relmap[t]]++] =
                                (int32_t)(uptr[ch] + (t - S.rowptr[ch] - cc));
                    }
            }
        });
        // factor nodes, tile storage and the tile task queue (nothing below
        // reads them before the uploads)
        side.run([&] { plan_factor_tasks(S, gptr.data(), fnode, fchild, cbnd, ftask, &front_total_, &nflags_); });
        // solve: per-supernode metadata and the task queue.  Forward tasks
        // level by level from the leaves (tiles of large supernodes first,
        // then bundles of up to 8 small ones), then backward tasks level by
        // level from the roots.  Every task depends only on earlier tasks.
        std::vector<SNodeH> meta(ns);
        auto small = [&](int r, int c) { return c <= kWarpMaxC && r <= kWarpMaxR; };
        std::vector<STaskH> tasks_s;
        std::vector<int32_t> bundle, fc_base, fc_n, bc_base, bc_n;
        int32_t fslots = 0, bslots = 0;
        // one thread per tiny leaf; everything else small goes to a warp
        auto tiny_leaf = [&](int s2) {
            return meta[s2].c <= kTinyC && meta[s2].r <= kTinyR && meta[s2].nchild == 0;
        };
        for (int32_t s2 = 0; s2 < ns; s2++) {
            const int r = (int)(S.rowptr[s2 + 1] - S.rowptr[s2]);
            const int c = S.sfirst[s2 + 1] - S.sfirst[s2];
            SNodeH &m = meta[s2];
            m.first = S.sfirst[s2]; m.c = c; m.r = r; m.ldg = (r + kLdgA - 1) & ~(kLdgA - 1);
            m.parent = S.sparent[s2];
            m.nchild = S.child_ptr[s2 + 1] - S.child_ptr[s2];
            m.nrc = (r + kST - 1) / kST;
            m.ncc = (c + kST - 1) / kST;
            m.gptr = gptr[s2]; m.g0 = S.rowptr[s2]; m.uptr = uptr[s2];
            m.fwd_expect = 0;
            m.bwd_expect = 0;
        }
        // completions a supernode reports: one per row chunk (forward) or
        // column chunk (backward) when it is cut into tiles, else one
        auto fwd_done_count = [&](int s2) {
            return small(meta[s2].r, meta[s2].c) ? 1 : meta[s2].nrc;
        };
        auto bwd_done_count = [&](int s2) {
            return small(meta[s2].r, meta[s2].c) ? 1 : meta[s2].ncc;
        };
        for (int32_t s2 = 0; s2 < ns; s2++) {
            const int p2 = meta[s2].parent;
            if (p2 >= 0) {
                meta[p2].fwd_expect += fwd_done_count(s2);
                meta[s2].bwd_expect = bwd_done_count(p2);
            } else {
                meta[s2].bwd_expect = fwd_done_count(s2);
            }
        }
        // The small supernodes of a level are bundled by decreasing work (rows
        // per lane, then pivots): a bundle's warps then finish together, and
        // the longest bundles are dequeued first.  Supernodes of one level do
        // not depend on each other, and each is computed the same way in any
        // bundle, so the results do not change.
        auto sort_by_work = [&](std::vector<int32_t> &v) {
            std::stable_sort(v.begin(), v.end(), [&](int32_t x, int32_t y2) {
                const int qx = (meta[x].r + 31) / 32, qy = (meta[y2].r + 31) / 32;
                if (qx != qy) return qx > qy;
                return meta[x].c > meta[y2].c;
            });
        };
        // Warp tasks: a small supernode whose whole subtree is small is solved
        // by one warp that dequeues it on its own (a tiny leaf by one lane of
        // a warp, 32 to a task), in a phase before (forward) or after
        // (backward) the block tasks.  A warp task then never waits for a
        // block task in the forward pass, and no block task waits for a warp
        // task of the backward pass, so neither phase can stall the other.
        std::vector<char> warpable(ns, 0);
        for (int l = 0; l < S.nlevels; l++)
            for (int32_t q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
                const int s2 = S.level_sup[q];
                bool ok = small(meta[s2].r, meta[s2].c);
                for (int32_t e = S.child_ptr[s2]; ok && e < S.child_ptr[s2 + 1]; e++)
                    ok = warpable[S.child_list[e]] != 0;
                warpable[s2] = ok;
            }
        std::vector<STaskH> wtasks_f, wtasks_b;
        auto emit_warp_level = [&](int l, bool fwd) {
            std::vector<int32_t> sm, ti;
            for (int32_t q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
                const int s2 = S.level_sup[q];
                if (!warpable[s2]) continue;
                if (tiny_leaf(s2)) ti.push_back(s2);
                else sm.push_back(s2);
            }
            sort_by_work(sm);
            std::vector<STaskH> &out = fwd ? wtasks_f : wtasks_b;
            for (int32_t s2 : sm) {
                out.push_back({fwd ? ST_FWD_BUNDLE : ST_BWD_BUNDLE, 0, 0, 0, 0,
                               (int)bundle.size(), 1, 0});
                bundle.push_back(s2);
            }
            for (size_t b0 = 0; b0 < ti.size(); b0 += 32) {
                const int nb = (int)std::min<size_t>(32, ti.size() - b0);
                out.push_back({fwd ? ST_FWD_THREADS : ST_BWD_THREADS, 0, 0, 0, 0,
                               (int)bundle.size(), nb, 0});
                bundle.insert(bundle.end(), ti.begin() + b0, ti.begin() + b0 + nb);
            }
        };
        for (int l = 0; l < S.nlevels; l++) emit_warp_level(l, true);
        for (int l = S.nlevels - 1; l >= 0; l--) emit_warp_level(l, false);
        for (int l = 0; l < S.nlevels; l++) {
            for (int32_t q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
                const int s2 = S.level_sup[q];
                const int r = meta[s2].r, c = meta[s2].c;
                if (small(r, c)) continue;
                const int nI = meta[s2].nrc, nS = (c + kStrip - 1) / kStrip;
                for (int I = 0; I < nI; I++) {
                    // strip S can hold a nonzero of row chunk I iff the chunk's
                    // last row >= the strip's first column
                    const int smax = std::min(nS - 1, (std::min(r, (I + 1) * kST) - 1) / kStrip);
                    const int chunk = (int)fc_base.size();
                    fc_base.push_back(fslots);
                    fc_n.push_back(smax + 1);
                    fslots += smax + 1;
                    for (int S2 = 0; S2 <= smax; S2++)
                        tasks_s.push_back({ST_FWD_TILE, s2, I, S2, chunk, 0, 0, 0});
                }
            }
            std::vector<int32_t> sm, ti;
            for (int32_t q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
                const int s2 = S.level_sup[q];
                if (warpable[s2]) continue;
                if (tiny_leaf(s2)) ti.push_back(s2);
                else if (small(meta[s2].r, meta[s2].c)) sm.push_back(s2);
            }
            sort_by_work(sm);
            for (size_t b0 = 0; b0 < sm.size(); b0 += kSWarps) {
                const int nb = (int)std::min<size_t>(kSWarps, sm.size() - b0);
                tasks_s.push_back({ST_FWD_BUNDLE, 0, 0, 0, 0, (int)bundle.size(), nb, 0});
                bundle.insert(bundle.end(), sm.begin() + b0, sm.begin() + b0 + nb);
            }
            for (size_t b0 = 0; b0 < ti.size(); b0 += kSThreads) {
                const int nb = (int)std::min<size_t>(kSThreads, ti.size() - b0);
                tasks_s.push_back({ST_FWD_THREADS, 0, 0, 0, 0, (int)bundle.size(), nb, 0});
                bundle.insert(bundle.end(), ti.begin() + b0, ti.begin() + b0 + nb);
            }
        }
        for (int l = S.nlevels - 1; l >= 0; l--) {
            for (int32_t q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
                const int s2 = S.level_sup[q];
                const int r = meta[s2].r, c = meta[s2].c;
                if (small(r, c)) continue;
                const int nJ = meta[s2].ncc, nS = (r + kStrip - 1) / kStrip;
                for (int J = 0; J < nJ; J++) {
                    // row strips from the one holding the chunk's first column
                    const int smin = (J * kST) / kStrip;
                    const int chunk = (int)bc_base.size();
                    bc_base.push_back(bslots);
                    bc_n.push_back(nS - smin);
                    bslots += nS - smin;
                    for (int S2 = smin; S2 < nS; S2++)
                        tasks_s.push_back({ST_BWD_TILE, s2, J, S2, chunk, 0, 0, 0});
                }
            }
            std::vector<int32_t> sm, ti;
            for (int32_t q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
                const int s2 = S.level_sup[q];
                if (warpable[s2]) continue;
                if (tiny_leaf(s2)) ti.push_back(s2);
                else if (small(meta[s2].r, meta[s2].c)) sm.push_back(s2);
            }
            sort_by_work(sm);
            for (size_t b0 = 0; b0 < sm.size(); b0 += kSWarps) {
                const int nb = (int)std::min<size_t>(kSWarps, sm.size() - b0);
                tasks_s.push_back({ST_BWD_BUNDLE, 0, 0, 0, 0, (int)bundle.size(), nb, 0});
                bundle.insert(bundle.end(), sm.begin() + b0, sm.begin() + b0 + nb);
            }
            for (size_t b0 = 0; b0 < ti.size(); b0 += kSThreads) {
                const int nb = (int)std::min<size_t>(kSThreads, ti.size() - b0);
                tasks_s.push_back({ST_BWD_THREADS, 0, 0, 0, 0, (int)bundle.size(), nb, 0});
                bundle.insert(bundle.end(), ti.begin() + b0, ti.begin() + b0 + nb);
            }
        }
        ntasks_ = (int)tasks_s.size();
        nfw_ = (int)wtasks_f.size();
        nbw_ = (int)wtasks_b.size();
        tasks_s.insert(tasks_s.end(), wtasks_f.begin(), wtasks_f.end());
        tasks_s.insert(tasks_s.end(), wtasks_b.begin(), wtasks_b.end());
        side.wait();
        int rc = 0;
        rc = rc ? rc : dupload(&d_cbnd_, cbnd.data(), cbnd.size(), st);
        rc = rc ? rc : dupload((FNodeH **)&d_fnode_, fnode.data(), fnode.size(), st);
        rc = rc ? rc : dupload((FChildH **)&d_fchild_, fchild.data(), fchild.size(), st);
        rc = rc ? rc : dupload((FTaskH **)&d_ftask_, ftask.data(), ftask.size(), st);
        nftask_ = (int)ftask.size();
        // tile flags | update tiles finished per parent | queue, status, error
        rc = rc ? rc : dmalloc(&d_fsync_, (size_t)nflags_ + ns + 3, st);
        rc = rc ? rc : dupload(&d_perm_, S.perm, n, st);
        rc = rc ? rc : dupload(&d_rows_, S.rows, (size_t)nrows_total_, st);
        rc = rc ? rc : dupload(&d_relmap_, S.relmap, (size_t)nrows_total_, st);
        rc = rc ? rc : dupload(&d_acolptr_, acolptr.data(), n + 1, st);
        rc = rc ? rc : dupload(&d_atpos_, atpos.data(), atpos.size(), st);
        rc = rc ? rc : dupload(&d_asrc_, asrc.data(), asrc.size(), st);
        {
            std::vector<int32_t> ch;
            ch.insert(ch.end(), fc_base.begin(), fc_base.end());
            ch.insert(ch.end(), fc_n.begin(), fc_n.end());
            ch.insert(ch.end(), bc_base.begin(), bc_base.end());
            ch.insert(ch.end(), bc_n.begin(), bc_n.end());
            rc = rc ? rc : dupload(&d_chunks_, ch.data(), ch.size(), st);
            nfc_ = (int32_t)fc_base.size();
            nbc_ = (int32_t)bc_base.size();
        }
        static_assert(sizeof(SNodeH) == sizeof(SNode), "metadata layout");
        static_assert(sizeof(STaskH) == sizeof(STask), "task layout");
        rc = rc ? rc : dupload((SNodeH **)&d_meta_, meta.data(), meta.size(), st);
        rc = rc ? rc : dupload((STaskH **)&d_stask_, tasks_s.data(), tasks_s.size(), st);
        rc = rc ? rc : dupload(&d_bundle_, bundle.data(), bundle.size(), st);
        fslots_ = fslots;
        bslots_ = bslots;
        rc = rc ? rc : dmalloc(&d_fpart_, (size_t)fslots * kST, st);
        rc = rc ? rc : dmalloc(&d_bpart_, (size_t)bslots * kST, st);
        rc = rc ? rc : dmalloc(&d_cnt_, (size_t)(nfc_ + nbc_), st);
        if (!rc) cudaMemsetAsync(d_cnt_, 0, sizeof(int) * (size_t)(nfc_ + nbc_), st);
        sync_ints_ = 2 + 5 * (size_t)ns;
        rc = rc ? rc : dmalloc(&d_sync_, sync_ints_, st);
        if (!rc) cudaMemsetAsync(d_sync_, 0, sizeof(int) * sync_ints_, st);
        rc = rc ? rc : dupload(&d_cptr_, cptr.data(), cptr.size(), st);
        rc = rc ? rc : dupload(&d_cidx_, cidx.data(), cidx.size(), st);
        rc = rc ? rc : dmalloc(&d_G_, (size_t)gptr[ns], st);
        // the solve reads whole tiles: the strictly upper part of every
        // inv(L11) block and the padding row stay zero for the plan's life
        if (!rc) cudaMemsetAsync(d_G_, 0, sizeof(Real) * (size_t)gptr[ns], st);
        rc = rc ? rc : dmalloc(&d_u_, (size_t)u_total_, st);
        rc = rc ? rc : dmalloc(&d_yf_, (size_t)n, st);
        rc = rc ? rc : dmalloc(&d_x_, (size_t)n, st);
        if (rc) return rc;
        // everything uploaded above comes from host vectors that die here
        if (cudaStreamSynchronize(st) != cudaSuccess) return SPEIGS_ERR_INTERNAL;
        // persistent grids
        int dev = 0, nsm = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(mf_factor, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FShared));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mf_factor, kFThreads, sizeof(FShared));
        if (per_sm <= 0 || nsm <= 0) return SPEIGS_ERR_INTERNAL;
        factor_grid_ = nsm * per_sm;
        solve_smem_ = solve_smem_bytes();
        if (solve_smem_ > 48 * 1024)
            cudaFuncSetAttribute(mf_solve_sf, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)solve_smem_);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mf_solve_sf, kSThreads, solve_smem_);
        if (per_sm <= 0 || nsm <= 0) return SPEIGS_ERR_INTERNAL;
        solve_grid_ = nsm * std::min(per_sm, 4);
    } catch (const std::bad_alloc &) {
        return SPEIGS_ERR_MEM;
    }
    return 0;
}

template <> int MultifrontalPlanT<Real>::factorize(const double *d_val, double shift, double pivtol,
                                cudaStream_t st) {
    if (!d_front_) {
        if (dmalloc(&d_front_, (size_t)front_total_, st)) return SPEIGS_ERR_MEM;
    }
    if (!d_params_) {
        if (dmalloc(&d_params_, 2, st)) return SPEIGS_ERR_MEM;
    }
    const double hp[2] = {shift, pivtol};
    cudaMemcpyAsync(d_params_, hp, sizeof hp, cudaMemcpyHostToDevice, st);
    note_h2d(sizeof hp);
    const size_t nsync = (size_t)nflags_ + ns_ + 3;
    cudaMemsetAsync(d_fsync_, 0, sizeof(int) * nsync, st);
    FactorArgs a;
    a.node = (const FNode *)d_fnode_;
    a.child = (const FChild *)d_fchild_;
    a.tasks = (const FTask *)d_ftask_;
    a.ntasks = nftask_;
    a.relmap = d_relmap_;
    a.cbnd = d_cbnd_;
    a.acolptr = d_acolptr_;
    a.atpos = d_atpos_;
    a.asrc = d_asrc_;
    a.val = d_val;
    a.params = d_params_;
    a.F = d_front_;
    a.G = d_G_;
    a.flags = d_fsync_;
    a.upd = d_fsync_ + nflags_;
    a.queue = a.upd + ns_;
    a.status = a.queue + 1;
    a.err = a.queue + 2;
    mf_factor<<<std::min(factor_grid_, nftask_), kFThreads, sizeof(FShared), st>>>(a);
    note_launch();
    int h[2] = {0, 0};
    cudaMemcpyAsync(h, a.status, sizeof h, cudaMemcpyDeviceToHost, st);
    note_d2h(sizeof h);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess || h[1]) {
        cudaGetLastError();
        return SPEIGS_ERR_INTERNAL;
    }
    return h[0] ? 1 : 0;
}

template <> void MultifrontalPlanT<Real>::solve(const double *b, double *x, cudaStream_t st,
                                                const int *skip) {
    SolveArgs a;
    a.meta = (const SNode *)d_meta_;
    a.tasks = (const STask *)d_stask_;
    a.ntasks = ntasks_;
    a.wtasks = a.tasks + ntasks_;
    a.nfw = nfw_;
    a.nbw = nbw_;
    a.ns = ns_;
    a.bundle = d_bundle_;
    a.perm = d_perm_;
    a.rows = d_rows_;
    a.cptr = d_cptr_;
    a.cidx = d_cidx_;
    a.G = d_G_;
    a.u = d_u_;
    a.yf = d_yf_;
    a.x = d_x_;
    a.fc_base = d_chunks_;
    a.fc_n = d_chunks_ + nfc_;
    a.bc_base = d_chunks_ + 2 * nfc_;
    a.bc_n = d_chunks_ + 2 * nfc_ + nbc_;
    a.fpart = d_fpart_;
    a.bpart = d_bpart_;
    a.fcnt = d_cnt_;
    a.bcnt = d_cnt_ + nfc_;
    a.sync = d_sync_;
    a.b = b;
    a.out = x;
    a.skip = skip;
    // queue, dependency counters and flags start at zero; the error word at
    // the end keeps its value so a failed solve stays visible until read
    cudaMemsetAsync(d_sync_, 0, sizeof(int) * (sync_ints_ - 1), st);
    mf_solve_sf<<<solve_grid_, kSThreads, solve_smem_, st>>>(a);
    note_launch();
}

namespace {
template <int NR>
void launch_bsolve(const BSolveArgs &a, int grid, size_t smem, cudaStream_t st) {
    mf_bsolve<NR><<<grid, kSThreads, smem, st>>>(a);
    note_launch();
}

template <int NR>
int bsolve_config(int *grid, size_t *smem) {
    *smem = bsolve_smem_bytes<NR>();
    if (cudaFuncSetAttribute(mf_bsolve<NR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)*smem) != cudaSuccess) {
        cudaGetLastError();
        return SPEIGS_ERR_INTERNAL;
    }
    int dev = 0, nsm = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mf_bsolve<NR>, kSThreads, *smem);
    if (per_sm <= 0 || nsm <= 0) return SPEIGS_ERR_INTERNAL;
    *grid = nsm * std::min(per_sm, 4);
    return 0;
}
}  // namespace

template <> int MultifrontalPlanT<Real>::solve_block(const double *B, int64_t ldb, double *X,
                                                     int64_t ldx, int nr, cudaStream_t st,
                                                     const int *skip, bool accumulate) {
    if (nr < 1 || nr > 32 || !d_meta_) return SPEIGS_ERR_ARG;
    const int w = (nr + 7) & ~7;          // 8, 16, 24 or 32 columns per row
    const int q = w / 8 - 1;
    if (w > bw_) {
        // (re)allocate the block buffers for rows of w doubles
        void *old[] = {d_byf_, d_bx_, d_bu_, d_bfp_, d_bbp_};
        for (void *p : old)
            if (p) cudaFreeAsync(p, st);
        d_byf_ = d_bx_ = d_bu_ = d_bfp_ = d_bbp_ = nullptr;
        bw_ = 0;
        int rc = 0;
        rc = rc ? rc : dmalloc(&d_byf_, (size_t)n_ * w, st);
        rc = rc ? rc : dmalloc(&d_bx_, (size_t)n_ * w, st);
        rc = rc ? rc : dmalloc(&d_bu_, (size_t)std::max<int64_t>(u_total_, 1) * w, st);
        rc = rc ? rc : dmalloc(&d_bfp_, (size_t)std::max(fslots_, 1) * kST * w, st);
        rc = rc ? rc : dmalloc(&d_bbp_, (size_t)std::max(bslots_, 1) * kST * w, st);
        if (rc) return rc;
        bw_ = w;
    }
    if (!bgrid_[q]) {
        const int rc = w == 8    ? bsolve_config<8>(&bgrid_[q], &bsmem_[q])
                       : w == 16 ? bsolve_config<16>(&bgrid_[q], &bsmem_[q])
                       : w == 24 ? bsolve_config<24>(&bgrid_[q], &bsmem_[q])
                                 : bsolve_config<32>(&bgrid_[q], &bsmem_[q]);
        if (rc) {
            bgrid_[q] = 0;
            return rc;
        }
    }
    BSolveArgs a;
    a.meta = (const SNode *)d_meta_;
    a.tasks = (const STask *)d_stask_;
    a.ntasks = ntasks_;
    a.wtasks = a.tasks + ntasks_;
    a.nfw = nfw_;
    a.nbw = nbw_;
    a.ns = ns_;
    a.bundle = d_bundle_;
    a.perm = d_perm_;
    a.rows = d_rows_;
    a.cptr = d_cptr_;
    a.cidx = d_cidx_;
    a.G = d_G_;
    a.u = d_bu_;
    a.yf = d_byf_;
    a.x = d_bx_;
    a.fc_base = d_chunks_;
    a.fc_n = d_chunks_ + nfc_;
    a.bc_base = d_chunks_ + 2 * nfc_;
    a.bc_n = d_chunks_ + 2 * nfc_ + nbc_;
    a.fpart = d_bfp_;
    a.bpart = d_bbp_;
    a.fcnt = d_cnt_;
    a.bcnt = d_cnt_ + nfc_;
    a.sync = d_sync_;
    a.bc = B;
    a.xc = X;
    a.ldb = ldb;
    a.ldx = ldx;
    a.nr = nr;
    a.accumulate = accumulate ? 1 : 0;
    a.skip = skip;
    cudaMemsetAsync(d_sync_, 0, sizeof(int) * (sync_ints_ - 1), st);
    if (w == 8)
        launch_bsolve<8>(a, bgrid_[q], bsmem_[q], st);
    else if (w == 16)
        launch_bsolve<16>(a, bgrid_[q], bsmem_[q], st);
    else if (w == 24)
        launch_bsolve<24>(a, bgrid_[q], bsmem_[q], st);
    else
        launch_bsolve<32>(a, bgrid_[q], bsmem_[q], st);
    return 0;
}

template <> int *MultifrontalPlanT<Real>::error_word() const { return d_sync_ ? d_sync_ + (sync_ints_ - 1) : nullptr; }

}  // namespace spx
