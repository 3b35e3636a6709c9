// Device multifrontal supernodal Cholesky (FP64) and the task-queue
// shift-invert solve.  See multifrontal.cuh for the storage scheme.
//
// The factorization is one persistent kernel over 64 x 64 tile tasks
// (mf_factor.cuh); the solve pair is another over panel tiles
// (mf_solve.cuh).  A
// pivot that is not positive records the failing column in a device status
// word (never a trap); the tasks after it do no work.
#include "multifrontal.cuh"
#include "../chain.cuh"
#include "../common.cuh"
#include "../counters.h"
#include "../host/parallel.h"

#include <algorithm>
#include <atomic>
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

// memory pool of the device (engine.cu): allocations are cached across calls
cudaMemPool_t device_pool(int dev);

namespace {

constexpr long kSpinLimit = 1L << 22;

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

// ---- bulk asynchronous copies into shared memory, tracked by an mbarrier
SPX_DEV uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
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

SPX_DEV void mbar_init_n(unsigned long long *bar, int n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(n) : "memory");
}
SPX_DEV void mbar_arrive(unsigned long long *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// FP64 tensor-core product, m8n8k4: lane = 4 g + t holds A[g][t], B[t][g] and
// D[g][2 t .. 2 t + 1]
SPX_DEV void dmma(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1) : "d"(a), "d"(b));
}

// The panel G of a supernode: blocks of 16 rows, each all c columns of 16
// rows, the row XORed by a function of the column (mf_solve.cuh says why).
// gswz: the XOR of column j; gix: the place of entry (i, j).
SPX_DEV int gswz(int j) { return sizeof(Real) == 8 ? (j & 3) << 2 : ((j >> 1) & 1) << 3; }
SPX_DEV int64_t gix(int i, int j, int c) {
    return ((int64_t)(i >> 4) * c + j) * 16 + ((i & 15) ^ gswz(j));
}

#include "mf_factor.cuh"
#include "mf_solve.cuh"


struct FNodeH {
    int first, c, r, unused0, parent, nchild, child0, expect;
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
// A task's key is an estimate of how early it can run (quarter microseconds):
// the longest path of column blocks below it, kStep for a column block of a
// front's diagonal chain and kFront for a front's assembly and hand-over.
// Tasks run in increasing key order, equal keys in the order they were made.
// The key grows along every dependency, which puts every task after the ones
// it waits for: a front starts after its children's update tiles, a column
// block after the one before it, rows after their diagonal tile, inverse
// tiles two column blocks behind the chain, W tiles last.  Starting the
// longest chains first instead (by the path above a task) or a mix of the two
// measured the same to 3 % (48^3 4.60 against 4.44 ms): the blocks held by
// tiles that wait for a chain cost what the chains gain.
static void plan_factor_tasks(const spx_symbolic &S, const int64_t *gptr,
                              std::vector<FNodeH> &node, std::vector<FChildH> &child,
                              std::vector<int32_t> &cbnd, std::vector<FTaskH> &tasks,
                              int64_t *storage, int64_t *nflags) {
    constexpr int kStep = 15, kFront = 12, kRes = 4;
    const int32_t ns = S.nsuper;
    int64_t off = 0, nfl = 0;
    std::vector<int64_t> early(ns, 0);           // key of a front's first task
    auto r4 = [](int64_t v) { return (v + 3) & ~(int64_t)3; };
    auto is_small = [&](int32_t s) { return node[s].nkb == 1 && node[s].nt <= 2; };
    for (int32_t s = 0; s < ns; s++) {
        FNodeH &m = node[s];
        m = FNodeH();
        m.first = S.sfirst[s];
        m.c = S.sfirst[s + 1] - S.sfirst[s];
        m.r = (int)(S.rowptr[s + 1] - S.rowptr[s]);
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
    auto span = [&](int32_t s) { return (int64_t)kRes * (kFront + kStep * node[s].nkb); };
    for (int32_t s = 0; s < ns; s++)
        if (node[s].parent >= 0) early[node[s].parent] = std::max(early[node[s].parent], early[s] + span(s));
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
    int32_t kmin = INT32_MAX, kmax = INT32_MIN;
    // `at`: quarter microseconds after the front's first task
    auto emit = [&](int kind, int s, int I, int J, int64_t at) {
        const int32_t k = (int32_t)(early[s] + at);
        t.push_back({kind, s, I, J});
        key.push_back(k);
        kmin = std::min(kmin, k);
        kmax = std::max(kmax, k);
    };
    for (int32_t s = 0; s < ns; s++) {
        const FNodeH &m = node[s];
        if (is_small(s)) {
            emit(FK_SMALL, s, 0, 0, 0);
            continue;
        }
        for (int J = 0; J < m.nkb; J++) {
            emit(FK_DIAG, s, J, J, kRes * kStep * J);
            for (int I = J + 1; I < m.nt; I++) emit(FK_ROWS, s, I, J, kRes * (kStep * J + 4));
        }
        for (int J = m.nkb; J < m.nt; J++)
            for (int I = J; I < m.nt; I++) emit(FK_SCHUR, s, I, J, kRes * (kStep * m.nkb + 4));
        for (int i = 1; i < m.nkb; i++)
            for (int j = 0; j < i; j++) emit(FK_INV, s, i, j, kRes * (kStep * i + kStep + 5));
        const int64_t tp = m.parent < 0 ? 0 : span(m.parent);
        for (int J = 0; J < m.nkb; J++)
            for (int I = m.nkb; I < m.nt; I++) emit(FK_WMUL, s, I, J, span(s) + kRes * (kStep + 6) + tp / 2);
    }
    const int64_t range = (int64_t)kmax - kmin + 1;
    tasks.resize(t.size());
    if (range <= 4 * (int64_t)t.size() + 65536) {
        std::vector<int32_t> cnt(range + 1, 0);
        for (int32_t k : key) cnt[k - kmin + 1]++;
        for (int64_t q = 0; q < range; q++) cnt[q + 1] += cnt[q];
        for (size_t i = 0; i < t.size(); i++) tasks[cnt[key[i] - kmin]++] = t[i];
    } else {
        std::vector<int32_t> ord(t.size());
        for (size_t i = 0; i < t.size(); i++) ord[i] = (int32_t)i;
        std::stable_sort(ord.begin(), ord.end(), [&](int32_t x, int32_t y) { return key[x] < key[y]; });
        for (size_t i = 0; i < t.size(); i++) tasks[i] = t[ord[i]];
    }
    *storage = off;
    *nflags = nfl;
}

// A supernode as the solves' tile queues see it, and its place in one of
// them: its first task and its first partial-sum slot.
struct SPlanNode {
    int first, c, r, parent;
    int has_child, probe;            // see STask; probe: of a forward task
    long long g, rows, u;
};
struct SPlanEntry { int s, task0, slot0; };

// Tiles of a supernode: cw columns of a forward strip, fh row blocks of a
// forward tile, bw columns of a backward tile, bh row blocks of a backward
// strip.
struct SGeo { int nrb, cw, fh, bw, bh; };
__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ inline int imin(int a, int b) { return a < b ? a : b; }
__host__ __device__ inline int imax(int a, int b) { return a > b ? a : b; }
__host__ __device__ inline SGeo solve_geo(int c, int r, bool vec) {
    SGeo g;
    const int strip = vec ? kVecStrip : kBlkStrip, tall = vec ? kVecTall : kBlkTall;
    g.nrb = ceil_div(r, 16);
    g.cw = ceil_div(c, ceil_div(c, strip));
    g.bh = ceil_div(g.nrb, ceil_div(g.nrb, tall));
    if (vec) {
        g.fh = imax(1, imin(kVecRows / 16, kVecElems / (16 * g.cw)));
        g.bw = imax(1, imin(kBwdCols, kVecElems / (16 * g.bh)));
    } else {
        g.fh = kBlkRows / 16;
        // whole groups of eight columns
        g.bw = imax(8, imin(kBwdCols, kBlkElems / (16 * g.bh)) & ~7);
    }
    return g;
}
// strips of forward row chunk i: those that hold a nonzero of its rows (the
// pivot block is lower triangular); of backward column chunk i: the row
// blocks from the diagonal down
__host__ __device__ inline int fwd_strips(const SGeo &g, int c, int r, int i) {
    return ceil_div(imin(c, imin(r, (i + 1) * g.fh * 16)), g.cw);
}
__host__ __device__ inline int bwd_strips(const SGeo &g, int i) {
    return ceil_div(g.nrb - i * g.bw / 16, g.bh);
}

// The tasks of chunk i of an entry (forward: a row chunk, backward: a column
// chunk), task = its strips in order.
__host__ __device__ inline void expand_chunk(const SPlanNode &m, const SGeo &g, bool fwd, int i,
                                             int task, int slot, const int32_t *cptr, STask *out) {
    STask k = {};
    k.kind = fwd ? SK_FWD : SK_BWD;
    k.first = m.first;
    k.c = m.c;
    k.r = m.r;
    k.rows = m.rows;
    k.u = m.u;
    k.has_child = m.has_child;
    k.slot0 = slot;
    if (fwd) {
        const int b0 = i * g.fh;
        k.probe_at = m.has_child ? 1 : 0;
        k.probe = m.has_child ? m.probe : 0;
        k.i0 = b0 * 16;
        k.nrb = imin(g.fh, g.nrb - b0);
        k.nrow = imin(m.r - k.i0, k.nrb * 16);
        k.nstrip = fwd_strips(g, m.c, m.r, i);
        const int cols = imin(m.c, k.i0 + k.nrow), rh = k.i0 + k.nrow;
        k.rl0 = cptr[m.rows + k.i0];
        k.rln = rh > imax(k.i0, m.c) ? cptr[m.rows + rh] - k.rl0 : 0;   // rows below the pivots
        for (int q = 0; q < k.nstrip; q++) {
            k.strip = q;
            k.j0 = q * g.cw;
            k.jn = imin(g.cw, cols - k.j0);
            k.pl0 = cptr[m.rows + k.j0];
            k.pln = cptr[m.rows + k.j0 + k.jn] - k.pl0;
            k.g = m.g + ((long long)b0 * m.c + k.j0) * 16;
            out[task + q] = k;
        }
    } else {
        // the probe: the parent's first pivot, in its tallest column chunk; a
        // root waits for its own last pivot of the forward pass
        k.probe_at = m.parent >= 0 ? 2 : 3;
        k.probe = m.parent >= 0 ? m.parent : m.first + m.c - 1;
        k.j0 = i * g.bw;
        k.jn = imin(g.bw, m.c - k.j0);
        k.nstrip = bwd_strips(g, i);
        const int b0 = k.j0 / 16, bh = ceil_div(g.nrb - b0, k.nstrip);
        for (int q = 0; q < k.nstrip; q++) {
            const int at = b0 + q * bh;
            k.strip = q;
            k.i0 = at * 16;
            k.nrb = imin(bh, g.nrb - at);
            k.nrow = imin(m.r - k.i0, k.nrb * 16);
            k.g = m.g + ((long long)at * m.c + k.j0) * 16;
            out[task + q] = k;
        }
    }
}

// Entry e (one warp) of a queue whose first ns entries are forward.  The
// records are 128 bytes a tile, so they are made on the device from 56 bytes
// a supernode instead of being built and uploaded by the host.
__global__ void __launch_bounds__(128)
expand_tasks_kernel(const SPlanNode *__restrict__ node, const SPlanEntry *__restrict__ ent, int ns,
                    bool vec, const int32_t *__restrict__ cptr, STask *__restrict__ out) {
    const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (e >= 2 * ns) return;
    const SPlanEntry en = ent[e];
    const SPlanNode m = node[en.s];
    const SGeo g = solve_geo(m.c, m.r, vec);
    const bool fwd = e < ns;
    const int nchunk = fwd ? ceil_div(g.nrb, g.fh) : ceil_div(m.c, g.bw);
    int task = en.task0, slot = en.slot0, at = 0;
    for (int i = lane; i < nchunk; i += 32) {
        for (; at < i; at++) {
            const int ns2 = fwd ? fwd_strips(g, m.c, m.r, at) : bwd_strips(g, at);
            task += ns2;
            slot += ns2 - 1;
        }
        expand_chunk(m, g, fwd, i, task, slot, cptr, out);
    }
}

// The tile queue of the solves for one right-hand side (vec) or a block: the
// supernodes in the order of their forward, then of their backward tasks.
//
// Keys (us, an estimate) order the queue: a forward task by the path that
// follows it up to the root, a backward task by the path that follows it down
// to the deepest leaf, both decreasing, so a task comes after the ones it
// waits for and the longest chains are started first.
static void plan_solve_order(const spx_symbolic &S, bool vec, std::vector<SPlanEntry> &ent,
                             SolvePlan *plan) {
    const int32_t ns = S.nsuper;
    std::vector<int32_t> fkey(ns), bkey(ns, 0);
    std::vector<SGeo> geo(ns);
    auto cols = [&](int32_t s) { return S.sfirst[s + 1] - S.sfirst[s]; };
    auto rows = [&](int32_t s) { return (int)(S.rowptr[s + 1] - S.rowptr[s]); };
    for (int32_t s = 0; s < ns; s++) {
        geo[s] = solve_geo(cols(s), rows(s), vec);
        fkey[s] = 3 + 2 * (cols(s) > geo[s].cw);
        bkey[s] += 3 + 2 * (geo[s].nrb > geo[s].bh);   // children came before: their largest is in
        const int32_t p = S.sparent[s];
        if (p >= 0) bkey[p] = std::max(bkey[p], bkey[s]);
    }
    int32_t kmax = 0;
    for (int32_t s = ns - 1; s >= 0; s--) {
        if (S.sparent[s] >= 0) fkey[s] += fkey[S.sparent[s]];
        kmax = std::max(kmax, std::max(fkey[s], bkey[s]));
    }
    // supernodes in decreasing key order (stable): counting sort when the keys
    // are few, as they are for any but a chain
    auto order = [&](const std::vector<int32_t> &key) {
        std::vector<int32_t> ord(ns);
        if (kmax <= 4 * (int64_t)ns + 65536) {
            std::vector<int32_t> cnt(kmax + 2, 0);
            for (int32_t s = 0; s < ns; s++) cnt[kmax - key[s] + 1]++;
            for (int32_t q = 0; q <= kmax; q++) cnt[q + 1] += cnt[q];
            for (int32_t s = 0; s < ns; s++) ord[cnt[kmax - key[s]]++] = s;
        } else {
            for (int32_t s = 0; s < ns; s++) ord[s] = s;
            std::stable_sort(ord.begin(), ord.end(), [&](int32_t x, int32_t y) { return key[x] > key[y]; });
        }
        return ord;
    };
    ent.clear();
    ent.reserve(2 * (size_t)ns);
    int32_t task = 0, fslots = 0, bslots = 0;
    for (int32_t s : order(fkey)) {
        ent.push_back({s, task, fslots});
        const SGeo &g = geo[s];
        for (int i = 0; i < ceil_div(g.nrb, g.fh); i++) {
            const int n = fwd_strips(g, cols(s), rows(s), i);
            task += n;
            fslots += n - 1;
        }
    }
    for (int32_t s : order(bkey)) {
        ent.push_back({s, task, bslots});
        const SGeo &g = geo[s];
        for (int i = 0; i < ceil_div(cols(s), g.bw); i++) {
            const int n = bwd_strips(g, i);
            task += n;
            bslots += n - 1;
        }
    }
    plan->ntasks = task;
    plan->fslots = std::max(1, fslots);
    plan->bslots = std::max(1, bslots);
}

template <int NR>
static int solve_config(int *grid) {
    int dev = 0, nsm = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (cudaFuncSetAttribute(mf_solve<NR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(SShared<NR>)) != cudaSuccess) {
        cudaGetLastError();
        return SPEIGS_ERR_INTERNAL;
    }
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mf_solve<NR>, SShared<NR>::kThreads,
                                                  sizeof(SShared<NR>));
    if (per_sm <= 0 || nsm <= 0) return SPEIGS_ERR_INTERNAL;
    *grid = nsm * per_sm;
    return 0;
}
template <class Tp>
static int dmalloc(Tp **p, size_t cnt, cudaStream_t st) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaMemPool_t pool = device_pool(dev);
    // 16 bytes more than asked for: the solve copies its index lists in
    // aligned 16-byte pieces, whose last one may reach past the list's end
    const size_t bytes = (cnt ? cnt : 1) * sizeof(Tp) + 16;
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
                     (void **)&d_fsync_, (void **)&d_acolptr_, (void **)&d_atpos_, (void **)&d_acolj_,
                     (void **)&d_asrc_,
                     (void **)&d_front_, (void **)&d_G_, (void **)&d_vtask_, (void **)&d_btask_,
                     (void **)&d_cptr_, (void **)&d_cidx_, (void **)&d_sync_, (void **)&d_sval_[0],
                     (void **)&d_sval_[1], (void **)&d_sval_[2], (void **)&d_sval_[3],
                     (void **)&d_sval_[4]};
    for (void **p : ptrs)
        if (*p) {
            cudaFreeAsync(*p, st);
            *p = nullptr;
        }
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
            gptr[s + 1] = gptr[s] + ((r + 15) & ~(int64_t)15) * c;
            uptr[s + 1] = uptr[s] + (r - c);
            gtri += c * (c + 1) / 2 + (r - c) * c;
        }
        g_total_ = gtri;
        u_total_ = uptr[ns];
        // The assembly entries, the solve gather lists and the child tile
        // bounds are independent of the task lists: they are built on side
        // threads while this thread builds the factor and solve task lists.
        std::vector<int32_t> acolptr(n + 1, 0);
        std::vector<int32_t> atpos, acolj, asrc;
        std::atomic<int> dup{0};
        std::vector<int32_t> cptr(nrows_total_ + 1, 0), cidx;
        std::vector<char> longlist(ns, 0);          // some gather list is long
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
            acolj.resize(acolptr[n]);
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
                        for (auto &e : tmp) {
                            if (d > acolptr[j] && atpos[d - 1] == e.first) dup = 1;
                            atpos[d] = e.first;
                            acolj[d] = j;
                            asrc[d++] = e.second;
                        }
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
                        if (++cptr[S.rowptr[par] + S.relmap[t] + 1] > kLongList) longlist[par] = 1;
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
        // the solves' tile queues
        std::vector<SPlanNode> pnode(ns);
        std::vector<SPlanEntry> vent, bent;
        side.run([&] { plan_solve_order(S, true, vent, &vplan_); });
        plan_solve_order(S, false, bent, &bplan_);
        for (int32_t s = 0; s < ns; s++) {
            SPlanNode &m = pnode[s];
            m.first = S.sfirst[s];
            m.c = S.sfirst[s + 1] - S.sfirst[s];
            m.r = (int)(S.rowptr[s + 1] - S.rowptr[s]);
            m.parent = S.sparent[s] >= 0 ? S.sfirst[S.sparent[s]] : -1;
            m.has_child = S.child_ptr[s + 1] > S.child_ptr[s];
            // the probe: the last update row of the tallest child, whose row
            // chunk has the most strips
            int32_t tall = 0;
            m.probe = 0;
            for (int32_t q = S.child_ptr[s]; q < S.child_ptr[s + 1]; q++) {
                const int32_t ch = S.child_list[q], rc = (int32_t)(S.rowptr[ch + 1] - S.rowptr[ch]);
                if (rc > tall) { tall = rc; m.probe = (int)(uptr[ch + 1] - 1); }
            }
            m.g = gptr[s];
            m.rows = S.rowptr[s];
            m.u = uptr[s];
        }
        side.wait();
        for (int32_t s = 0; s < ns; s++)
            if (longlist[s]) pnode[s].has_child = 2;
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
        rc = rc ? rc : dupload(&d_acolj_, acolj.data(), acolj.size(), st);
        rc = rc ? rc : dupload(&d_asrc_, asrc.data(), asrc.size(), st);
        dup_ = dup;
        // per column count 1, 8, 16, 24, 32: queue, blocks gone, copy in use;
        // then the error word
        rc = rc ? rc : dmalloc(&d_sync_, 16, st);
        if (!rc) cudaMemsetAsync(d_sync_, 0, sizeof(int) * 16, st);
        rc = rc ? rc : dupload(&d_cptr_, cptr.data(), cptr.size(), st);
        rc = rc ? rc : dupload(&d_cidx_, cidx.data(), cidx.size(), st);
        rc = rc ? rc : dmalloc((STask **)&d_vtask_, (size_t)vplan_.ntasks, st);
        rc = rc ? rc : dmalloc((STask **)&d_btask_, (size_t)bplan_.ntasks, st);
        SPlanNode *dn = nullptr;
        SPlanEntry *dv = nullptr, *db = nullptr;
        rc = rc ? rc : dupload(&dn, pnode.data(), pnode.size(), st);
        rc = rc ? rc : dupload(&dv, vent.data(), vent.size(), st);
        rc = rc ? rc : dupload(&db, bent.data(), bent.size(), st);
        if (!rc) {
            const int nblk = (2 * ns + 3) / 4;
            if (launch_plain(expand_tasks_kernel, nblk, 128, 0, st, dn, dv, ns, true, d_cptr_,
                             (STask *)d_vtask_) != cudaSuccess ||
                launch_plain(expand_tasks_kernel, nblk, 128, 0, st, dn, db, ns, false, d_cptr_,
                             (STask *)d_btask_) != cudaSuccess)
                rc = SPEIGS_ERR_INTERNAL;
        }
        if (dn) cudaFreeAsync(dn, st);
        if (dv) cudaFreeAsync(dv, st);
        if (db) cudaFreeAsync(db, st);
        rc = rc ? rc : dmalloc(&d_G_, (size_t)gptr[ns], st);
        // the solve reads whole tiles: the strictly upper part of every
        // inv(L11) block and the padding row stay zero for the plan's life
        if (!rc) cudaMemsetAsync(d_G_, 0, sizeof(Real) * (size_t)gptr[ns], st);
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
        if (int e = solve_setup(0, st)) return e;
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
    a.acolj = d_acolj_;
    a.asrc = d_asrc_;
    a.dup = dup_;
    a.val = d_val;
    a.params = d_params_;
    a.F = d_front_;
    a.G = d_G_;
    a.flags = d_fsync_;
    a.upd = d_fsync_ + nflags_;
    a.queue = a.upd + ns_;
    a.status = a.queue + 1;
    a.err = a.queue + 2;
    cudaError_t e = launch_plain(mf_factor, std::min(factor_grid_, nftask_), kFThreads,
                                 sizeof(FShared), st, a);
    int h[2] = {0, 0};
    cudaMemcpyAsync(h, a.status, sizeof h, cudaMemcpyDeviceToHost, st);
    note_d2h(sizeof h);
    if (cudaError_t es = cudaStreamSynchronize(st)) e = es;
    if (e != cudaSuccess || h[1]) {
        cudaGetLastError();
        return SPEIGS_ERR_INTERNAL;
    }
    return h[0] ? 1 : 0;
}

// The values that pass between the tasks of an nr-column solve (nr = 1 or a
// multiple of 8), both copies unset, on first use.
template <> int MultifrontalPlanT<Real>::solve_setup(int q, cudaStream_t st) {
    if (d_sval_[q]) return 0;
    const int nr = q ? 8 * q : 1;
    int rc = q == 0   ? solve_config<1>(&sgrid_[0])
             : q == 1 ? solve_config<8>(&sgrid_[1])
             : q == 2 ? solve_config<16>(&sgrid_[2])
             : q == 3 ? solve_config<24>(&sgrid_[3])
                      : solve_config<32>(&sgrid_[4]);
    if (rc) return rc;
    const SolvePlan &p = q ? bplan_ : vplan_;
    // u, yf, x, forward partial sums, backward partial sums
    const int64_t len = (u_total_ + 2 * (int64_t)n_ + (int64_t)p.fslots * (q ? kBlkRows : kVecRows) +
                         (int64_t)p.bslots * kBwdCols) * nr;
    sstride_[q] = (len + 1) & ~(int64_t)1;
    if ((rc = dmalloc(&d_sval_[q], (size_t)sstride_[q] * 2, st))) return rc;
    return launch_plain(fill_unset_kernel, 2 * 148, 256, 0, st, d_sval_[q], 2 * sstride_[q]) ==
                   cudaSuccess ? 0 : SPEIGS_ERR_INTERNAL;
}

template <> int MultifrontalPlanT<Real>::run_solve(int q, const double *B, int64_t ldb, double *X,
                                                   int64_t ldx, int nr, cudaStream_t st,
                                                   const int *skip, bool accumulate) {
    if (int rc = solve_setup(q, st)) return rc;
    const SolvePlan &p = q ? bplan_ : vplan_;
    const int w = q ? 8 * q : 1;
    SolveArgs a = {};
    a.tasks = (const STask *)(q ? d_btask_ : d_vtask_);
    a.ntasks = p.ntasks;
    a.perm = d_perm_;
    a.rows = d_rows_;
    a.cptr = d_cptr_;
    a.cidx = d_cidx_;
    a.G = d_G_;
    a.val = d_sval_[q];
    a.stride = sstride_[q];
    a.o_yf = u_total_ * w;
    a.o_x = a.o_yf + (int64_t)n_ * w;
    a.o_fp = a.o_x + (int64_t)n_ * w;
    a.o_bp = a.o_fp + (int64_t)p.fslots * (q ? kBlkRows : kVecRows) * w;
    a.sync = d_sync_ + 3 * q;
    a.err = error_word();
    a.bc = B;
    a.xc = X;
    a.ldb = ldb;
    a.ldx = ldx;
    a.nr = nr;
    a.accumulate = accumulate ? 1 : 0;
    a.skip = skip;
    const int grid = std::min(sgrid_[q], a.ntasks);
    const cudaError_t e =
        q == 0   ? launch_chained(mf_solve<1>, grid, kVecThreads, sizeof(SShared<1>), st, a)
        : q == 1 ? launch_chained(mf_solve<8>, grid, kBlkThreads, sizeof(SShared<8>), st, a)
        : q == 2 ? launch_chained(mf_solve<16>, grid, kBlkThreads, sizeof(SShared<16>), st, a)
        : q == 3 ? launch_chained(mf_solve<24>, grid, kBlkThreads, sizeof(SShared<24>), st, a)
                 : launch_chained(mf_solve<32>, grid, kBlkThreads, sizeof(SShared<32>), st, a);
    return e == cudaSuccess ? 0 : SPEIGS_ERR_INTERNAL;
}

template <> void MultifrontalPlanT<Real>::solve(const double *b, double *x, cudaStream_t st,
                                                const int *skip) {
    run_solve(0, b, n_, x, n_, 1, st, skip, false);
}

template <> int MultifrontalPlanT<Real>::solve_block(const double *B, int64_t ldb, double *X,
                                                     int64_t ldx, int nr, cudaStream_t st,
                                                     const int *skip, bool accumulate) {
    if (nr < 1 || nr > 32 || !d_btask_) return SPEIGS_ERR_ARG;
    return run_solve((nr + 7) / 8, B, ldb, X, ldx, nr, st, skip, accumulate);
}

template <> int *MultifrontalPlanT<Real>::error_word() const { return d_sync_ ? d_sync_ + 15 : nullptr; }

}  // namespace spx
