// The numeric factorization as one persistent kernel (included by
// multifrontal.cu inside its anonymous namespace, once per storage type).
//
// Every front is cut into 64 x 64 tiles: tiles of the pivots first, then
// tiles of the rows below.  A task computes one tile from start to end
// (left-looking): it assembles the tile (entries of A, the shift, the
// children's update matrices), subtracts the products of the finished tiles
// to its left and finishes it.  Tasks come from an atomic queue sorted by
// the earliest time they can run (the longest path below them), and wait on a
// flag per tile, so there is no barrier between column blocks or tree levels and no
// launch per step.  The queue order is topological (a task waits only for
// tasks before it, which running blocks hold), so the waits cannot deadlock
// whatever number of blocks is resident; they are bounded all the same.
//
//   FK_DIAG   (J,J), J < nkb : L_JJ and X_JJ = inv(L_JJ) of the tile
//   FK_ROWS   (I,J), J < nkb : L_IJ = T_IJ X_JJ^T
//   FK_SCHUR  (I,J), J >= nkb: a tile of the update matrix, for the parent
//   FK_INV    (i,j), j < i < nkb: X_ij = -X_ii sum_{j<=k<i} L_ik X_kj
//   FK_WMUL   (I,j), I >= nkb: W_Ij = sum_{j<=k<nkb} L_Ik X_kj
//   FK_SMALL  a whole front of at most 64 pivots and 64 rows below
//
// X and W are the panel G of the solve.  All products have the form
// acc += A_k B_k^T with A_k and B_k tiles stored by columns, so one loop
// serves them all (X_kj is kept transposed for that): a producer thread
// waits for the tiles' flags and copies 16-column chunks of both into a ring
// of four shared buffers (bulk copies, mbarriers), four warps multiply on
// the FP64 tensor cores, each a 32 x 32 quarter of the tile in registers.
//
// What bounds it: at the top of the tree the chain of diagonal tiles of the
// large separators (about 30 us a column block: 11 us for the 64 x 64
// Cholesky and inverse, two tile products and three hand-overs of about 2 us;
// a launch per step took 55), elsewhere the tiles' latencies -- 5 us of
// assembly and 3 us of stores around 2.2 us a product, two tiles an SM -- and
// then the FP64 pipe (1.4 of 4.4 ms at 48^3, 7.6 of 15.7 at 64^3).  Measured
// on 3-D grids, against one launch per column-block step (a graph of 590
// launches at 48^3) on the narrower supernodes of before: 20^3 2.0 -> 0.63 ms,
// 33x35x37 4.67 -> 1.76, 48^3 9.84 -> 4.45, 64^3 28.8 -> 15.7.
constexpr int FT = 64;
constexpr int kFConsumers = 128;
constexpr int kFThreads = kFConsumers + 32;
constexpr int kFStages = 4;
constexpr int kFChunk = 16;                    // columns per stage
enum { FK_DIAG = 0, FK_ROWS, FK_SCHUR, FK_INV, FK_WMUL, FK_SMALL };

struct FNode {          // per-supernode factor metadata (96 bytes)
    int4 a;             // first column, c, r, unused
    int4 b;             // parent, children, first child record, update tiles expected
    longlong2 p;        // pivot tile storage, update tile storage (in Reals)
    longlong2 g;        // panel offset, row-list offset
    int4 f;             // first tile flag, nkb, nt, unused
    int4 pad;
};
struct FChild {         // per child, in the parent's child order (32 bytes)
    long long uptr;     // its update tile storage
    long long relmap;   // offset of its update rows' positions in the parent
    int cbnd;           // offset of its bounds per 64-row tile of the parent
    int nb;             // its update rows
    int pad[2];
};
struct FTask { int kind, s, I, J; };

struct FactorArgs {
    const FNode *node;
    const FChild *child;
    const FTask *tasks;
    int ntasks;
    const int32_t *relmap, *cbnd, *acolptr, *atpos, *acolj, *asrc;
    int dup;                     // some entry of A is stored more than once
    const double *val;
    const double *params;        // shift, pivot tolerance
    Real *F, *G;
    int *flags;                  // one per pivot tile of L and X
    int *upd;                    // update tiles finished, per parent
    int *queue, *status, *err;
};

// Tile storage: column-major, 64 rows, the row index XORed within its
// 16-row group by a function of the column, so that the fragment reads
// (8 rows x 4 columns, or 8 columns x 4 rows) of a warp meet no bank
// conflicts without padding and any run of columns is one contiguous copy.
template <class MT>
SPX_DEV int tix(int i, int j) {
    return j * FT + (i ^ (sizeof(MT) == 8 ? (j & 3) << 2 : (j & 3) << 3));
}
SPX_DEV int round4(int v) { return (v + 3) & ~3; }

struct FGeo {
    int c, r, nkb, nt, wc, wl;   // widths of the last pivot tile and of the last row tile
    SPX_DEV int width(int J) const {
        return J < nkb - 1 ? FT : J == nkb - 1 ? wc : J < nt - 1 ? FT : wl;
    }
    SPX_DEV int start(int J) const { return J < nkb ? J * FT : c + (J - nkb) * FT; }
    // pivot tile (I, J), J < nkb, I >= J: column blocks back to back
    SPX_DEV int64_t ltile(int I, int J) const {
        const int64_t base = (int64_t)FT * FT * ((int64_t)J * nt - (int64_t)J * (J - 1) / 2);
        return base + (int64_t)(I - J) * FT * (J == nkb - 1 ? round4(wc) : FT);
    }
    // transposed inverse tile (j, k), j <= k < nkb, after the pivot tiles
    SPX_DEV int64_t xtile(int j, int k) const {
        const int w4 = round4(wc);
        const int64_t nl = (int64_t)FT * FT * ((int64_t)(nkb - 1) * nt -
                                               (int64_t)(nkb - 1) * (nkb - 2) / 2) +
                           (int64_t)FT * w4 * (nt - nkb + 1);
        return nl + (int64_t)FT * FT * ((int64_t)j * (nkb - 1) - (int64_t)j * (j - 1) / 2) +
               (int64_t)FT * w4 * j + (int64_t)(k - j) * FT * FT;
    }
    SPX_DEV int lflag(int I, int J) const { return J * nt + I; }
    SPX_DEV int xflag(int j, int k) const { return nkb * nt + j * nkb + k; }
};
// update tile (I, J), counted from the first row tile, of a front with nb
// rows below
SPX_DEV int64_t utile(int nb, int I, int J) {
    const int nu = (nb + FT - 1) / FT;
    return (int64_t)FT * FT * ((int64_t)J * nu - (int64_t)J * (J - 1) / 2) +
           (int64_t)(I - J) * FT * (J == nu - 1 ? round4(nb - (nu - 1) * FT) : FT);
}

SPX_DEV FGeo geo_of(const FNode &nd) {
    FGeo f;
    f.c = nd.a.y;
    f.r = nd.a.z;
    f.nkb = nd.f.y;
    f.nt = nd.f.z;
    f.wc = f.c - (f.nkb - 1) * FT;
    f.wl = f.r - f.c - (f.nt - f.nkb - 1) * FT;
    return f;
}

SPX_DEV void bar_consumers() { asm volatile("bar.sync 1, %0;" ::"n"(kFConsumers) : "memory"); }
SPX_DEV void fence_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }
// Bounded wait for *p >= target; gives up (and flags *err) after some
// seconds, or soon after another wait has given up.
SPX_DEV void fwait(const int *p, int target, int *err) {
    for (int it = 0; it < 64; it++)
        if (ld_acquire(p) >= target) return;
    for (long it = 0; it < kSpinLimit; it++) {
        if (ld_acquire(p) >= target) return;
        __nanosleep(40);
        if ((it & 255) == 0 && *(volatile int *)err) return;
    }
    atomicExch(err, 1);
}

struct FShared {
    double S[FT * FT];                                  // assembled tile, T, D
    unsigned char stage[kFStages * 2 * kFChunk * FT * 8];   // ring; X and P of FK_DIAG/FK_SMALL
    double scratch[2][64];
    unsigned long long full[kFStages], empty[kFStages];
    FTask task[2];
    FNode node[2];
};

using Acc = double[4][4][2];

SPX_DEV void acc_zero(Acc &acc) {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
}

// acc += A B^T over nk4 groups of four columns (A, B tiles or chunks of
// them), fragments inside the first mi x nj of this warp's 4 x 4 only
template <class AT, class BT>
SPX_DEV void mma_cols(Acc &acc, const AT *A, const BT *B, int nk4, int m0, int n0, int mi, int nj) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if (mi <= 0 || nj <= 0) return;
    for (int q = 0; q < nk4; q++) {
        const int k = 4 * q + t;
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = (double)A[tix<AT>(m0 + 8 * i + g, k)];
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = (double)B[tix<BT>(n0 + 8 * j + g, k)];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (i < mi && j < nj) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
}

// f(m, n, value) for every accumulator element of this warp
template <class Fn>
SPX_DEV void acc_each(const Acc &acc, int m0, int n0, Fn f) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int e = 0; e < 2; e++)
#pragma unroll
            for (int i = 0; i < 4; i++) f(m0 + 8 * i + g, n0 + 8 * j + 2 * t + e, acc[i][j][e]);
}

// Up to 32 children, one a lane (update matrix U of order nb, its rows' places
// rm), that touch the tile with at most kTiny rows (update rows ia .. ia + hi)
// and kTiny columns (ja .. ja + wj) each: every lane loads its child's
// entries, and for one place (u, v) of them after the other the lanes that meet
// in an entry of the tile sum theirs, in the children's order, and add the sum.
// A vertex with many small children below it is bound by their loads' latency:
// one child at a time takes 0.7 us each, this 0.14.  Star of 5,000 vertices
// 3.65 -> 0.74 ms, 20,000 vertices at three of ten hubs each 27.3 -> 9.1, grids
// the same (their fronts have up to 25 children).
constexpr int kTiny = 4;
__device__ __noinline__ void add_tiny_children(const Real *U, const int32_t *rm, double *S, int nb, int ia,
                                               int hi, int ja, int wj, int ra, int ca) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int ri[kTiny], rj[kTiny];
    double x[kTiny][kTiny];
#pragma unroll
    for (int u = 0; u < kTiny; u++) {
        ri[u] = u < hi && wj > 0 ? rm[ia + u] - ra : -1;
        rj[u] = u < wj && hi > 0 ? rm[ja + u] - ca : -1;
        if ((rj[u] & 3) != wid) rj[u] = -1;              // another warp's column
    }
#pragma unroll
    for (int v = 0; v < kTiny; v++)
#pragma unroll
        for (int u = 0; u < kTiny; u++) {
            const int i = ia + u, j = ja + v;
            x[u][v] = 0.0;
            if (ri[u] >= 0 && rj[v] >= 0 && i >= j)
                x[u][v] = (double)__ldcg(U + utile(nb, i / FT, j / FT) + tix<Real>(i % FT, j % FT));
        }
#pragma unroll
    for (int v = 0; v < kTiny; v++)
#pragma unroll
        for (int u = 0; u < kTiny; u++) {
            const bool mine = ri[u] >= 0 && rj[v] >= 0 && ia + u >= ja + v;
            if (!__any_sync(full, mine)) continue;
            const int at = mine ? tix<double>(ri[u], rj[v]) : -1 - lane;
            const unsigned same = __match_any_sync(full, at);
            double s = 0.0;
            for (unsigned m = same; __any_sync(full, m != 0); m &= m - 1) {
                const double y = __shfl_sync(full, x[u][v], m ? __ffs(m) - 1 : lane);
                if (m) s += y;
            }
            if (mine && lane == __ffs(same) - 1) S[at] += s;
            __syncwarp();
        }
}

// S(i, j) = the assembled tile of rows [ra, ra + h) x columns [ca, ca + w)
// of the front: children's update matrices in child order, then A and the
// shift.  Each warp owns the target columns j with j % 4 = its index, so the
// children need no barrier between them and the sums have a fixed order.
SPX_DEV void assemble(const FactorArgs &a, const FNode &nd, double *S, int I, int J, int ra, int h,
                      int ca, int w, bool pivots) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int t = tid; t < FT * FT / 2; t += kFConsumers)
        reinterpret_cast<double2 *>(S)[t] = make_double2(0.0, 0.0);
    bar_consumers();
    const unsigned full = 0xffffffffu;
    for (int q0 = 0; q0 < nd.b.y; q0 += 32) {
        // the children's records and bounds, one child per lane
        const int q = q0 + lane;
        FChild ch = {};
        int ia = 0, hi = 0, ja = 0, wj = 0;
        if (q < nd.b.y) {
            ch = a.child[nd.b.z + q];
            const int32_t *bd = a.cbnd + ch.cbnd;
            ia = bd[I];
            hi = bd[I + 1] - ia;
            ja = bd[J];
            wj = bd[J + 1] - ja;
        }
        unsigned live = __ballot_sync(full, hi > 0 && wj > 0);
        if (__popc(live) >= 4 && __all_sync(full, hi <= kTiny && wj <= kTiny)) {
            add_tiny_children(a.F + ch.uptr, a.relmap + ch.relmap, S, ch.nb, ia, hi, ja, wj, ra, ca);
            continue;
        }
        while (live) {
            const int src = __ffs(live) - 1;
            live &= live - 1;
            const long long up = __shfl_sync(full, ch.uptr, src), rp = __shfl_sync(full, ch.relmap, src);
            const int nb = __shfl_sync(full, ch.nb, src);
            const int ia2 = __shfl_sync(full, ia, src), hi2 = __shfl_sync(full, hi, src);
            const int ja2 = __shfl_sync(full, ja, src), wj2 = __shfl_sync(full, wj, src);
            const int32_t *rm = a.relmap + rp;
            // the child's update rows of this tile: lane + 32 u
            int ri[2], rj[2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int x = lane + 32 * u;
                ri[u] = x < hi2 ? rm[ia2 + x] - ra : -1;
                rj[u] = x < wj2 ? rm[ja2 + x] - ca : -1;
            }
#pragma unroll
            for (int v = 0; v < 2; v++) {
                unsigned mine = __ballot_sync(full, rj[v] >= 0 && (rj[v] & 3) == wid);
                while (mine) {
                    // up to eight columns at a time, their loads in flight together
                    constexpr int U = 8;
                    int jc[U], tj[U];
                    double x0[U], x1[U];
#pragma unroll
                    for (int e = 0; e < U; e++) {
                        jc[e] = mine ? __ffs(mine) - 1 : -1;
                        mine &= mine - 1;
                        tj[e] = __shfl_sync(full, rj[v], jc[e] < 0 ? 0 : jc[e]);
                        x0[e] = x1[e] = 0.0;
                        if (jc[e] >= 0) {
                            const int j = ja2 + 32 * v + jc[e], Jc = j / FT, jl = j % FT;
#pragma unroll
                            for (int u = 0; u < 2; u++) {
                                const int i = ia2 + lane + 32 * u;
                                if (ri[u] >= 0 && i >= j) {
                                    const double z = (double)__ldcg(
                                        a.F + up + utile(nb, i / FT, Jc) + tix<Real>(i % FT, jl));
                                    if (u == 0) x0[e] = z; else x1[e] = z;
                                }
                            }
                        }
                    }
#pragma unroll
                    for (int e = 0; e < U; e++) {
                        if (jc[e] >= 0) {
                            if (ri[0] >= 0) S[tix<double>(ri[0], tj[e])] += x0[e];
                            if (ri[1] >= 0) S[tix<double>(ri[1], tj[e])] += x1[e];
                        }
                    }
                    __syncwarp();
                }
            }
            __syncwarp();
        }
    }
    if (pivots) {
        const int col0 = nd.a.x + ca;
        const int e0 = a.acolptr[col0], e1 = a.acolptr[col0 + w];
        bar_consumers();
        if (!a.dup) {
            // the columns' entries are one range: a thread an entry
            for (int e = e0 + tid; e < e1; e += kFConsumers) {
                const int i = a.atpos[e] - ra;
                if (i >= 0 && i < h) S[tix<double>(i, a.acolj[e] - col0)] += a.val[a.asrc[e]];
            }
            bar_consumers();
            if (I == J && tid < w) S[tix<double>(tid, tid)] += a.params[0];
        } else if (tid < w) {
            // repeated entries are added in their order: a thread a column
            for (int e = a.acolptr[col0 + tid]; e < a.acolptr[col0 + tid + 1]; e++) {
                const int i = a.atpos[e] - ra;
                if (i >= 0 && i < h) S[tix<double>(i, tid)] += a.val[a.asrc[e]];
            }
            if (I == J) S[tix<double>(tid, tid)] += a.params[0];
        }
    }
    bar_consumers();
}

// Places of an 8 x 8 block's elements in a tile of the S layout, as a lane's
// constants plus one XOR and one add a block (the blocks start at multiples of
// 8, so the layout's XOR splits into its bit 3 and the bits below):
//   nn: element (row0 + lane / 4, col0 + 4 ks + lane % 4), ks = 0, 1
//   tn: element (row0 + 4 ks + lane % 4, col0 + lane / 4)
//   cc: element (row0 + lane / 4, col0 + 2 (lane % 4) + e), e = 0, 1
struct Blk8 {
    int a0, ax, b0[2], bx, c0[2], cx[2];
    SPX_DEV Blk8() {
        const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
        a0 = t * FT + (g ^ ((t << 2) & 4));
        ax = (t << 2) & 8;
        const int c = (g & 3) << 2;
        bx = c & 8;
#pragma unroll
        for (int ks = 0; ks < 2; ks++) b0[ks] = g * FT + ((4 * ks) ^ (c & 4)) + t;
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int q = ((2 * t + e) & 3) << 2;
            c0[e] = (2 * t + e) * FT + (g ^ (q & 4));
            cx[e] = q & 8;
        }
    }
    SPX_DEV int nn(int row0, int col0, int ks) const { return a0 + (row0 ^ ax) + (col0 + 4 * ks) * FT; }
    SPX_DEV int tn(int row0, int col0, int ks) const { return b0[ks] + (row0 ^ bx) + col0 * FT; }
    SPX_DEV int cc(int row0, int col0, int e) const { return c0[e] + (row0 ^ cx[e]) + col0 * FT; }
};

// Cholesky factor and inverse of one 8 x 8 block, by a whole warp: every lane
// factors the block in its own registers (no exchanges on the chain of
// pivots) and carries column lane % 8 of the identity along, which leaves
// that column of the inverse; lanes 0..7 write X_pp.  A pivot <= pivtol
// records its column and is replaced by 1.
SPX_DEV void chol8(const double *D, double *X, int o, double pivtol, int *status,
                                   int colbase, int w) {
    const int lane = threadIdx.x & 31, c = lane & 7;
    double l[8][8], x[8];
    // the block's columns with bit 3 of the layout's XOR clear and set
    const double *p0 = D + o * FT + o, *p8 = D + o * FT + (o ^ 8);
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
        for (int i = j; i < 8; i++) l[i][j] = ((j & 2) ? p8 : p0)[j * FT + (i ^ ((j & 1) << 2))];
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = (i == c) ? 1.0 : 0.0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        double d = l[j][j];
        if (!(d > pivtol)) {
            if (lane == 0 && o + j < w) atomicCAS(status, 0, colbase + o + j + 1);
            d = 1.0;
        }
        const double r = rsqrt(d);
#pragma unroll
        for (int i = j + 1; i < 8; i++) l[i][j] *= r;
#pragma unroll
        for (int k = j + 1; k < 8; k++)
#pragma unroll
            for (int i = k; i < 8; i++) l[i][k] -= l[i][j] * l[k][j];
        x[j] *= r;
#pragma unroll
        for (int i = j + 1; i < 8; i++) x[i] -= l[i][j] * x[j];
    }
    if (lane < 8) {
        double *q = X + (o + c) * FT + (o ^ ((c & 2) << 2));
#pragma unroll
        for (int i = 0; i < 8; i++) q[i ^ ((c & 1) << 2)] = x[i];
    }
    __syncwarp();
}

// Cholesky factor and inverse of the w x w tile D (lower triangle read; rows
// and columns from w to the next multiple of 8 hold the identity), by the
// four consumer warps.  X receives inv(L) (its lower 8 x 8 blocks); L's
// off-diagonal blocks L_ip are left transposed in place: block (i, p) of L at
// block (p, i) of D.  Per 8 pivots: warp 0 runs the chain (block p+1's row,
// update, factor), warps 1-3 the rest of the panel, the trailing update and
// row p of the inverse beside it, each in groups of independent blocks: the
// blocks' latencies, not their products, are what they cost.  21,300 cycles for
// a full tile (26,000 with one block at a time); the chain alone, a factored
// 8 x 8 block every 1,970 cycles, is 15,800 of them.
SPX_DEV void chol_inv64(double *D, double *X, double *scr, int w, double pivtol, int *status,
                        int colbase) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3, nb = (w + 7) >> 3;
    const Blk8 at;
#pragma unroll 1
    for (int p = -1; p < nb; p++) {                      // p = -1: the first block alone
        double xp[2] = {0.0, 0.0};
        if (p >= 0)
#pragma unroll
            for (int ks = 0; ks < 2; ks++) xp[ks] = X[at.nn(8 * p, 8 * p, ks)];
        if (wid == 0 && p + 1 < nb) {
            const int i = p + 1;
            if (p >= 0) {
                const int c0 = at.cc(8 * i, 8 * i, 0), c1 = at.cc(8 * i, 8 * i, 1);
                const double e0 = D[c0], e1 = D[c1];
                double d0 = 0.0, d1 = 0.0;                   // L_ip = A_ip X_pp^T
#pragma unroll
                for (int ks = 0; ks < 2; ks++) dmma(d0, d1, D[at.nn(8 * i, 8 * p, ks)], xp[ks]);
                scr[(2 * t) * 8 + g] = d0;                   // L_ip(g, k) at scr[8 k + g]
                scr[(2 * t + 1) * 8 + g] = d1;
                __syncwarp();
                double u0 = 0.0, u1 = 0.0;
#pragma unroll
                for (int ks = 0; ks < 2; ks++) {
                    const double f = scr[(4 * ks + t) * 8 + g];
                    dmma(u0, u1, f, f);
                }
                D[c0] = e0 - u0;
                D[c1] = e1 - u1;
                __syncwarp();
            }
            chol8(D, X, 8 * i, pivtol, status, colbase, w);
        }
        if (wid > 0 && p >= 0 && p + 1 < nb) {
            // the panel: rows i = p + wid + 3 q, L_ip transposed into block (p, i)
            double d[3][2];
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const int i = p + wid + 3 * q;
                d[q][0] = d[q][1] = 0.0;
                if (i < nb)
#pragma unroll
                    for (int ks = 0; ks < 2; ks++) dmma(d[q][0], d[q][1], D[at.nn(8 * i, 8 * p, ks)], xp[ks]);
            }
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const int i = p + wid + 3 * q;
                if (i < nb) {
                    D[tix<double>(8 * p + 2 * t, 8 * i + g)] = d[q][0];
                    D[tix<double>(8 * p + 2 * t + 1, 8 * i + g)] = d[q][1];
                }
            }
            asm volatile("bar.sync 2, 96;" ::: "memory");
            // trailing blocks (i, j), p < j <= i, without (p+1, p+1): block
            // rows from the bottom, dealt to the warps, all blocks of a row
            // together
            for (int i = nb - wid; i > p + 1; i -= 3) {
                double a[2];
#pragma unroll
                for (int ks = 0; ks < 2; ks++) a[ks] = D[at.tn(8 * p, 8 * i, ks)];
#pragma unroll 1
                for (int j0 = p + 1; j0 <= i; j0 += 4) {
                    double u[4][2];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        u[q][0] = u[q][1] = 0.0;
                        if (j0 + q > i) break;
#pragma unroll
                        for (int ks = 0; ks < 2; ks++)
                            dmma(u[q][0], u[q][1], a[ks], D[at.tn(8 * p, 8 * (j0 + q), ks)]);
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (j0 + q > i) break;
#pragma unroll
                        for (int z = 0; z < 2; z++) D[at.cc(8 * i, 8 * (j0 + q), z)] -= u[q][z];
                    }
                }
            }
        }
        // row p of the inverse, a few blocks j a warp: X_pj = -X_pp sum_{j <= k < p}
        // L_pk X_kj, with L_pk(m, s) at D(8k + s, 8p + m); warp 0 joins in
        // once its chain is through
        const bool all = p + 1 == nb;
        const int nw = all ? 4 : 3, me = all ? wid : wid - 1;
        if (me >= 0 && p > 0) {
            double y[3][2];
#pragma unroll
            for (int q = 0; q < 3; q++) y[q][0] = y[q][1] = 0.0;
            for (int k = 0; k < p; k++) {
                double a[2];
#pragma unroll
                for (int ks = 0; ks < 2; ks++) a[ks] = D[at.tn(8 * k, 8 * p, ks)];
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    if (me + nw * q > k) break;
#pragma unroll
                    for (int ks = 0; ks < 2; ks++)
                        dmma(y[q][0], y[q][1], a[ks], X[at.tn(8 * k, 8 * (me + nw * q), ks)]);
                }
            }
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const int j = me + nw * q;
                if (j >= p) break;
                double r0 = 0.0, r1 = 0.0;
#pragma unroll
                for (int ks = 0; ks < 2; ks++) {
                    // accumulator (row g, columns 2t, 2t+1) to the B fragment
                    // (row t + 4 ks, column g)
                    const int src = (t + 4 * ks) * 4 + (g >> 1);
                    const double b0 = __shfl_sync(0xffffffffu, y[q][0], src);
                    const double b1 = __shfl_sync(0xffffffffu, y[q][1], src);
                    dmma(r0, r1, xp[ks], (g & 1) ? b1 : b0);
                }
                X[at.cc(8 * p, 8 * j, 0)] = -r0;
                X[at.cc(8 * p, 8 * j, 1)] = -r1;
            }
        }
        bar_consumers();
    }
}

// ---- producer: chunks of the task's operand tiles into the ring --------
struct FPipe {
    unsigned it = 0;                 // chunks since the kernel's start
};

SPX_DEV void produce_chunks(const FactorArgs &a, FShared &sh, FPipe &pp, const Real *A,
                            const Real *B, int w) {
    const int w4 = round4(w);
    Real *ring = reinterpret_cast<Real *>(sh.stage);
    for (int c0 = 0; c0 < w4; c0 += kFChunk, pp.it++) {
        const int st = pp.it % kFStages;
        mbar_wait(&sh.empty[st], ((pp.it / kFStages) & 1u) ^ 1u, a.err);
        const uint32_t bytes = (uint32_t)(min(kFChunk, w4 - c0) * FT * sizeof(Real));
        Real *dst = ring + (size_t)st * 2 * kFChunk * FT;
        mbar_expect(&sh.full[st], bytes * ((A != nullptr) + (B != nullptr)));
        if (A) bulk_load(dst, A + (size_t)c0 * FT, bytes, &sh.full[st]);
        if (B) bulk_load(dst + kFChunk * FT, B + (size_t)c0 * FT, bytes, &sh.full[st]);
    }
}

SPX_DEV void fproduce(const FactorArgs &a, FShared &sh, FPipe &pp, const FTask &tk,
                      const FNode &nd) {
    const FGeo f = geo_of(nd);
    const Real *Fp = a.F + nd.p.x;
    const int *fl = a.flags + nd.f.x;
    const int I = tk.I, J = tk.J;
    auto need = [&](int id) { fwait(fl + id, 1, a.err); };
    switch (tk.kind) {
        case FK_DIAG:
        case FK_ROWS:
        case FK_SCHUR: {
            const int k1 = min(J, f.nkb);
            for (int k = 0; k < k1; k++) {
                need(f.lflag(I, k));
                if (I != J) need(f.lflag(J, k));
                fence_async_all();
                produce_chunks(a, sh, pp, Fp + f.ltile(I, k), I == J ? nullptr : Fp + f.ltile(J, k),
                               f.width(k));
            }
            if (tk.kind == FK_ROWS) {
                need(f.lflag(J, J));
                fence_async_all();
                produce_chunks(a, sh, pp, nullptr, Fp + f.ltile(J, J), f.width(J));
            }
            break;
        }
        case FK_INV:
        case FK_WMUL: {
            const int k1 = tk.kind == FK_INV ? I : f.nkb;
            for (int k = J; k < k1; k++) {
                need(f.lflag(I, k));
                need(f.xflag(J, k));
                fence_async_all();
                produce_chunks(a, sh, pp, Fp + f.ltile(I, k), Fp + f.xtile(J, k), f.width(k));
            }
            if (tk.kind == FK_INV) {
                need(f.lflag(I, I));
                fence_async_all();
                produce_chunks(a, sh, pp, Fp + f.ltile(I, I), nullptr, f.width(I));
            }
            break;
        }
        default: break;
    }
}

// ---- consumers ----------------------------------------------------------
// acc += the products of `chunks` column blocks of width w; SA / SB: the
// operand is the tile S (shared, FP64) instead of the ring's
template <bool SA, bool SB>
SPX_DEV void consume_block(FShared &sh, FPipe &pp, Acc &acc, bool same, int w, int m0, int n0,
                           int mi, int nj, int *err) {
    const int w4 = round4(w);
    const Real *ring = reinterpret_cast<const Real *>(sh.stage);
    for (int c0 = 0; c0 < w4; c0 += kFChunk, pp.it++) {
        const int st = pp.it % kFStages;
        mbar_wait(&sh.full[st], (pp.it / kFStages) & 1u, err);
        const Real *A = ring + (size_t)st * 2 * kFChunk * FT;
        const Real *B = same ? A : A + kFChunk * FT;
        const int nk4 = min(kFChunk, w4 - c0) >> 2;
        if constexpr (SA) mma_cols(acc, sh.S + c0 * FT, B, nk4, m0, n0, mi, nj);
        else if constexpr (SB) mma_cols(acc, A, sh.S + c0 * FT, nk4, m0, n0, mi, nj);
        else mma_cols(acc, A, B, nk4, m0, n0, mi, nj);
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(&sh.empty[st]);
    }
}

// publish: every consumer's global writes, then one release increment
SPX_DEV void publish(int *p) {
    fence_async_all();               // the tile is read by bulk copies elsewhere
    bar_consumers();
    if (threadIdx.x == 0) add_release(p, 1);
}

// S = identity-padded lower tile for chol_inv64
SPX_DEV void store_diag(FShared &sh, const Acc &acc, int w, int m0, int n0) {
    acc_each(acc, m0, n0, [&](int m, int n, double v) {
        double &d = sh.S[tix<double>(m, n)];
        d = (m < w && n < w) ? d - v : (m == n ? 1.0 : 0.0);
    });
}

// X_JJ (w x w lower, zero elsewhere) to tile storage; first of all, because
// the chain waits for it (pairs of entries: the layouts of X and of an FP64
// tile are the same)
SPX_DEV void write_inverse_tile(const double *X, int w, Real *L) {
    for (int t = threadIdx.x; t < FT / 2 * round4(w); t += kFConsumers) {
        const int j = t >> 5;
        if constexpr (sizeof(Real) == 8) {
            const int i = (2 * (t & 31)) ^ ((j & 3) << 2);       // even, as the XOR is
            double2 v = reinterpret_cast<const double2 *>(X)[t];
            if (!(i >= j && i < w && j < w)) v.x = 0.0;
            if (!(i + 1 >= j && i + 1 < w && j < w)) v.y = 0.0;
            reinterpret_cast<double2 *>(L)[t] = v;
        } else {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int i = 2 * (t & 31) + e;
                L[tix<Real>(i, j)] = (Real)((i >= j && i < w && j < w) ? X[tix<double>(i, j)] : 0.0);
            }
        }
    }
}
// and to the panel, and transposed to the inverse's tile storage (if any)
SPX_DEV void write_inverse(const double *X, int w, Real *G, int at, int c, Real *Xt) {
    const int w4 = round4(w);
    for (int t = threadIdx.x; t < FT * w4; t += kFConsumers) {
        const int i = t & (FT - 1), j = t >> 6;
        if (j < w && i < w && i >= j) G[gix(at + i, at + j, c)] = (Real)X[tix<double>(i, j)];
        if (Xt) Xt[tix<Real>(i, j)] = (Real)((i < w && j < w && j >= i) ? X[tix<double>(j, i)] : 0.0);
    }
}

SPX_DEV void fconsume(const FactorArgs &a, FShared &sh, FPipe &pp, const FTask &tk,
                      const FNode &nd) {
    const FGeo f = geo_of(nd);
    const int tid = threadIdx.x, wid = tid >> 5;
    const int m0 = (wid & 1) * 32, n0 = (wid >> 1) * 32;
    Real *Fp = a.F + nd.p.x, *Gp = a.G + nd.g.x;
    int *fl = a.flags + nd.f.x;
    const int I = tk.I, J = tk.J;
    double *X = reinterpret_cast<double *>(sh.stage);
    Acc acc;
    acc_zero(acc);
    if (tk.kind == FK_INV || tk.kind == FK_WMUL) {
        const int h = f.width(I), w = f.width(J);
        const int mi = min(4, (h - m0 + 7) >> 3), nj = min(4, (w - n0 + 7) >> 3);
        const int k1 = tk.kind == FK_INV ? I : f.nkb;
        for (int k = J; k < k1; k++)
            consume_block<false, false>(sh, pp, acc, false, f.width(k), m0, n0, mi, nj, a.err);
        if (tk.kind == FK_WMUL) {
            const int ra = f.start(I), ca = f.start(J);
            acc_each(acc, m0, n0, [&](int m, int n, double v) {
                if (m < h && n < w) Gp[gix(ra + m, ca + n, f.c)] = (Real)v;
            });
            return;
        }
        // S(n, k) = the sum transposed (zero past the rows of L_ik), then
        // X_ij = -X_ii S^T
        acc_each(acc, m0, n0, [&](int m, int n, double v) {
            sh.S[tix<double>(n, m)] = m < h ? v : 0.0;
        });
        bar_consumers();
        acc_zero(acc);
        consume_block<false, true>(sh, pp, acc, false, h, m0, n0, mi, nj, a.err);
        Real *Xt = Fp + f.xtile(J, I);
        const int ra = f.start(I), ca = f.start(J), h4 = round4(h);
        acc_each(acc, m0, n0, [&](int m, int n, double v) {
            if (m < h4) Xt[tix<Real>(n, m)] = (Real)(m < h ? -v : 0.0);
            if (m < h && n < w) Gp[gix(ra + m, ca + n, f.c)] = (Real)-v;
        });
        publish(fl + f.xflag(J, I));
        return;
    }
    // tiles of the front proper start with their assembly
    if (nd.b.y > 0 && tid == 0) fwait(a.upd + tk.s, nd.b.w, a.err);
    if (nd.b.y > 0) bar_consumers();
    const bool small = tk.kind == FK_SMALL;
    const int ra = f.start(I), ca = f.start(J), h = f.width(I), w = f.width(J);
    const int mi = min(4, (h - m0 + 7) >> 3), nj = min(4, (w - n0 + 7) >> 3);
    assemble(a, nd, sh.S, I, J, ra, h, ca, w, J < f.nkb);
    const int k1 = small ? 0 : min(J, f.nkb);
    for (int k = 0; k < k1; k++)
        consume_block<false, false>(sh, pp, acc, I == J, f.width(k), m0, n0, mi, nj, a.err);
    if (tk.kind == FK_SCHUR) {
        Real *U = a.F + nd.p.y + utile(f.r - f.c, I - f.nkb, J - f.nkb);
        const bool diag = I == J;
        acc_each(acc, m0, n0, [&](int m, int n, double v) {
            if (m < h && n < w && (!diag || n <= m))
                U[tix<Real>(m, n)] = (Real)(sh.S[tix<double>(m, n)] - v);
        });
        if (nd.b.x >= 0) publish(a.upd + nd.b.x);
        return;
    }
    if (tk.kind == FK_ROWS) {
        const int w4 = round4(w);
        acc_each(acc, m0, n0, [&](int m, int n, double v) {
            double &d = sh.S[tix<double>(m, n)];
            d = n < w ? d - v : 0.0;
        });
        bar_consumers();
        acc_zero(acc);
        consume_block<true, false>(sh, pp, acc, false, w, m0, n0, mi, nj, a.err);
        Real *L = Fp + f.ltile(I, J);
        acc_each(acc, m0, n0, [&](int m, int n, double v) {
            if (n < w4) L[tix<Real>(m, n)] = (Real)(n < w ? v : 0.0);
        });
        publish(fl + f.lflag(I, J));
        return;
    }
    // FK_DIAG, FK_SMALL: the ring is drained (the task has no further chunks)
    // and holds X and, for FK_SMALL, the rows below
    double *P = X + FT * FT;
    const int nb = f.r - f.c, w4 = round4(w);
    store_diag(sh, acc, w, m0, n0);
    if (small && nb > 0) assemble(a, nd, P, 1, 0, w, nb, 0, w, true);
    else bar_consumers();
    chol_inv64(sh.S, X, sh.scratch[0], w, a.params[1], a.status, nd.a.x + ca);
    if (!small) {
        write_inverse_tile(X, w, Fp + f.ltile(J, J));
        publish(fl + f.lflag(J, J));
        write_inverse(X, w, Gp, ca, f.c, Fp + f.xtile(J, J));
        publish(fl + f.xflag(J, J)); // (also orders the ring's reuse by bulk copies)
        return;
    }
    // zero above the diagonal blocks, for the products
    for (int t = tid; t < FT * w4; t += kFConsumers) {
        const int i = t & (FT - 1), j = t >> 6;
        if (i < j || i >= w || j >= w) X[tix<double>(i, j)] = 0.0;
    }
    bar_consumers();
    write_inverse(X, w, Gp, 0, f.c, nullptr);
    if (nb > 0) {
        const int mb = min(4, (nb - m0 + 7) >> 3), nb2 = min(4, (nb - n0 + 7) >> 3);
        acc_zero(acc);
        mma_cols(acc, P, X, w4 >> 2, m0, n0, mb, nj);              // L21 = P X^T
        bar_consumers();
        acc_each(acc, m0, n0, [&](int m, int n, double v) {
            // FP32 storage rounds L21 as a stored tile would be
            if (n < w4) P[tix<double>(m, n)] = n < w ? (double)(Real)v : 0.0;
        });
        // S(n, k) = X(k, n): the second operand of W = L21 X
        for (int t = tid; t < FT * w4; t += kFConsumers) {
            const int n = t & (FT - 1), k = t >> 6;
            sh.S[tix<double>(n, k)] = (n < w && k < w && k >= n) ? (double)(Real)X[tix<double>(k, n)] : 0.0;
        }
        bar_consumers();
        acc_zero(acc);
        mma_cols(acc, P, sh.S, w4 >> 2, m0, n0, mb, nj);
        acc_each(acc, m0, n0, [&](int m, int n, double v) {
            if (m < nb && n < w) Gp[gix(w + m, n, f.c)] = (Real)v;
        });
        bar_consumers();
        assemble(a, nd, sh.S, 1, 1, w, nb, w, nb, false);
        acc_zero(acc);
        mma_cols(acc, P, P, w4 >> 2, m0, n0, mb, nb2);
        Real *U = a.F + nd.p.y;
        acc_each(acc, m0, n0, [&](int m, int n, double v) {
            if (m < nb && n <= m) U[tix<Real>(m, n)] = (Real)(sh.S[tix<double>(m, n)] - v);
        });
        if (nd.b.x >= 0) publish(a.upd + nd.b.x);
    }
    fence_async_all();               // the ring's memory goes back to the bulk copies
}

// After a pivot failure the remaining tasks do no work but still publish, so
// nothing waits for them.
SPX_DEV void fskip(const FactorArgs &a, const FTask &tk, const FNode &nd) {
    if (threadIdx.x != 0) return;
    const FGeo f = geo_of(nd);
    int *fl = a.flags + nd.f.x;
    switch (tk.kind) {
        case FK_DIAG: add_release(fl + f.xflag(tk.J, tk.J), 1);
        case FK_ROWS: add_release(fl + f.lflag(tk.I, tk.J), 1); break;
        case FK_INV: add_release(fl + f.xflag(tk.J, tk.I), 1); break;
        case FK_SMALL: if (f.r == f.c) break;   // no update matrix
        case FK_SCHUR: if (nd.b.x >= 0) add_release(a.upd + nd.b.x, 1); break;
        default: break;
    }
}

// (168 registers a thread: ten warps an SM put three on some sub-partitions)
__global__ void __launch_bounds__(kFThreads, 2) mf_factor(FactorArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    FShared &sh = *reinterpret_cast<FShared *>(smem_raw);
    const int tid = threadIdx.x;
    const bool producer = tid == kFConsumers;
    FPipe pp;
    auto fetch = [&](int slot) {
        const int t = atomicAdd(a.queue, 1);
        FTask tk = {-1, 0, 0, 0};
        if (t < a.ntasks && !*(volatile int *)a.err) {
            tk = a.tasks[t];
            sh.node[slot] = a.node[tk.s];
            if (*(volatile int *)a.status) tk.kind |= 16;     // skip
        }
        sh.task[slot] = tk;
    };
    if (tid == 0) {
        for (int q = 0; q < kFStages; q++) {
            mbar_init_n(&sh.full[q], 1);
            mbar_init_n(&sh.empty[q], kFConsumers / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (producer) fetch(0);
    __syncthreads();
    for (int it = 0;; it++) {
        const FTask tk = sh.task[it & 1];
        if (tk.kind < 0) break;
        if (producer) {
            if (!(tk.kind & 16)) fproduce(a, sh, pp, tk, sh.node[it & 1]);
            fetch((it + 1) & 1);
        } else if (tid < kFConsumers) {
            if (tk.kind & 16) {
                FTask t2 = tk;
                t2.kind &= 15;
                fskip(a, t2, sh.node[it & 1]);
            } else {
                fconsume(a, sh, pp, tk, sh.node[it & 1]);
            }
        }
        __syncwarp();
        __syncthreads();
    }
}
