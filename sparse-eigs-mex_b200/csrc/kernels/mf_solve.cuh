// The shift-invert solve: X = (A + shift I)^{-1} B for one right-hand side
// (NR = 1) or NR = 8, 16, 24 or 32 of them, one persistent launch (included
// by multifrontal.cu inside its anonymous namespace, once per storage type).
//
// Tasks are tiles of the panels G, from an atomic queue in a topological
// order: forward tasks (leaves to root), then backward tasks (root to
// leaves).  A task waits for the values it reads, one by one: every vector
// entry that passes between tasks is written once per solve, and until then
// holds kUnset, a NaN that no task writes.  So there are no flags, fences or
// counters between tasks: a value's arrival is the signal, and a level of the
// tree costs one store and one load.  The entries exist twice, and a solve
// that uses one copy resets the other for the solve after it.  Waits are
// bounded; they cannot deadlock, since a task waits only for tasks before it
// in the queue, which running blocks hold and finish in order.
//
//   forward, supernode s:  f = b(pivots) + the children's update vectors
//     (host-built gather list per front row, children in a fixed order);
//     [x1; r2] = G f;  yf(pivots) = x1;  u_s = f(rows below) - r2
//   backward:  x1 = G^T [yf(pivots); -x(rows below)]
//
// Panel layout: blocks of 16 rows, each all c columns of 16 rows (the row
// XORed by a function of the column, which keeps the tensor-core fragment
// reads free of bank conflicts).  A forward tile is then one contiguous piece
// per row block and a backward tile a few columns of every row block, both
// long enough for bulk copies.
//
// What bounds it: the tasks' latency and, with one right-hand side, the
// instructions around their few products, not bytes.  A task is a chain of a
// dozen short waits (queue, gather, barriers), so throughput is the number of
// tiles in flight: small blocks (one right-hand side: four warps, eight blocks
// to an SM with a 16 KB tile each), and the next task's record fetched and its
// tile and lists copied while the current one finishes.  A block takes the
// next task's number only when the current one's probe is there: a block that
// waits for its inputs then holds no other task back (taken at the start of
// the task, 33x35x37 0.134 ms instead of 0.094, 46^3 0.186 instead of 0.162).
// The tiles of the single solve are a few rows times all columns (forward) or
// a few columns times all rows (backward), so that most supernodes need no sum
// across blocks.  A row (column) chunk wider (taller) than a tile is cut into
// strips whose partial products the task of the last strip waits for and adds
// in a fixed order, so results are the same every run.  With several
// right-hand sides the gathers cost more than the panel, so forward tiles are
// 64 x 64 and backward ones a few columns of 256 rows.
//
// Measured against the solve of before (flags and last-arrival counters,
// 64 x 128 tiles, two blocks an SM) on the same supernodes: one right-hand
// side 20^3 0.089 -> 0.049 ms, 33x35x37 0.188 -> 0.082, 46^3 0.347 -> 0.148,
// 64^3 1.03 -> 0.467 (1.66 GB of panels, 3.6 TB/s); eight at 48^3 0.442 ->
// 0.290, 24 at 48^3 0.80 -> 0.67.
constexpr int kVecThreads = 128, kBlkThreads = 256;
constexpr int kVecElems = 2048;      // panel entries of a tile, NR = 1
constexpr int kVecRows = 128;        // rows of a forward tile, NR = 1
constexpr int kVecStrip = 128;       // columns of a forward strip, NR = 1
constexpr int kVecTall = 32;         // row blocks of a backward strip, NR = 1
constexpr int kBlkElems = 4096;      // panel entries of a tile, NR >= 8
constexpr int kBlkRows = 64;         // rows of a forward tile, NR >= 8
constexpr int kBlkStrip = 64;        // columns of a forward strip, NR >= 8
constexpr int kBlkTall = 16;         // row blocks of a backward strip, NR >= 8
constexpr int kBwdCols = 64;         // columns of a backward tile at most
constexpr int kListInts = 384;       // gather entries staged per task
constexpr int kLongList = 16;        // longer gather lists are summed by many threads (grids have
                                     // lists of up to 6, geometric graphs of up to 10)

enum { SK_FWD = 0, SK_BWD = 1 };

struct STask {                       // 128 bytes: all a tile needs
    int kind, first, c, r;           // first: first pivot column of the supernode
    int probe_at, probe, pad2;       // a value that arrives late among those this task reads:
                                     // 0 none, 1 u, 2 x, 3 yf, and its index
    int i0, nrow, nrb;               // rows [i0, i0 + nrow) in nrb 16-row blocks
    int j0, jn;                      // columns [j0, j0 + jn)
    int strip, nstrip, slot0, pad3;  // strip of its chunk, strips, first partial slot
    int pl0, pln, rl0, rln;          // gather entries of the pivots j0.. and of the rows
    int has_child, pad0;             // has_child: 2 where the supernode has long gather lists
    long long g;                     // panel offset of (i0, j0)
    long long rows;                  // row-list offset of the supernode
    long long u;                     // update-vector offset (row c's entry)
    int pad[4];
};
static_assert(sizeof(STask) == 128, "task layout");

// What an entry holds until it is written (a result with this very bit
// pattern is written as another NaN).
constexpr long long kUnset = 0x7ffcb200b200b200LL;

struct SolveArgs {
    const STask *tasks;
    int ntasks;
    const int32_t *perm, *rows, *cptr, *cidx;
    const Real *G;
    double *val;                     // two copies of `stride` values: u, yf, x (rows of NR,
    int64_t stride;                  // factor order) and the strips' partial sums
    int64_t o_yf, o_x, o_fp, o_bp;   // their offsets (u: 0)
    int *sync;                       // queue, blocks gone, copy in use
    int *err;
    const double *bc;                // right-hand sides, column-major, original order
    double *xc;                      // results; a tree's writes follow its whole forward
                                     // pass, so xc may be bc (other overlaps may not)
    int64_t ldb, ldx;
    int nr;                          // columns given (the rest read as zero)
    int accumulate;                  // xc += the solution (else xc = it)
    const int *skip;                 // when set and nonzero: nothing to do
};

template <int NR>
struct SShared {
    static constexpr int kThreads = NR == 1 ? kVecThreads : kBlkThreads;
    static constexpr int kElems = NR == 1 ? kVecElems : kBlkElems;
    // staged ints of a task: see lists_of
    static constexpr int kLists = NR == 1 ? 3 * (kVecStrip + 8) + kListInts + 40
                                          : 2 * (kBlkStrip + 8) + kBlkRows + 8 + kListInts + 40;
    // row stride of the block form's vector segment: fragment reads of 4 rows
    // x 8 columns fall in distinct banks
    static constexpr int SEG = NR + 4;
    Real panel[kElems];
    int lists[kLists];
    double vec[NR == 1 ? kVecTall * 16 : kBlkTall * 16 * SEG];
    double part[2 * kVecThreads];        // NR = 1
    STask task[2];
    unsigned long long lfull, pfull;     // lists, panel in place
};
static_assert(kVecTall * 16 + 8 + kBwdCols + 8 <= SShared<1>::kLists, "backward lists");
static_assert(kBlkTall * 16 + 8 + kBwdCols + 8 <= SShared<8>::kLists, "backward lists");
// the block form's backward product leaves 8 warps x 8 columns x NR partial
// sums in vec
static_assert(8 * 8 * 32 <= kBlkTall * 16 * SShared<32>::SEG, "partial sums");

// offsets of the staged lists (ints); every list is copied from the 16-byte
// boundary at or before its first entry
SPX_DEV int lead(long long at) { return (int)(at & 3); }
struct SLists { const int *perm, *cp, *ci, *rp, *ri, *rows; };
template <int NR>
SPX_DEV SLists lists_of(const STask &k, const int *base) {
    SLists l;
    l.perm = base + lead(k.first + k.j0);
    if (k.kind == SK_FWD) {
        constexpr int C = (NR == 1 ? kVecStrip : kBlkStrip) + 8, R = (NR == 1 ? kVecRows : kBlkRows) + 8;
        l.cp = base + C + lead(k.rows + k.j0);
        l.rp = base + 2 * C + lead(k.rows + k.i0);
        l.ci = base + 2 * C + R + lead(k.pl0);
        l.ri = base + 2 * C + R + ((lead(k.pl0) + k.pln + 3) & ~3) + lead(k.rl0);
        l.rows = nullptr;
    } else {
        l.rows = base + (kBwdCols + 8) + lead(k.rows + k.i0);
        l.cp = l.ci = l.rp = l.ri = nullptr;
    }
    return l;
}
SPX_DEV uint32_t list_bytes(long long at, int n) { return (uint32_t)((lead(at) + n + 3) & ~3) * 4; }

// One warp copies a task's lists and tile into place.
template <int NR>
SPX_DEV void solve_stage(const SolveArgs &a, const STask &k, SShared<NR> &sh) {
    const int lane = threadIdx.x & 31;
    if (k.kind < 0) return;
    const bool fwd = k.kind == SK_FWD, staged = k.pln + k.rln <= kListInts;
    if (lane == 0) {
        uint32_t bytes = list_bytes(k.first + k.j0, k.jn);
        if (!fwd) bytes += list_bytes(k.rows + k.i0, k.nrow);
        else if (k.has_child) {
            bytes += list_bytes(k.rows + k.j0, k.jn + 1) + list_bytes(k.rows + k.i0, k.nrow + 1);
            if (staged) bytes += (k.pln ? list_bytes(k.pl0, k.pln) : 0) + (k.rln ? list_bytes(k.rl0, k.rln) : 0);
        }
        mbar_expect(&sh.lfull, bytes);
        mbar_expect(&sh.pfull, (uint32_t)(k.nrb * k.jn * 16 * sizeof(Real)));
    }
    __syncwarp();
    const SLists l = lists_of<NR>(k, sh.lists);
    auto copy = [&](const int *dst, const int32_t *src, long long at, int n) {
        bulk_load(const_cast<int *>(dst) - lead(at), src + (at - lead(at)), list_bytes(at, n), &sh.lfull);
    };
    if (lane == 0) copy(l.perm, a.perm, k.first + k.j0, k.jn);
    if (fwd && k.has_child) {
        if (lane == 1) copy(l.cp, a.cptr, k.rows + k.j0, k.jn + 1);
        if (lane == 2) copy(l.rp, a.cptr, k.rows + k.i0, k.nrow + 1);
        if (staged && lane == 3 && k.pln) copy(l.ci, a.cidx, k.pl0, k.pln);
        if (staged && lane == 4 && k.rln) copy(l.ri, a.cidx, k.rl0, k.rln);
    } else if (!fwd && lane == 1) {
        copy(l.rows, a.rows, k.rows + k.i0, k.nrow);
    }
    // row block b of the tile: jn columns of 16 entries
    for (int b = lane; b < k.nrb; b += 32)
        bulk_load(sh.panel + (size_t)b * k.jn * 16, a.G + k.g + (int64_t)b * k.c * 16,
                  (uint32_t)(k.jn * 16 * sizeof(Real)), &sh.pfull);
}

// The next task, fetched in three steps by the block's last warp while the
// block works on the current one: its number, its record, its tile and lists.
template <int NR>
struct SNext {
    static constexpr int kThreads = SShared<NR>::kThreads;
    int number, word;
    SPX_DEV bool mine() const { return threadIdx.x >= kThreads - 32; }
    SPX_DEV void take(const SolveArgs &a) {
        if (threadIdx.x == kThreads - 32) number = atomicAdd(a.sync, 1);
    }
    SPX_DEV void read(const SolveArgs &a) {
        if (!mine()) return;
        const int t = __shfl_sync(0xffffffffu, number, 0);
        word = t < a.ntasks ? __ldg(reinterpret_cast<const int *>(a.tasks + t) + (threadIdx.x & 31)) : -1;
    }
    SPX_DEV void stage(const SolveArgs &a, STask &slot, SShared<NR> &sh) {
        if (!mine()) return;
        reinterpret_cast<int *>(&slot)[threadIdx.x & 31] = word;
        __syncwarp();
        solve_stage<NR>(a, slot, sh);
    }
};

// The entries of the copy in use (cur) and of the other one.
struct SVals {
    double *cur;
    int64_t other;                   // the other copy, relative to cur
};
SPX_DEV bool unset(double v) { return __double_as_longlong(v) == kUnset; }
SPX_DEV double ld_val(const double *p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
SPX_DEV double2 ld_val2(const double *p) {
    double2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}
// the value at p once it is there (v: what a first load gave)
__device__ __noinline__ double await_val(const double *p, int *err) {
    double v = ld_val(p);
    for (long it = 0; unset(v) && it < kSpinLimit; it++) {
        __nanosleep(40);
        if ((it & 255) == 255 && *(volatile int *)err) return v;
        v = ld_val(p);
    }
    if (unset(v)) atomicExch(err, 1);
    return v;
}
SPX_DEV double got(double v, const double *p, int *err) { return unset(v) ? await_val(p, err) : v; }
SPX_DEV double2 got2(double2 v, const double *p, int *err) {
    return make_double2(got(v.x, p, err), got(v.y, p + 1, err));
}
SPX_DEV double clean(double v) {
    return unset(v) ? __longlong_as_double(0x7ff8000000000000LL) : v;
}
SPX_DEV void put(const SVals &w, int64_t at, double v) {
    double *p = w.cur + at;
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(clean(v)) : "memory");
    p[w.other] = __longlong_as_double(kUnset);
}
SPX_DEV void put2(const SVals &w, int64_t at, double a, double b) {
    double *p = w.cur + at;
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(clean(a)), "d"(clean(b)) : "memory");
    const double n = __longlong_as_double(kUnset);
    *reinterpret_cast<double2 *>(p + w.other) = make_double2(n, n);
}
// Wait for the task's probe: whole warps poll one address, so that a task
// whose inputs are far off does not load the memory system with its gathers.
// The first load is issued when the task starts (v).
template <int NR>
SPX_DEV const double *probe_ptr(const SolveArgs &a, const STask &k, const double *cur) {
    return cur + (k.probe_at == 2 ? a.o_x : k.probe_at == 3 ? a.o_yf : 0) + (int64_t)k.probe * NR;
}

// n partial sums `step` apart, in order, eight loads in flight
SPX_DEV double sum_strips(const double *p0, int64_t step, int n, int *err) {
    double s = 0.0;
    for (int q = 0; q < n; q += 8) {
        double v[8];
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = q + e < n ? ld_val(p0 + (q + e) * step) : 0.0;
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (q + e < n) s += got(v[e], p0 + (q + e) * step, err);
    }
    return s;
}
// the same for NCH pairs 8 entries apart
template <int NCH>
SPX_DEV void sum_strips2(double2 (&s)[NCH], const double *p0, int64_t step, int n, int *err) {
    constexpr int U = NCH == 1 ? 6 : NCH == 2 ? 3 : 2;
#pragma unroll
    for (int ch = 0; ch < NCH; ch++) s[ch] = make_double2(0.0, 0.0);
    for (int q = 0; q < n; q += U) {
        double2 v[U][NCH];
#pragma unroll
        for (int e = 0; e < U; e++)
#pragma unroll
            for (int ch = 0; ch < NCH; ch++)
                v[e][ch] = q + e < n ? ld_val2(p0 + (q + e) * step + 8 * ch) : make_double2(0.0, 0.0);
#pragma unroll
        for (int e = 0; e < U; e++)
            if (q + e < n)
#pragma unroll
                for (int ch = 0; ch < NCH; ch++) {
                    const double2 u = got2(v[e][ch], p0 + (q + e) * step + 8 * ch, err);
                    s[ch].x += u.x;
                    s[ch].y += u.y;
                }
    }
}

// entries q0 <= q < q1 of the gather list, summed in order; two loads at a
// time in flight (most rows get one or two)
SPX_DEV double sum_vals(const double *u, const int32_t *cidx, const int *ci, int lo, bool staged,
                        int q0, int q1, int *err) {
    double s = 0.0;
    for (int q = q0; q < q1; q += 2) {
        const bool two = q + 1 < q1;
        const double *p0 = u + (staged ? ci[q - lo] : cidx[q]);
        const double *p1 = two ? u + (staged ? ci[q + 1 - lo] : cidx[q + 1]) : p0;
        const double v0 = ld_val(p0);
        double v1 = 0.0;
        if (two) v1 = ld_val(p1);
        s += got(v0, p0, err);
        if (two) s += got(v1, p1, err);
    }
    return s;
}

// The gather lists of a supernode that has long ones (a vertex with thousands
// of children below it): one row's entries follow one another at an L2 latency
// for two, so a row of more than kLongList is summed by its thread's warp,
// four loads a lane in flight, in a fixed order.  n rows, one a thread, with
// list offsets at ptr[0..n]; their sums are added to out[0..n).  Solves: star
// of 5,000 vertices 1.33 -> 0.070 ms, of 50,000 13.1 -> 0.45, 20,000 vertices
// at three of ten hubs each 3.3 -> 0.27.  (Inlined: as a function of its own
// it makes the kernel spill.)
SPX_DEV void add_long_lists(const double *u, const int32_t *cidx, const int *ptr, int n, double *out,
                            int *err) {
    const int t = threadIdx.x, lane = t & 31;
    const int q0 = t < n ? ptr[t] : 0, q1 = t < n ? ptr[t + 1] : 0;
    const bool mine = q1 - q0 > kLongList;
    double s = mine ? 0.0 : sum_vals(u, cidx, nullptr, 0, false, q0, q1, err);
    for (unsigned m = __ballot_sync(0xffffffffu, mine); m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        const int p0 = __shfl_sync(0xffffffffu, q0, src), p1 = __shfl_sync(0xffffffffu, q1, src);
        double v = 0.0;
        for (int q = p0 + lane; q < p1; q += 32 * 4) {
            int at[4];
            double x[4];
#pragma unroll
            for (int e = 0; e < 4; e++) at[e] = q + 32 * e < p1 ? cidx[q + 32 * e] : -1;
#pragma unroll
            for (int e = 0; e < 4; e++) x[e] = at[e] >= 0 ? ld_val(u + at[e]) : 0.0;
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (at[e] >= 0) v += got(x[e], u + at[e], err);
        }
        v = warp_sum(v);
        if (lane == src) s = v;
    }
    if (t < n) out[t] += s;
}

// ---- one right-hand side ------------------------------------------------
// Thread t works on rows 2 (t % 8) and the next of its group's row blocks;
// the 16 groups share the tile's row blocks and, where those are fewer, its
// columns (forward); or its columns and, where those are fewer, its row blocks
// (backward).  Either way 16 products a thread in pairs, then one small sum.
// Pairs because instructions count: the SMs issue every other cycle over the
// whole solve (ncu, 48^3: 51 % of the slots).  20^3 57 -> 49 us, 33x35x37 94 ->
// 82, 46^3 161 -> 148, 64^3 492 -> 467 against one row a thread and gathers in
// fours.
SPX_DEV int log2_at_least(int v) { return v <= 1 ? 0 : 32 - __clz(v - 1); }
SPX_DEV int pow2_at_least(int v) { return 1 << log2_at_least(v); }
// two adjacent rows of the tile (the swizzle keeps aligned groups of four)
SPX_DEV double2 ld_pair(const double *p) { return *reinterpret_cast<const double2 *>(p); }
SPX_DEV double2 ld_pair(const float *p) {
    const float2 v = *reinterpret_cast<const float2 *>(p);
    return make_double2(v.x, v.y);
}

SPX_DEV void vec_fwd(const SolveArgs &a, const SVals &w, const STask &k, STask &next, SNext<1> &nx,
                     uint32_t ph, SShared<1> &sh) {
    const int t = threadIdx.x, j0 = k.j0, jn = k.jn;
    const SLists l = lists_of<1>(k, sh.lists);
    const bool staged = k.pln + k.rln <= kListInts;
    const double *pp = probe_ptr<1>(a, k, w.cur);
    double pv = 0.0;
    if (k.probe_at) pv = ld_val(pp);
    mbar_wait(&sh.lfull, ph, a.err);
    double bv = 0.0;
    if (t < jn) bv = __ldg(a.bc + l.perm[t]);
    const bool below = k.strip == k.nstrip - 1 && t < k.nrow && k.i0 + t >= k.c;
    double bsum = 0.0;
    if (k.probe_at) got(pv, pp, a.err);
    nx.take(a);
    if (k.has_child == 2) {
        // into the vector segment: the columns' sums with b, the rows' behind it
        double *rows = sh.vec + kVecStrip;
        const int r0 = k.strip == k.nstrip - 1 ? min(k.nrow, max(0, k.c - k.i0)) : k.nrow;
        sh.vec[t] = bv;
        if (r0 + t < k.nrow) rows[r0 + t] = 0.0;
        add_long_lists(w.cur, a.cidx, l.cp, jn, sh.vec, a.err);
        add_long_lists(w.cur, a.cidx, l.rp + r0, k.nrow - r0, rows + r0, a.err);
    } else if (k.has_child) {
        if (t < jn) bv += sum_vals(w.cur, a.cidx, l.ci, k.pl0, staged, l.cp[t], l.cp[t + 1], a.err);
        if (below) bsum = sum_vals(w.cur, a.cidx, l.ri, k.rl0, staged, l.rp[t], l.rp[t + 1], a.err);
    }
    if (t < jn && k.has_child != 2) sh.vec[t] = bv;
    nx.read(a);
    mbar_wait(&sh.pfull, ph, a.err);
    __syncthreads();
    const int row = 2 * (t & 7), grp = t >> 3, lb = log2_at_least(k.nrb), P = kVecThreads / 8 >> lb;
    const int rb = grp & ((1 << lb) - 1), p = grp >> lb;
    double2 acc = make_double2(0.0, 0.0);
    if (rb < k.nrb) {
        const Real *G = sh.panel + rb * jn * 16;
        for (int j = p; j < jn; j += P) {
            const double2 g = ld_pair(G + j * 16 + (row ^ gswz(j0 + j)));
            const double v = sh.vec[j];
            acc.x += g.x * v;
            acc.y += g.y * v;
        }
    }
    *reinterpret_cast<double2 *>(sh.part + (p << lb) * 16 + rb * 16 + row) = acc;
    __syncthreads();
    if (t < k.nrow) {
        double own = 0.0;
        for (int q = 0; q < P; q++) own += sh.part[(q << lb) * 16 + t];
        if (k.strip < k.nstrip - 1) {
            put(w, a.o_fp + (int64_t)(k.slot0 + k.strip) * kVecRows + t, own);
        } else {
            // the chunk's other strips came before this one in the queue
            const double *p0 = w.cur + a.o_fp + (int64_t)k.slot0 * kVecRows + t;
            own += sum_strips(p0, kVecRows, k.nstrip - 1, a.err);
            const int ii = k.i0 + t;
            if (ii < k.c) put(w, a.o_yf + k.first + ii, own);
            else put(w, k.u + (ii - k.c), (k.has_child == 2 ? sh.vec[kVecStrip + t] : bsum) - own);
        }
    }
    nx.stage(a, next, sh);          // this task's tile and lists are done with
    __syncthreads();
}

SPX_DEV void vec_bwd(const SolveArgs &a, const SVals &w, const STask &k, STask &next, SNext<1> &nx,
                     uint32_t ph, SShared<1> &sh) {
    const int t = threadIdx.x, jn = k.jn;
    const SLists l = lists_of<1>(k, sh.lists);
    const double *pp = probe_ptr<1>(a, k, w.cur);
    const double pv = ld_val(pp);
    mbar_wait(&sh.lfull, ph, a.err);
    got(pv, pp, a.err);
    nx.take(a);
    constexpr int Q = kVecTall * 16 / kVecThreads;
    const double *src[Q];
    double v[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int i = t + q * kVecThreads, ii = k.i0 + i;
        v[q] = 0.0;
        if (i < k.nrow) {
            src[q] = w.cur + (ii < k.c ? a.o_yf + k.first + ii : a.o_x + l.rows[i]);
            v[q] = ld_val(src[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int i = t + q * kVecThreads;
        if (i < k.nrb * 16) {
            const double z = i < k.nrow ? got(v[q], src[q], a.err) : 0.0;
            sh.vec[i] = k.i0 + i < k.c ? z : -z;
        }
    }
    const int orow = t < jn ? l.perm[t] : 0;
    nx.read(a);
    mbar_wait(&sh.pfull, ph, a.err);
    __syncthreads();
    const int row = 2 * (t & 7), grp = t >> 3, lw = min(4, log2_at_least(jn));
    const int w2 = 1 << lw, P = kVecThreads / 8 >> lw, p = grp >> lw;
    static_assert(kVecThreads == 128, "16 groups");
    for (int j = grp & (w2 - 1); j < jn; j += w2) {
        double acc = 0.0;
        const Real *G = sh.panel + j * 16 + (row ^ gswz(k.j0 + j));
        for (int b = p; b < k.nrb; b += P) {
            const double2 g = ld_pair(G + b * jn * 16);
            const double2 v = *reinterpret_cast<const double2 *>(sh.vec + b * 16 + row);
            acc += g.x * v.x;
            acc += g.y * v.y;
        }
        const unsigned part = 0xffu << (t & 24);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(part, acc, o);
        if (row == 0) sh.part[p * w2 + j] = acc;
    }
    __syncthreads();
    if (t < jn) {
        double own = 0.0;
        for (int q = 0; q < P; q++) own += sh.part[q * w2 + t];
        if (k.strip < k.nstrip - 1) {
            put(w, a.o_bp + (int64_t)(k.slot0 + k.strip) * kBwdCols + t, own);
        } else {
            const double *p0 = w.cur + a.o_bp + (int64_t)k.slot0 * kBwdCols + t;
            own += sum_strips(p0, kBwdCols, k.nstrip - 1, a.err);
            put(w, a.o_x + k.first + k.j0 + t, own);
            a.xc[orow] = a.accumulate ? a.xc[orow] + own : own;
        }
    }
    nx.stage(a, next, sh);
    __syncthreads();
}

// ---- NR right-hand sides on the FP64 tensor cores -----------------------
// Fragment layout of m8n8k4: lane = 4 gq + tq holds A[gq][tq], B[tq][gq] and
// D[gq][2 tq .. 2 tq + 1].
// right-hand-side columns col, col + 1 of original row `row`
SPX_DEV double2 brhs2(const SolveArgs &a, int64_t row, int col) {
    return make_double2(col < a.nr ? __ldg(a.bc + (int64_t)col * a.ldb + row) : 0.0,
                        col + 1 < a.nr ? __ldg(a.bc + (int64_t)(col + 1) * a.ldb + row) : 0.0);
}

// The lists of more than kLongList entries among a forward tile's columns (cp,
// jn of them) and rows r0 <= r < nrow (rp), by the whole block: a thread takes
// a pair of right-hand sides and every so-and-so-many'th entry, four loads in
// flight; the shares are added in order.  Columns' sums are added to the
// vector segment at vec, rows' are left in the second half of it (see
// blk_long_rows).  A star of 5,000 vertices, 24 right-hand sides: 1.72 -> 0.14
// ms a solve.
template <int NR>
SPX_DEV double *blk_long_rows(double *vec) {
    return vec + kBlkStrip * SShared<NR>::SEG + kBlkThreads / (NR / 2) * NR;
}
template <int NR>
SPX_DEV void blk_long_lists(const double *u, const int32_t *cidx, const int *cp, int jn,
                            const int *rp, int r0, int nrow, double *vec, int *err) {
    constexpr int H = NR / 2, NS = kBlkThreads / H, SEG = SShared<NR>::SEG;
    static_assert(kBlkStrip * SEG + NS * NR + kBlkRows * NR <= kBlkTall * 16 * SEG, "long lists");
    double *part = vec + kBlkStrip * SEG, *rows = blk_long_rows<NR>(vec);
    const int t = threadIdx.x, h = t % H, sl = t / H;
    __syncthreads();                                      // the segment is written
    for (int e = 0; e < jn + nrow - r0; e++) {
        const bool pivot = e < jn;
        const int *p = pivot ? cp + e : rp + r0 + (e - jn);
        const int q0 = p[0], q1 = p[1];
        if (q1 - q0 <= kLongList) continue;               // for every thread
        double2 s = make_double2(0.0, 0.0);
        for (int q = q0 + sl; q < q1 && sl < NS; q += 4 * NS) {
            const double *src[4];
            double2 x[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                src[i] = u + (int64_t)(q + NS * i < q1 ? cidx[q + NS * i] : 0) * NR + 2 * h;
#pragma unroll
            for (int i = 0; i < 4; i++)
                x[i] = q + NS * i < q1 ? ld_val2(src[i]) : make_double2(0.0, 0.0);
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (q + NS * i < q1) {
                    const double2 v = got2(x[i], src[i], err);
                    s.x += v.x;
                    s.y += v.y;
                }
        }
        if (sl < NS) *reinterpret_cast<double2 *>(part + sl * NR + 2 * h) = s;
        __syncthreads();
        if (t < NR) {
            double v = 0.0;
            for (int i = 0; i < NS; i++) v += part[i * NR + t];
            if (pivot) vec[e * SEG + t] += v;
            else rows[(r0 + e - jn) * NR + t] = v;
        }
        __syncthreads();
    }
}

// rows x columns (64 x jn) times (jn x NR): warp w holds rows 8 w .. 8 w + 7
template <int NR>
SPX_DEV void blk_fwd(const SolveArgs &a, const SVals &w, const STask &k, STask &next, SNext<NR> &nx,
                     uint32_t ph, SShared<NR> &sh) {
    constexpr int NCH = NR / 8, H = NR / 2, SEG = SShared<NR>::SEG;
    constexpr int PP = kBlkStrip * H / kBlkThreads;       // (column, pair) items per thread
    const int t = threadIdx.x, jn = k.jn;
    const int lane = t & 31, wid = t >> 5, gq = lane >> 2, tq = lane & 3;
    const SLists l = lists_of<NR>(k, sh.lists);
    const bool staged = k.pln + k.rln <= kListInts, finish = k.strip == k.nstrip - 1;
    const double *pp = probe_ptr<NR>(a, k, w.cur);
    double pv = 0.0;
    if (k.probe_at) pv = ld_val(pp);
    mbar_wait(&sh.lfull, ph, a.err);
    double2 v[PP];
    // f = b + the children's updates of these pivots: the first two of a
    // pivot's gather entries for all of the thread's items at once
#pragma unroll
    for (int p = 0; p < PP; p++) {
        const int e = t + kBlkThreads * p, jj = e / H, h = e % H;
        v[p] = (jj < jn) ? brhs2(a, l.perm[jj], 2 * h) : make_double2(0.0, 0.0);
    }
    if (k.probe_at) got(pv, pp, a.err);
    nx.take(a);
    if (k.has_child) {
        const double *s0[PP], *s1[PP];
        double2 z0[PP], z1[PP];
        int q0[PP], q1[PP];
        auto entry = [&](int q) { return staged ? l.ci[q - k.pl0] : a.cidx[q]; };
#pragma unroll
        for (int p = 0; p < PP; p++) {
            const int e = t + kBlkThreads * p, jj = e / H, h = e % H;
            q0[p] = jj < jn ? l.cp[jj] : 0;
            q1[p] = jj < jn ? l.cp[jj + 1] : 0;
            if (k.has_child == 2 && q1[p] - q0[p] > kLongList) q1[p] = q0[p];
            s0[p] = w.cur + (int64_t)(q0[p] < q1[p] ? entry(q0[p]) : 0) * NR + 2 * h;
            s1[p] = w.cur + (int64_t)(q0[p] + 1 < q1[p] ? entry(q0[p] + 1) : 0) * NR + 2 * h;
            z0[p] = z1[p] = make_double2(0.0, 0.0);
            if (q0[p] < q1[p]) z0[p] = ld_val2(s0[p]);
            if (q0[p] + 1 < q1[p]) z1[p] = ld_val2(s1[p]);
        }
#pragma unroll
        for (int p = 0; p < PP; p++) {
            const double2 u0 = got2(z0[p], s0[p], a.err), u1 = got2(z1[p], s1[p], a.err);
            v[p].x = (v[p].x + u0.x) + u1.x;
            v[p].y = (v[p].y + u0.y) + u1.y;
            const int h = (t + kBlkThreads * p) % H;
            for (int q = q0[p] + 2; q < q1[p]; q++) {
                const double *sq = w.cur + (int64_t)entry(q) * NR + 2 * h;
                const double2 u = got2(ld_val2(sq), sq, a.err);
                v[p].x += u.x;
                v[p].y += u.y;
            }
        }
    }
#pragma unroll
    for (int p = 0; p < PP; p++) {
        const int e = t + kBlkThreads * p, jj = e / H, h = e % H;
        sh.vec[jj * SEG + 2 * h] = v[p].x;
        sh.vec[jj * SEG + 2 * h + 1] = v[p].y;
    }
    // the children's part of this lane's row below the pivots
    const int lr = wid * 8 + gq, ii = k.i0 + lr;
    double2 add[NCH];
#pragma unroll
    for (int ch = 0; ch < NCH; ch++) add[ch] = make_double2(0.0, 0.0);
    if (k.has_child == 2) {
        // rows below the pivots, of the chunk's finishing strip
        const int r0 = min(k.nrow, max(0, k.c - k.i0));
        blk_long_lists<NR>(w.cur, a.cidx, l.cp, jn, l.rp, r0, finish ? k.nrow : r0, sh.vec, a.err);
    }
    if (k.has_child && finish && lr < k.nrow && ii >= k.c) {
        const int q0 = l.rp[lr], n = l.rp[lr + 1] - q0;
        const bool summed = k.has_child == 2 && n > kLongList;
        if (summed)
#pragma unroll
            for (int ch = 0; ch < NCH; ch++)
                add[ch] = *reinterpret_cast<const double2 *>(blk_long_rows<NR>(sh.vec) + lr * NR +
                                                             8 * ch + 2 * tq);
        const int q1 = summed ? q0 : q0 + n;
        for (int q = q0; q < q1; q++) {
            const double *src = w.cur + (int64_t)(staged ? l.ri[q - k.rl0] : a.cidx[q]) * NR + 2 * tq;
            double2 z[NCH];
#pragma unroll
            for (int ch = 0; ch < NCH; ch++) z[ch] = ld_val2(src + 8 * ch);
#pragma unroll
            for (int ch = 0; ch < NCH; ch++) {
                const double2 u = got2(z[ch], src + 8 * ch, a.err);
                add[ch].x += u.x;
                add[ch].y += u.y;
            }
        }
    }
    nx.read(a);
    mbar_wait(&sh.pfull, ph, a.err);
    __syncthreads();
    double d[NCH][2];
#pragma unroll
    for (int ch = 0; ch < NCH; ch++) d[ch][0] = d[ch][1] = 0.0;
    if ((wid >> 1) < k.nrb) {
        const Real *G = sh.panel + (wid >> 1) * jn * 16;
        const int nks = (jn + 3) >> 2, rr = (wid & 1) * 8 + gq;
#pragma unroll 4
        for (int ks = 0; ks < nks; ks++) {
            const int j = ks * 4 + tq;
            const double av = j < jn ? (double)G[j * 16 + (rr ^ gswz(k.j0 + j))] : 0.0;
            const double *sb = sh.vec + j * SEG + gq;
#pragma unroll
            for (int ch = 0; ch < NCH; ch++) dmma(d[ch][0], d[ch][1], av, sb[8 * ch]);
        }
    }
    __syncthreads();
    if (lr < k.nrow) {
        if (!finish) {
            const int64_t at = a.o_fp + ((int64_t)(k.slot0 + k.strip) * kBlkRows + lr) * NR + 2 * tq;
#pragma unroll
            for (int ch = 0; ch < NCH; ch++) put2(w, at + 8 * ch, d[ch][0], d[ch][1]);
        } else {
            const double *p0 = w.cur + a.o_fp + ((int64_t)k.slot0 * kBlkRows + lr) * NR + 2 * tq;
            double2 tot[NCH];
            sum_strips2<NCH>(tot, p0, (int64_t)kBlkRows * NR, k.nstrip - 1, a.err);
            const int64_t at = ii < k.c ? a.o_yf + (int64_t)(k.first + ii) * NR : (k.u + (ii - k.c)) * NR;
#pragma unroll
            for (int ch = 0; ch < NCH; ch++) {
                const double s0 = tot[ch].x + d[ch][0], s1 = tot[ch].y + d[ch][1];
                if (ii < k.c) put2(w, at + 8 * ch + 2 * tq, s0, s1);
                else put2(w, at + 8 * ch + 2 * tq, add[ch].x - s0, add[ch].y - s1);
            }
        }
    }
    nx.stage(a, next, sh);
    __syncthreads();
}

// D = v^T G: M the right-hand sides, N eight columns, K the tile's rows.  The
// eight warps share the tile's columns and, where those are fewer than eight
// groups of eight, its rows.
template <int NR>
SPX_DEV void blk_bwd(const SolveArgs &a, const SVals &w, const STask &k, STask &next, SNext<NR> &nx,
                     uint32_t ph, SShared<NR> &sh) {
    constexpr int NCH = NR / 8, H = NR / 2, SEG = SShared<NR>::SEG;
    constexpr int PP = 4;                                // loads in flight per thread
    const int t = threadIdx.x, jn = k.jn;
    const int lane = t & 31, wid = t >> 5, gq = lane >> 2, tq = lane & 3;
    const SLists l = lists_of<NR>(k, sh.lists);
    const double *pp = probe_ptr<NR>(a, k, w.cur);
    const double pv = ld_val(pp);
    mbar_wait(&sh.lfull, ph, a.err);
    got(pv, pp, a.err);
    nx.take(a);
    for (int e0 = t; e0 < k.nrb * 16 * H; e0 += kBlkThreads * PP) {
        const double *src[PP];
        double2 v[PP];
#pragma unroll
        for (int p = 0; p < PP; p++) {
            const int e = e0 + kBlkThreads * p, i = e / H, h = e % H, ii = k.i0 + i;
            src[p] = w.cur + (ii < k.c ? a.o_yf + (int64_t)(k.first + ii) * NR
                                       : a.o_x + (int64_t)(i < k.nrow ? l.rows[i] : 0) * NR) + 2 * h;
            v[p] = i < k.nrow ? ld_val2(src[p]) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int p = 0; p < PP; p++) {
            const int e = e0 + kBlkThreads * p, i = e / H, h = e % H;
            if (i >= k.nrb * 16) continue;
            double2 z = i < k.nrow ? got2(v[p], src[p], a.err) : v[p];
            if (k.i0 + i >= k.c) { z.x = -z.x; z.y = -z.y; }
            sh.vec[i * SEG + 2 * h] = z.x;
            sh.vec[i * SEG + 2 * h + 1] = z.y;
        }
    }
    nx.read(a);
    mbar_wait(&sh.pfull, ph, a.err);
    __syncthreads();
    const int n8 = pow2_at_least((jn + 7) >> 3), parts = 8 / n8;   // column groups, row parts
    const int pc = (wid & (n8 - 1)) * 8 + gq;            // this lane's column (B side)
    double d[NCH][2];
#pragma unroll
    for (int ch = 0; ch < NCH; ch++) d[ch][0] = d[ch][1] = 0.0;
    if (pc - gq < jn) {
        const int sw = gswz(k.j0 + pc);
#pragma unroll 4
        for (int ks = wid / n8; ks < 4 * k.nrb; ks += parts) {
            const int i = ks * 4 + tq;
            const double bg = pc < jn ? (double)sh.panel[((i >> 4) * jn + pc) * 16 + ((i & 15) ^ sw)] : 0.0;
            const double *sa = sh.vec + i * SEG + gq;
#pragma unroll
            for (int ch = 0; ch < NCH; ch++) dmma(d[ch][0], d[ch][1], sa[8 * ch], bg);
        }
    }
    int orow[(kBwdCols * NR + kBlkThreads - 1) / kBlkThreads];
#pragma unroll
    for (int m = 0; m < (kBwdCols * NR + kBlkThreads - 1) / kBlkThreads; m++) {
        const int o = t + m * kBlkThreads;
        orow[m] = o < jn * NR ? l.perm[o / NR] : 0;
    }
    __syncthreads();
    // lane holds D[right-hand side 8 ch + gq][column 2 tq + e of its eight]
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
        for (int ch = 0; ch < NCH; ch++) sh.vec[(wid * 8 + 2 * tq + e) * NR + 8 * ch + gq] = d[ch][e];
    __syncthreads();
    const bool finish = k.strip == k.nstrip - 1;
#pragma unroll
    for (int m = 0; m < (kBwdCols * NR + kBlkThreads - 1) / kBlkThreads; m++) {
        const int o = t + m * kBlkThreads;               // (column, right-hand side)
        if (o >= jn * NR) break;
        double v = 0.0;
        for (int q = 0; q < parts; q++) v += sh.vec[q * n8 * 8 * NR + o];
        if (!finish) {
            put(w, a.o_bp + (int64_t)(k.slot0 + k.strip) * kBwdCols * NR + o, v);
        } else {
            v += sum_strips(w.cur + a.o_bp + (int64_t)k.slot0 * kBwdCols * NR + o, (int64_t)kBwdCols * NR,
                            k.nstrip - 1, a.err);
            put(w, a.o_x + (int64_t)(k.first + k.j0) * NR + o, v);
            const int rhs = o % NR;
            if (rhs < a.nr) {
                double *out = a.xc + (int64_t)rhs * a.ldx + orow[m];
                *out = a.accumulate ? *out + v : v;
            }
        }
    }
    nx.stage(a, next, sh);
    __syncthreads();
}

template <int NR>
__global__ void __launch_bounds__(SShared<NR>::kThreads, NR == 1 ? 8 : NR == 8 ? 3 : 2) mf_solve(SolveArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SShared<NR> &sh = *reinterpret_cast<SShared<NR> *>(smem_raw);
    chain_begin();
    if (a.skip && *(volatile const int *)a.skip) return;
    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init_n(&sh.lfull, 1);
        mbar_init_n(&sh.pfull, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int copy = *(volatile const int *)(a.sync + 2);
    const SVals w = {a.val + (copy ? a.stride : 0), copy ? -a.stride : a.stride};
    SNext<NR> nx = {0, -1};
    nx.take(a);
    nx.read(a);
    nx.stage(a, sh.task[0], sh);
    __syncthreads();
    for (unsigned it = 0;; it++) {
        const STask &k = sh.task[it & 1];
        if (k.kind < 0) break;
        STask &next = sh.task[(it & 1) ^ 1];
        if constexpr (NR == 1) {
            if (k.kind == SK_FWD) vec_fwd(a, w, k, next, nx, it & 1u, sh);
            else vec_bwd(a, w, k, next, nx, it & 1u, sh);
        } else {
            if (k.kind == SK_FWD) blk_fwd<NR>(a, w, k, next, nx, it & 1u, sh);
            else blk_bwd<NR>(a, w, k, next, nx, it & 1u, sh);
        }
    }
    // the last block to leave clears the queue and turns to the other copy for
    // the next solve
    if (tid == 0) {
        int old;
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(a.sync + 1) : "memory");
        if (old == (int)gridDim.x - 1) {
            a.sync[0] = 0;
            a.sync[1] = 0;
            a.sync[2] = copy ^ 1;
        }
    }
}

__global__ void fill_unset_kernel(double *p, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = __longlong_as_double(kUnset);
}
