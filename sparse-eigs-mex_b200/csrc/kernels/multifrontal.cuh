// Device multifrontal supernodal Cholesky and the shift-invert solve.
//
// Replaces cholmod_l_factorize_p (reference src/speigs_core.c:940, :966) and
// cholmod_l_solve2 (:96) for the 'sm' operator.  The host symbolic analysis
// (host/symbolic.h) fixes the supernodes and tree levels; this file owns the
// device copy of that structure, the tile task lists, and the kernels.
//
// Storage.  Every supernode s has 64 x 64 tiles for its pivot columns, the
// inverse of their triangle and its update matrix, live only during the
// factorization, and a persistent r x c panel
//     G_s = [ inv(L11) ; L21 * inv(L11) ]
// that replaces the usual [L11 ; L21].  With G, both triangular solves are a
// single dense (transposed) product per supernode, so every supernode of a
// tree level is solved in parallel with no sequential substitution.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "../host/symbolic.h"

namespace spx {

struct SolvePlan {      // one tile queue of the solve
    int ntasks = 0, fslots = 1, bslots = 1;
};

// Real is the storage type of the fronts and of the panels G: double for
// the plain FP64 operator, float for the mixed-precision one (FP64 products of
// FP32 tiles; the caller refines each solve in FP64).  Vectors are FP64 always.
template <class Real>
class MultifrontalPlanT {
public:
    MultifrontalPlanT() = default;
    ~MultifrontalPlanT();
    MultifrontalPlanT(const MultifrontalPlanT &) = delete;
    MultifrontalPlanT &operator=(const MultifrontalPlanT &) = delete;

    // Upload the symbolic structure and build the task lists.  rowptr/col
    // are the host copy of the full symmetric CSR (original numbering) whose
    // values live on the device at the same positions.  Returns 0 or a
    // negative SPEIGS_ERR_* code.
    int init(const spx_symbolic &S, const int64_t *rowptr, const int32_t *col,
             cudaStream_t st);

    // Numeric factorization of A + shift*I from the device CSR values.
    // A pivot <= pivtol counts as not positive.  Returns 0, 1 when a pivot
    // was not positive (A + shift*I not PD), or a negative error code.
    int factorize(const double *d_val, double shift, double pivtol, cudaStream_t st);

    // x = (A + shift I)^{-1} b  (b, x device vectors in the original order).
    // When `skip` is given and *skip is nonzero on the device, the launch
    // does nothing (refinement steps that are no longer needed).
    void solve(const double *b, double *x, cudaStream_t st, const int *skip = nullptr);

    // X = (A + shift I)^{-1} B for nr <= 32 right-hand sides at once: B and X
    // are column-major n x nr device arrays in the original order (leading
    // dimensions ldb, ldx).  One persistent launch runs the same task queue
    // as solve() with every vector entry widened to nr columns, so the panel
    // and the level structure are paid once for all columns.  `skip` as in
    // solve(); with `accumulate`, X += the solution instead of X = it.
    // Returns 0 or a negative code (device buffers for the block are
    // allocated on first use).
    int solve_block(const double *B, int64_t ldb, double *X, int64_t ldx, int nr,
                    cudaStream_t st, const int *skip = nullptr, bool accumulate = false);

    void release(cudaStream_t st);

    // device word set when a solve's dependency wait gave up (0 otherwise)
    int *error_word() const;

    int64_t n() const { return n_; }
    double factor_flops() const { return flops_; }
    int64_t panel_entries() const { return g_total_; }
    int64_t solve_bytes() const;      // algorithmic bytes of one solve pair
    int levels() const { return nlevels_; }

private:
    int32_t n_ = 0, ns_ = 0, nlevels_ = 0;
    double flops_ = 0.0;
    int64_t front_total_ = 0, g_total_ = 0, u_total_ = 0, nrows_total_ = 0;
    // device symbolic
    int32_t *d_perm_ = nullptr, *d_rows_ = nullptr, *d_relmap_ = nullptr;
    int32_t *d_acolptr_ = nullptr;   // [n+1] assembly entries per new column
    int32_t *d_atpos_ = nullptr;     // row position within the front
    int32_t *d_acolj_ = nullptr;     // column (new numbering)
    int32_t *d_asrc_ = nullptr;      // index into the CSR values
    int dup_ = 0;                    // some entry of A is stored more than once
    int32_t *d_cbnd_ = nullptr;      // child bounds per parent 64-row tile
    // factor: per-supernode metadata, child records, tile task queue, flags
    void *d_fnode_ = nullptr, *d_fchild_ = nullptr, *d_ftask_ = nullptr;
    int *d_fsync_ = nullptr;
    int64_t nflags_ = 0;
    int nftask_ = 0, factor_grid_ = 0;
    // solve: tile queues for one right-hand side and for a block, gather
    // lists; per column count (1, 8, 16, 24, 32) the values that pass between
    // tasks (two copies), their length and the grid
    SolvePlan vplan_, bplan_;
    void *d_vtask_ = nullptr, *d_btask_ = nullptr;
    int32_t *d_cptr_ = nullptr, *d_cidx_ = nullptr;
    int *d_sync_ = nullptr;
    double *d_sval_[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    int64_t sstride_[5] = {0, 0, 0, 0, 0};
    int sgrid_[5] = {0, 0, 0, 0, 0};
    int solve_setup(int q, cudaStream_t st);
    int run_solve(int q, const double *B, int64_t ldb, double *X, int64_t ldx, int nr,
                  cudaStream_t st, const int *skip, bool accumulate);
    // numeric
    Real *d_front_ = nullptr;
    Real *d_G_ = nullptr;
    double *d_params_ = nullptr;     // shift, pivot tolerance
};

using MultifrontalPlan = MultifrontalPlanT<double>;
using MultifrontalPlan32 = MultifrontalPlanT<float>;

// The members are defined in multifrontal.cu, which is compiled once per
// storage type; each translation unit specialises them for its type.
#define SPX_MF_DECLARE(R)                                                                    \
    template <> MultifrontalPlanT<R>::~MultifrontalPlanT();                                \
    template <> int MultifrontalPlanT<R>::init(const spx_symbolic &, const int64_t *,      \
                                               const int32_t *, cudaStream_t);             \
    template <> int MultifrontalPlanT<R>::factorize(const double *, double, double,        \
                                                    cudaStream_t);                         \
    template <> void MultifrontalPlanT<R>::solve(const double *, double *, cudaStream_t,   \
                                                 const int *);                            \
    template <> int MultifrontalPlanT<R>::solve_block(const double *, int64_t, double *,   \
                                                      int64_t, int, cudaStream_t,         \
                                                      const int *, bool);                 \
    template <> int MultifrontalPlanT<R>::solve_setup(int, cudaStream_t);                  \
    template <> int MultifrontalPlanT<R>::run_solve(int, const double *, int64_t,          \
                                                    double *, int64_t, int, cudaStream_t,  \
                                                    const int *, bool);                    \
    template <> void MultifrontalPlanT<R>::release(cudaStream_t);                          \
    template <> int *MultifrontalPlanT<R>::error_word() const;                             \
    template <> int64_t MultifrontalPlanT<R>::solve_bytes() const;
SPX_MF_DECLARE(double)
SPX_MF_DECLARE(float)
#undef SPX_MF_DECLARE

}  // namespace spx
