// Sizes of the symbolic analysis for the test of its amalgamation: supernodes,
// tree levels, entries of the supernodes and of the factor before any merge
// (the column counts of the ordering the analysis ends with, by the row
// subtrees of the elimination tree).
#include "symbolic.h"

#include <vector>

extern "C" int symbolic_sizes(int32_t n, const int64_t *rp, const int32_t *ci, int64_t *out) {
    spx_symbolic S;
    if (int rc = spx_analyze(n, rp, ci, SPX_ORDER_AUTO, &S)) return rc;
    int64_t entries = 0, exact = n;
    for (int32_t s = 0; s < S.nsuper; s++) {
        const int64_t c = S.sfirst[s + 1] - S.sfirst[s], r = S.rowptr[s + 1] - S.rowptr[s];
        entries += c * (c + 1) / 2 + (r - c) * c;
    }
    std::vector<int32_t> par(n, -1), anc(n, -1), mark(n, -1);
    for (int32_t k = 0; k < n; k++)
        for (int64_t q = rp[S.perm[k]]; q < rp[S.perm[k] + 1]; q++)
            for (int32_t i = S.iperm[ci[q]], next; i >= 0 && i < k; i = next) {
                next = anc[i];
                anc[i] = k;
                if (next < 0) par[i] = k;
            }
    for (int32_t k = 0; k < n; k++) {
        mark[k] = k;
        for (int64_t q = rp[S.perm[k]]; q < rp[S.perm[k] + 1]; q++)
            for (int32_t i = S.iperm[ci[q]]; i < k && mark[i] != k; i = par[i]) {
                mark[i] = k;
                exact++;
            }
    }
    out[0] = S.nsuper;
    out[1] = S.nlevels;
    out[2] = entries;
    out[3] = exact;
    spx_symbolic_free(&S);
    return 0;
}
