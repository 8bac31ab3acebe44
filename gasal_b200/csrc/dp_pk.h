/*
 * dp_pk.h -- plan and launch of the packed (two bands per lane, int16x2)
 * sweeps of dp_pk.cuh.
 */
#ifndef GB_DP_PK_H
#define GB_DP_PK_H

#include <functional>

#include "gb_internal.h"

namespace gb {

/* Launch constants of the packed kernels (kernel parameter space: the cell
 * loop reads them as constant-bank operands).  Words named for a packed use
 * hold the value in both halves. */
struct PkConst {
    int32_t c0, a, b;   /* value'' = value + c0 + a*(k+1) + b*(bc+1) */
    int32_t mk;         /* match + mismatch */
    int32_t zero;       /* 0 */
    uint32_t m1;        /* packed add of match + a + b */
    uint32_t n0;        /* packed a + b: N against anything, outside GLOBAL */
    uint32_t no;        /* packed -gap_open */
    uint32_t be;        /* packed b - gap_extend (GLOBAL) */
    uint32_t tadd;      /* packed add of b - gap_open - gap_extend (GLOBAL) */
    uint32_t ra, rb;    /* packed add of -8a, -8b */
    uint32_t fl[15];    /* LOCAL: packed floor (value 0) on the block's antidiagonals */
    uint32_t kk[8];     /* LOCAL: packed add turning 4*H'' of row k into its column key */
    uint32_t kc[8];     /* LOCAL: packed -4*b*(bc+1) */
};

using PkKernel = void (*)(DpArgs, PkConst, const uint32_t *, int, int);
using PkLaunchFn = std::function<cudaError_t(PkKernel)>;

/* calls f with the kernel of (algo, group, start, scoring) */
cudaError_t pk_visit_local(int group, int start, bool fast, const PkLaunchFn &f);
cudaError_t pk_visit_global(int group, int start, bool fast, const PkLaunchFn &f);
cudaError_t pk_visit_semi(int group, int start, bool fast, const PkLaunchFn &f);

/* lengths (words) of up to 256 pairs standing for a launch's */
struct PkSample {
    int n = 0;
    int qw[256], tw[256];
};

/* The packed kernels take LOCAL, GLOBAL and target-tail SEMI_GLOBAL without a
 * second best (SEMI_GLOBAL: without a traceback): scores of pk_scores_ok, and
 * pairs whose longest query, longest target and longest min(query, target)
 * keep every value within 15 bits (pk_fits). */
bool pk_scores_ok(int algo, const Scores &sc);
bool pk_fits(int algo, const Scores &sc, uint32_t max_q, uint32_t max_t, uint32_t max_min);
PkConst pk_const(int algo, const Scores &sc);
/* launch shape for n pairs (forced: a lane group, 0 = by the model) */
WcLaunch pk_plan(int algo, int start, bool fast, int n, uint32_t max_q, const PkSample &sample, int sms, int forced);
/* wq: three zeroed words (the two launches' work counters, the count of
 * pairs the first leaves to the second); defer: nlist words */
cudaError_t launch_dp_pk(int algo, int start, const DpArgs &a, const PkConst &pc, const uint32_t *list, int nlist,
                         uint32_t max_q, const WcLaunch &fast, const WcLaunch &cmp, uint32_t *defer, uint32_t *wq,
                         cudaStream_t s);

} // namespace gb

#endif
