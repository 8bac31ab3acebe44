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

/* query words between neighbouring warps of a multi-warp group */
constexpr int PK_FIFO = 32;

/* One class of a launch: pairs list[first, first + n) on `group` lanes each
 * (32 * the block's warps: the block), with rings of ring_cols words for
 * queries of up to max_q8 bases (in whole words). */
struct PkClass {
    int32_t group, first, n, ring_cols, max_q8;
    int32_t many; /* compare scoring: from this many pairs on one lane each, from a fifth two (0: never) */
};
constexpr int PK_CLASSES = 6;
struct PkClasses {
    int32_t n = 0, warp_words = 0; /* shared memory of a warp */
    PkClass k[PK_CLASSES] = {};
};

using PkKernel = void (*)(DpArgs, PkConst, PkClasses, const uint32_t *);
/* Compare scoring takes queries of PK_CMP_LONG bases on 32 lanes, shorter ones
 * on 4 (100k SEMI_GLOBAL 150 bp pairs with such targets: 8 lanes 4.1 ms).  Where
 * no query has more than PK_CMP_NARROW bases (32 rings of a warp then leave room
 * for 11 warps an SM), many pairs take fewer: 4 lanes are 8 virtual ones, more
 * than such a query's words or its rest of bands.  The kernel counts what is
 * left to it: from PK_CMP_MANY pairs an SM 1 lane, from a fifth of that 2.
 * LOCAL, us a call on 4 lanes / 1: 8k pairs 33 x 40 bases 57 / 68, 100 x 130
 * 129 / 298, 20 x 2,000 664 / 919; 40k 135 / 101, 409 / 528, 2,495 / 1,686; 60k
 * 175 / 103, 564 / 526, 3,519 / 1,703; 300k 692 / 309, 2,682 / 1,920, 17,190 /
 * 6,730. */
constexpr int PK_CMP_LONG = 64 * 8, PK_CMP_NARROW = 128, PK_CMP_MANY = 272;
/* compare scoring; table scoring in blocks of 1, 2, 4 warps */
enum PkVariant { PK_CMP, PK_W1, PK_W2, PK_W4, PK_VARIANTS };
PkKernel pk_kernel_local(PkVariant v, int start);
PkKernel pk_kernel_global(PkVariant v, int start);
PkKernel pk_kernel_semi(PkVariant v, int start);

/* lengths of the pairs of one class: their number, the longest query, target
 * and min(query, target) in whole words (8 bases), and (words) up to 128 of them */
struct PkLengths {
    int n = 0;
    uint32_t max_q = 0, max_t = 0, max_min = 0;
    int ns = 0;
    int qw[128], tw[128];
};
/* the shapes of a batch's launches */
struct PkPlan {
    int group[PK_CLASSES] = {};
    int ring_cols[PK_CLASSES] = {}, max_q8[PK_CLASSES] = {};
    int warp_words = 0, warps = 0, blocks = 0;         /* blocks: most that are resident */
    /* compare scoring: long pairs (32 lanes), short ones (4) */
    int cmp_cols[2] = {}, cmp_q8[2] = {}, cmp_many = 0, cmp_words = 0, cmp_blocks = 0;
};

/* The packed kernels take LOCAL, GLOBAL and target-tail SEMI_GLOBAL without a
 * second best (SEMI_GLOBAL: without a traceback): scores of pk_scores_ok, and
 * pairs whose longest query, longest target and longest min(query, target)
 * (in whole words) keep every value within 15 bits (pk_fits). */
bool pk_scores_ok(int algo, const Scores &sc);
bool pk_fits(int algo, const Scores &sc, uint32_t max_q, uint32_t max_t, uint32_t max_min);
PkConst pk_const(int algo, const Scores &sc);
/* false: no shape fits.  forced: least lanes per pair (1 to 32), or the 64 or
 * 128 of a two- or four-warp block; 0 = by the model */
bool pk_plan(int algo, int start, const PkLengths *cl, int sms, int forced, PkPlan &p);
/* n[c]: the pairs of class c, in list order.  wq: PK_QUEUE_WORDS zeroed words;
 * defer: a word per pair */
constexpr int PK_QUEUE_WORDS = PK_CLASSES + 4;
cudaError_t launch_dp_pk(int algo, int start, const DpArgs &a, const PkConst &pc, const PkPlan &p, const uint32_t *list,
                         const int *n, uint32_t *defer, uint32_t *wq, cudaStream_t s);

} // namespace gb

#endif
