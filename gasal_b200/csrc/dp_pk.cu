/*
 * dp_pk.cu -- which batches the packed kernels (dp_pk.cuh) take, their launch
 * constants, lane group and grid.
 */
#include "dp_pk.h"
#include "engine.h"

#include <algorithm>
#include <mutex>

namespace gb {

namespace {

uint32_t add2(int v) { return (uint32_t)v * 0x10001u; }                     /* for 32-bit adds: no carry between halves */
uint32_t two(int v) { return ((uint32_t)v & 0xFFFFu) | ((uint32_t)v << 16); } /* two signed 16-bit operands */

constexpr int C0_SIGNED = 16384; /* GLOBAL, SEMI_GLOBAL: zero in the middle of the 15 bits */

int c0_of(int algo, const Scores &sc)
{
    return algo == LOCAL_ ? sc.mismatch + 2 * sc.oe + 16 * sc.e + 64 : C0_SIGNED;
}
int b_of(int algo, const Scores &sc) { return algo == GLOBAL_ ? sc.mismatch - sc.e : sc.e; }

PkKernel pk_kernel(int algo, PkVariant v, int start)
{
    if (algo == LOCAL_) return pk_kernel_local(v, start);
    if (algo == GLOBAL_) return pk_kernel_global(v, start);
    return pk_kernel_semi(v, start);
}

/* registers and static shared memory of a kernel, read once */
struct KernelUse {
    int regs = 0, smem = 0;
};
KernelUse kernel_use(int algo, PkVariant v, int start)
{
    static std::mutex mu;
    static KernelUse cache[3][PK_VARIANTS][3];
    const int ai = algo == LOCAL_ ? 0 : algo == GLOBAL_ ? 1 : 2;
    std::lock_guard<std::mutex> lk(mu);
    KernelUse &u = cache[ai][v][start];
    if (u.regs == 0) {
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, (const void *)pk_kernel(algo, v, start)) == cudaSuccess)
            u.regs = fa.numRegs, u.smem = (int)fa.sharedSizeBytes;
        else
            cudaGetLastError();
    }
    return u;
}

/* resident warps per SM of `warps`-warp blocks with `smem` dynamic bytes (0: it cannot run) */
int resident_warps(const KernelUse &u, int warps, size_t smem)
{
    const size_t per_block = smem + (size_t)u.smem + 1024; /* 1 KB per block is the system's */
    if (u.regs == 0 || per_block > (227u << 10)) return 0;
    const int warp_regs = (u.regs * 32 + 255) / 256 * 256;
    int blocks = 65536 / (warp_regs * warps);
    blocks = std::min(blocks, (int)((228u << 10) / per_block));
    blocks = std::min(blocks, 64 / warps);
    blocks = std::min(blocks, 32);
    return blocks * warps;
}

} // namespace

bool pk_scores_ok(int algo, const Scores &sc)
{
    return sc.match >= 0 && sc.match <= 60 && sc.mismatch >= 0 && sc.mismatch <= 60 && sc.o >= 0 && sc.o <= 1000 &&
           sc.e >= 0 && sc.e <= 30 && (algo != GLOBAL_ || sc.mismatch >= sc.e);
}

/* Every value of the sweep must stay within the 15 bits of its half.  LOCAL:
 * the column key 4*H + 4*b*(bc+1) + 3 <= 32767.  max_min counts whole words: a
 * LOCAL sweep scores what follows a sequence in its last word.  GLOBAL / SEMI_GLOBAL: H lies between
 * the all-gap path, at least -(2o + e*(q+t) + mismatch), and match*min(q, t);
 * a gap opened from a mismatch below the lower end is the lowest value held. */
bool pk_fits(int algo, const Scores &sc, uint32_t max_q, uint32_t max_t, uint32_t max_min)
{
    const int64_t q8 = (max_q + 7) & ~7u, t8 = (max_t + 7) & ~7u;
    if (q8 > 12000 || t8 > 65528) return false;
    const int64_t top = (int64_t)sc.match * max_min;
    const int ab8 = 9 * (sc.e + b_of(algo, sc));
    if (algo == LOCAL_) return top <= 8191 - 8 * sc.e;
    const int64_t low = 3 * (int64_t)sc.o + 4 * (int64_t)sc.mismatch +
                        (int64_t)sc.e * (std::max<int64_t>(q8, 512) + t8 + 64) + ab8 + 256;
    return low <= C0_SIGNED - 64 && top + ab8 + sc.match + sc.mismatch <= 32767 - C0_SIGNED - 64;
}

PkConst pk_const(int algo, const Scores &sc)
{
    PkConst p{};
    p.c0 = c0_of(algo, sc), p.a = sc.e, p.b = b_of(algo, sc);
    p.mk = sc.match + sc.mismatch;
    p.m1 = add2(sc.match + p.a + p.b);
    p.n0 = add2(p.a + p.b);
    p.no = two(-sc.o);
    p.be = two(p.b - sc.e);
    p.tadd = add2(p.b - sc.oe);
    p.ra = add2(-8 * p.a), p.rb = add2(-8 * p.b);
    for (int d = 0; d < 15; d++) p.fl[d] = add2(p.c0 + sc.e * (d + 2));
    for (int k = 0; k < 8; k++) {
        p.kk[k] = add2(-4 * p.c0 - 4 * p.a * (k + 1) + 3 - (k & 3));
        p.kc[k] = two(-4 * p.b * (k + 1));
    }
    return p;
}

/* ring of a pair: a word per step of a round (an odd multiple of 4 words, so
 * the 128-bit accesses of groups side by side hit different banks) */
static int ring_words(int group, uint32_t max_q)
{
    return std::max((int)((max_q + 7) & ~7u), 16 * group) + 4;
}

/* steps of a pair of qw query words and nb bands on g lanes: rounds of its
 * bands over 2g virtual lanes, and as many more as the last round has bands */
static double steps_of(int g, int qw, int nb)
{
    const int V = 2 * g, rounds = (nb + V - 1) / V;
    return (double)rounds * (rounds > 1 ? std::max(qw, V) : qw) + (nb + V - 1) % V;
}

/* Lane group of each class, block and grid.  Narrow groups waste fewer
 * lane-steps on fill, drain and the last round; wide ones give each pair less
 * time and the chip more warps, and hold fewer rings.  A class's narrowest
 * group is the one whose rings fit RING_WORDS per warp (with the score table and
 * the system's share 11 one-warp blocks per SM; registers allow 16 warps).  From there the longest pairs' groups are widened
 * -- to 32 lanes, or to the block's two or four warps -- until the launch's
 * modelled time, the larger of all warps' steps at the SMs' rate and any
 * class's longest pair, stops falling.  A step of one of A resident warps of
 * an SM is modelled as max(A, 4) + 2.5 units (one warp a scheduler waits for
 * its own dependency chains: 65% of the integer pipe, two reach 73%); handing
 * over between two or four warps costs 15 or 45% more (20 pairs of 250-2,000
 * bp: 1,983 us with one warp, 1,427 with two, 1,236 with four). */
bool pk_plan(int algo, int start, const PkLengths *cl, int sms, int forced, PkPlan &p)
{
    constexpr int RING_WORDS = 4096 + 32 * 4;
    constexpr int WIDE = 6; /* group index of the whole block; below: 1 << k lanes */
    p = PkPlan();
    uint32_t max_q = 0;
    int n = 0;
    for (int c = 0; c < PK_CLASSES; c++)
        if (cl[c].n) n += cl[c].n, max_q = std::max(max_q, cl[c].max_q);
    double best_t = 0;
    for (int w : {1, 2, 4}) {
        if (forced > 32 && 32 * w != forced) continue;
        const KernelUse u = kernel_use(algo, w == 4 ? PK_W4 : w == 2 ? PK_W2 : PK_W1, start);
        const double hand = w == 4 ? 1.45 : 1.15;
        double cost[PK_CLASSES][WIDE + 1], longest[PK_CLASSES][WIDE + 1], limits[PK_CLASSES * (WIDE + 1)];
        int low[PK_CLASSES], nlimits = 0;
        const int top = w > 1 ? WIDE : WIDE - 1;
        for (int c = 0; c < PK_CLASSES; c++) {
            low[c] = 0;
            if (cl[c].n == 0) continue;
            const int qw = (int)((cl[c].max_q + 7) >> 3), tw = (int)((cl[c].max_t + 7) >> 3);
            while (low[c] < WIDE - 1 && ring_words(1 << low[c], cl[c].max_q) * (32 >> low[c]) > RING_WORDS) low[c]++;
            for (int k = low[c]; k <= top; k++) {
                const int g = k == WIDE ? 32 * w : 1 << k;
                const double f = k == WIDE ? hand : 1.0;
                double steps = 0;
                for (int x = 0; x < cl[c].ns; x++) steps += steps_of(g, cl[c].qw[x], cl[c].tw[x]);
                cost[c][k] = f * steps / std::max(cl[c].ns, 1) * cl[c].n * g / 32;
                longest[c][k] = f * steps_of(g, qw, tw);
                limits[nlimits++] = longest[c][k];
            }
            while (low[c] < WIDE - 1 && cost[c][low[c] + 1] < cost[c][low[c]]) low[c]++;
        }
        for (int x = 0; x < nlimits; x++) {
            int k[PK_CLASSES] = {}, words = 0;
            size_t wide_words = 0;
            double total = 0, work = 0, tail = 0;
            for (int c = 0; c < PK_CLASSES; c++) {
                if (cl[c].n == 0) continue;
                k[c] = low[c];
                if (forced > 32) k[c] = top;
                else if (forced > 0) while (k[c] < WIDE - 1 && (1 << k[c]) < forced) k[c]++;
                else while (k[c] < top && longest[c][k[c]] > limits[x]) k[c]++;
                const int g = k[c] == WIDE ? 32 * w : 1 << k[c];
                if (k[c] == WIDE)
                    wide_words = std::max<size_t>(wide_words, ring_words(g, cl[c].max_q) + (w - 1) * 8 * PK_FIFO);
                else words = std::max(words, ring_words(g, cl[c].max_q) * (32 / g));
                total += (double)cl[c].n * g / 32;
                work += cost[c][k[c]];
                tail = std::max(tail, longest[c][k[c]]);
            }
            words = std::max(words, (int)((wide_words / w + 7) & ~3));
            const int res = resident_warps(u, w, (size_t)words * w * 4);
            if (res == 0) continue;
            const double a = std::max(std::min(total / sms, (double)res), 1.0), step = std::max(a, 4.0) + 2.5;
            const double t = std::max(work / sms / a, tail) * step;
            if (p.warps == 0 || t < best_t) {
                best_t = t;
                p.warp_words = words, p.warps = w;
                p.blocks = std::max(sms * res / w, sms);
                for (int c = 0; c < PK_CLASSES; c++)
                    if (cl[c].n) {
                        p.group[c] = k[c] == WIDE ? 32 * w : 1 << k[c];
                        p.ring_cols[c] = ring_words(p.group[c], cl[c].max_q);
                        p.max_q8[c] = (int)((cl[c].max_q + 7) & ~7u);
                    }
            }
        }
    }
    if (p.warps == 0) return false;
    p.cmp_q8[0] = (int)((max_q + 7) & ~7u), p.cmp_q8[1] = std::min(p.cmp_q8[0], PK_CMP_LONG);
    p.cmp_cols[0] = p.cmp_q8[0] >= PK_CMP_LONG ? ring_words(32, max_q) : 0;
    p.cmp_cols[1] = ring_words(4, (uint32_t)p.cmp_q8[1]);
    p.cmp_many = p.cmp_q8[0] <= PK_CMP_NARROW ? PK_CMP_MANY * sms : 0;
    p.cmp_words = std::max(p.cmp_cols[0], (p.cmp_many ? 32 : 8) * p.cmp_cols[1]);
    const int res = resident_warps(kernel_use(algo, PK_CMP, start), 1, (size_t)p.cmp_words * 4);
    p.cmp_blocks = std::min(p.cmp_cols[0] ? n : (n + 7) / 8, std::max(sms * res, sms));
    return res > 0;
}

cudaError_t launch_dp_pk(int algo, int start, const DpArgs &a, const PkConst &pc, const PkPlan &p, const uint32_t *list,
                         const int *n, uint32_t *defer, uint32_t *wq, cudaStream_t s)
{
    PkClasses cl;
    int total = 0;
    long warps = 0;
    cl.warp_words = p.warp_words;
    for (int c = 0; c < PK_CLASSES; c++) {
        if (n[c] == 0) continue;
        cl.k[cl.n++] = {p.group[c], total, n[c], p.ring_cols[c], p.max_q8[c], 0};
        warps += ((long)n[c] * p.group[c] + 31) / 32;
        total += n[c];
    }
    if (total == 0) return cudaSuccess;
    auto launch = [&](PkVariant which, const DpArgs &x, const PkClasses &k, const uint32_t *l, int nb, int w) {
        const PkKernel f = pk_kernel(algo, which, start);
        const cudaError_t e = allow_dyn_smem_fn((const void *)f);
        if (e != cudaSuccess) return e;
        f<<<nb, 32 * w, (size_t)k.warp_words * w * 4, s>>>(x, pc, k, l);
        return cudaGetLastError();
    };
    /* the table-scoring launch, then the compare-scoring one over the pairs it
     * left (a target with another code than A, C, G, T, N) */
    DpArgs f = a;
    f.queue = wq, f.defer = defer, f.ndefer = wq + PK_CLASSES + 2, f.n_dev = nullptr;
    cudaError_t e = launch(p.warps == 4 ? PK_W4 : p.warps == 2 ? PK_W2 : PK_W1, f, cl, list,
                           (int)std::min<long>((warps + p.warps - 1) / p.warps, p.blocks), p.warps);
    if (e != cudaSuccess) return e;
    DpArgs c = f;
    c.queue = wq + PK_CLASSES, c.defer = nullptr, c.ndefer = nullptr, c.n_dev = f.ndefer;
    PkClasses left;
    left.warp_words = p.cmp_words;
    if (p.cmp_cols[0]) left.k[left.n++] = {32, 0, total, p.cmp_cols[0], p.cmp_q8[0], 0};
    left.k[left.n++] = {4, 0, total, p.cmp_cols[1], p.cmp_q8[1], p.cmp_many};
    return launch(PK_CMP, c, left, defer, std::min(total, p.cmp_blocks), 1);
}

} // namespace gb
