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

cudaError_t pk_visit(int algo, int group, int start, bool fast, const PkLaunchFn &f)
{
    if (algo == LOCAL_) return pk_visit_local(group, start, fast, f);
    if (algo == GLOBAL_) return pk_visit_global(group, start, fast, f);
    return pk_visit_semi(group, start, fast, f);
}

/* registers and static shared memory of a kernel, read once */
struct KernelUse {
    int regs = 0, smem = 0;
};
KernelUse kernel_use(int algo, int group, int start, bool fast)
{
    static std::mutex mu;
    static KernelUse cache[3][6][3][2];
    const int ai = algo == LOCAL_ ? 0 : algo == GLOBAL_ ? 1 : 2;
    const int gi = group == 2 ? 0 : group == 4 ? 1 : group == 8 ? 2 : group == 16 ? 3 : 4;
    std::lock_guard<std::mutex> lk(mu);
    KernelUse &u = cache[ai][gi][start][fast];
    if (u.regs == 0) {
        pk_visit(algo, group, start, fast, [&](PkKernel k) {
            cudaFuncAttributes fa;
            const cudaError_t e = cudaFuncGetAttributes(&fa, (const void *)k);
            if (e == cudaSuccess) u.regs = fa.numRegs, u.smem = (int)fa.sharedSizeBytes;
            return e;
        });
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
 * the column key 4*H + 4*b*(bc+1) + 3.  GLOBAL / SEMI_GLOBAL: H lies between
 * the all-gap path, at least -(2o + e*(q+t) + mismatch), and match*min(q, t);
 * a gap opened from a mismatch below the lower end is the lowest value held. */
bool pk_fits(int algo, const Scores &sc, uint32_t max_q, uint32_t max_t, uint32_t max_min)
{
    const int64_t q8 = (max_q + 7) & ~7u, t8 = (max_t + 7) & ~7u;
    if (q8 > 12000 || t8 > 65528) return false;
    const int64_t top = (int64_t)sc.match * max_min;
    const int ab8 = 9 * (sc.e + b_of(algo, sc));
    if (algo == LOCAL_) return top <= 8100 - 8 * sc.e;
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

/* Lane group, block and grid of a launch over the pairs `sample` stands for.
 * A pair on G lanes takes rounds*words steps (rounds: its bands over 2G) and
 * as many more as the last round has bands, so narrow groups waste fewer lane-steps on fill, drain and the last
 * round, and wide ones give each pair less time and the chip more warps.  An
 * SM with A resident warps was modelled as running A/(A+4) of its peak rate
 * (a lone warp waits for its own dependency chains); the group with the least
 * modelled time is taken.  Rings (one word per query column and pair) bound
 * the resident warps of narrow groups on long queries. */
WcLaunch pk_plan(int algo, int start, bool fast, int n, uint32_t max_q, const PkSample &sample, int sms, int forced)
{
    WcLaunch best;
    double best_t = 0;
    for (int g : {2, 4, 8, 16, 32}) {
        if (!fast && g != 8) continue;
        if (fast && forced > 0 && g != forced) continue;
        const KernelUse u = kernel_use(algo, g, start, fast);
        const int V = 2 * g;
        const size_t ring = std::max<size_t>((max_q + 7) & ~7u, 8 * V) * 4;
        double steps = 0;
        for (int k = 0; k < sample.n; k++) {
            const int qw = sample.qw[k], nb = sample.tw[k];
            const int rounds = (nb + V - 1) / V;
            steps += (double)rounds * (rounds > 1 ? std::max(qw, V) : qw) + (nb + V - 1) % V;
        }
        steps /= std::max(sample.n, 1);
        int res = 0, warps = 0;
        for (int wpb : {2, 4, 1}) {
            const int r = resident_warps(u, wpb, ring * wpb * (32 / g));
            if (r > res) res = r, warps = wpb;
        }
        if (res == 0) continue;
        const double total = ((double)n * g + 31) / 32 / sms; /* warps per SM */
        const double t = total <= res ? steps * (total + 4) : steps * total * (res + 4) / res;
        if (best.group == 0 || t < best_t) {
            best_t = t;
            if (total <= 4) warps = 1; /* small grids spread over the SMs */
            best.group = g, best.warps = warps, best.smem = ring * warps * (32 / g);
            best.resident_warps = res;
            const int per_block = warps * 32 / g;
            const int need = (n + per_block - 1) / per_block, cap = std::max(sms * res / warps, sms);
            best.blocks = std::min(need, cap);
        }
    }
    return best;
}

cudaError_t launch_dp_pk(int algo, int start, const DpArgs &a, const PkConst &pc, const uint32_t *list, int nlist,
                         uint32_t max_q, const WcLaunch &fast, const WcLaunch &cmp, uint32_t *defer, uint32_t *wq,
                         cudaStream_t s)
{
    if (nlist <= 0) return cudaSuccess;
    auto launch = [&](const DpArgs &x, const uint32_t *l, const WcLaunch &w, bool is_fast) {
        return pk_visit(algo, w.group, start, is_fast, [&](PkKernel k) {
            const cudaError_t e = allow_dyn_smem_fn((const void *)k);
            if (e != cudaSuccess) return e;
            const int ring_cols = (int)std::max<uint32_t>((max_q + 7) & ~7u, 16u * w.group);
            k<<<w.blocks, 32 * w.warps, w.smem, s>>>(x, pc, l, nlist, ring_cols);
            return cudaGetLastError();
        });
    };
    /* the table-scoring launch, then the compare-scoring one over the pairs it
     * left (a target with another code than A, C, G, T, N) */
    DpArgs f = a;
    f.queue = wq, f.defer = defer, f.ndefer = wq + 2, f.n_dev = nullptr;
    cudaError_t e = launch(f, list, fast, true);
    if (e != cudaSuccess) return e;
    DpArgs c = a;
    c.queue = wq + 1, c.defer = nullptr, c.ndefer = nullptr, c.n_dev = wq + 2;
    return launch(c, defer, cmp, false);
}

} // namespace gb
