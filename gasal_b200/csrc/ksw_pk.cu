/*
 * ksw_pk.cu -- ksw seed extension, one warp per pair, row-parallel, two
 * columns per register (int16x2).
 *
 * The rows are ksw_wc.cu's (reference src/kernels/ksw_kernel_template.h:
 * 46-199): target order, each over the trimmed range [beg, end) that the
 * previous row's zero and non-zero eh entries decide.  What bounds a row is
 * instructions: per column the score lookup, M', the gap opened from it, E, F
 * and H, and per tile the F scan over the lanes, the row maximum and the
 * trimming.  A 16x2 instruction does two columns at the price of one, and a
 * lane that takes 16 columns halves the tiles of a row, so:
 *
 *   eh lives in shared memory as words of 8 columns, H and E apart, a word's
 *   columns k and k+4 (k = 0..3) in the halves of one register: one 128-bit
 *   access each per word.  A lane takes one word per tile (256 columns), or
 *   two (512) while more than 256 columns remain.
 *
 *   F's fold and its second pass run on both halves at once (columns 0-3 and
 *   4-7 of a word), the second half starting from the first one's fold; the
 *   scan over lanes is ksw_wc.cu's, one value per lane.
 *
 *   M' = M ? M + s : 0 is min(M + s, M * (match + 1)): that is M + s for M >= 1
 *   and 0 or less for M = 0, which every use treats as 0.
 *
 *   Entries at and right of `end` are 0 (the first row spans the query, and a
 *   row is only cut where its entries are 0), so a row's last tile stores 0
 *   there instead of leaving them.
 *
 * Measured on a B200 against ksw_wc.cu's kernel: 50k pairs of 250-2,000 bp 44.2
 * to 30.8 ms, 200k of 50-5,000 bp 57.7 to 40.9 ms (lane groups for the short
 * ones in both); about 400 instructions per row, the integer pipe at 70%.
 *
 * Takes pairs of plain codes whose largest value times match + 1 fits 15 bits;
 * the others go to a list for ksw_wc.cu's kernels.
 */
#include "dp_core.cuh"

#include <algorithm>

namespace gb {
namespace {

constexpr unsigned ALL = 0xFFFFFFFFu;

__device__ __forceinline__ int lo16(uint32_t x) { return (int)(x & 0xFFFFu); }
__device__ __forceinline__ int hi16u(uint32_t x) { return (int)(x >> 16); }

/* Words lie even ones first, then odd ones `half` further (half = 4 mod 8, 64
 * bytes across the banks): the 128-bit accesses of a tile hit all banks whether
 * its lanes take consecutive words or every other one. */
struct Words {
    uint4 *H, *E;
    uint4 *sel; /* prmt selectors of a word's four column pairs */
    int n, half;
    __device__ __forceinline__ int at(int g) const { return (g >> 1) + ((g & 1) ? half : 0); }
    /* column j's halfword in H or E */
    __device__ __forceinline__ int hw(int j) const { return at(j >> 3) * 8 + ((j & 3) << 1 | ((j >> 2) & 1)); }
    __device__ __forceinline__ uint16_t *h16() const { return reinterpret_cast<uint16_t *>(H); }
    __device__ __forceinline__ uint16_t *e16() const { return reinterpret_cast<uint16_t *>(E); }
};

struct RowConst {
    uint2 tab;
    uint32_t cmul, noe, ne; /* match + 1; packed -(gap open + extend), -gap extend */
    int e, lane, end;
    const uint4 *keep; /* keep[v]: the first v columns of a word */
};
struct RowState {
    int fcarry, hcarry; /* F and H entering the next tile */
    int m, mcol;        /* row maximum so far; the last of its columns is one of 16 from here */
    int first, last;    /* the row's non-zero entries start among the two words from `first`, end among
                           the two up to `last` (-1: none) */
};

/* One tile: NW words per lane from word g0 on.  FULL: all its columns lie
 * before the row's end.  Right of the end M', E and the gap values come out 0
 * of zero entries; only F can spill, so H is stored up to eh[end] and 0 after
 * it, and the row maximum needs no mask (a spilled F lies below the H it was
 * opened from, or ties with it -- the column search reads stored values). */
template <int NW, bool FULL>
__device__ __forceinline__ void row_tile(const Words &wd, const RowConst &c, int g0, RowState &st)
{
    const int lane = c.lane, g = g0 + lane * NW;
    uint32_t M[NW][4], T[NW][4], E[NW][4], H[NW][4], agg[NW];
    int at[NW];
#pragma unroll
    for (int w = 0; w < NW; w++) {
        at[w] = wd.at(FULL || g + w < wd.n ? g + w : 0); /* (lanes past the row read word 0) */
        const uint4 h4 = wd.H[at[w]], e4 = wd.E[at[w]], s4 = wd.sel[at[w]];
        const uint32_t h[4] = {h4.x, h4.y, h4.z, h4.w}, s[4] = {s4.x, s4.y, s4.z, s4.w};
        E[w][0] = e4.x, E[w][1] = e4.y, E[w][2] = e4.z, E[w][3] = e4.w;
#pragma unroll
        for (int p = 0; p < 4; p++) {
            M[w][p] = __viaddmin_s16x2(h[p], prmt(c.tab.x, c.tab.y, s[p]), h[p] * c.cmul);
            T[w][p] = __viaddmax_s16x2(M[w][p], c.noe, 0u);
            agg[w] = p == 0 ? T[w][0] : __viaddmax_s16x2(agg[w], c.ne, T[w][p]);
        }
    }
    /* F leaving the lane from its own columns; scan over lanes (a lane below
     * the shift gets its own value back, which never wins: e >= 0) */
    int x = 0;
#pragma unroll
    for (int w = 0; w < NW; w++) {
        x = w == 0 ? lo16(agg[0]) : __viaddmax_s32(x, -4 * c.e, lo16(agg[w]));
        x = __viaddmax_s32(x, -4 * c.e, hi16u(agg[w]));
    }
    const int eL = 8 * NW * c.e;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) x = __viaddmax_s32(__shfl_up_sync(ALL, x, d), -eL * d, x);
    const int ex = __shfl_up_sync(ALL, x, 1);
    int f = lane == 0 ? st.fcarry : __viaddmax_s32(st.fcarry, -eL * lane, ex);
    f = max(f, 0);
    st.fcarry = __shfl_sync(ALL, __viaddmax_s32(st.fcarry, -eL * (lane + 1), x), 31);
    uint32_t top = 0;
#pragma unroll
    for (int w = 0; w < NW; w++) {
        const int f4 = __viaddmax_s32(f, -4 * c.e, lo16(agg[w]));
        uint32_t F = mad_lo_u32((uint32_t)f4, 65536u, (uint32_t)f);
        if (w + 1 < NW) f = __viaddmax_s32(f4, -4 * c.e, hi16u(agg[w]));
#pragma unroll
        for (int p = 0; p < 4; p++) {
            H[w][p] = __vimax3_s16x2(M[w][p], E[w][p], F);
            E[w][p] = __viaddmax_s16x2(E[w][p], c.ne, T[w][p]);
            if (p < 3) F = __viaddmax_s16x2(F, c.ne, T[w][p]);
        }
        top = __vimax3_s16x2(top, H[w][0], H[w][1]);
        top = __vimax3_s16x2(top, H[w][2], H[w][3]);
    }
    /* row maximum, and which lane has it last (ties: the later tile's) */
    const int mine = max(lo16(top), hi16u(top)), tm = __reduce_max_sync(ALL, mine);
    const unsigned who = __ballot_sync(ALL, mine == tm);
    if (tm >= st.m) st.m = tm, st.mcol = (g0 + (31 - __clz((int)who)) * NW) << 3;
    /* store: H moves one column right */
    uint32_t in = __shfl_up_sync(ALL, H[NW - 1][3], 1);
    if (lane == 0) in = (uint32_t)st.hcarry << 16;
    st.hcarry = hi16u(__shfl_sync(ALL, H[NW - 1][3], 31));
    const int left = c.end - (g << 3); /* columns of the row from this lane's first on */
    uint32_t any = 0;
#pragma unroll
    for (int w = 0; w < NW; w++) {
        uint4 hv = make_uint4(prmt(w == 0 ? in : H[w > 0 ? w - 1 : 0][3], H[w][3], 0x5432u), H[w][0], H[w][1], H[w][2]);
        const uint4 ev = make_uint4(E[w][0], E[w][1], E[w][2], E[w][3]);
        if (!FULL) {
            const uint4 k = c.keep[min(max(left + 1 - 8 * w, 0), 8)];
            hv.x &= k.x, hv.y &= k.y, hv.z &= k.z, hv.w &= k.w;
        }
        if (FULL || left >= 8 * w) wd.H[at[w]] = hv, wd.E[at[w]] = ev;
        any |= (hv.x | hv.y | hv.z) | (hv.w | ev.x | ev.y) | (ev.z | ev.w);
    }
    /* lanes with a non-zero entry: the first one's first and the last one's last word */
    const unsigned bm = __ballot_sync(ALL, any != 0);
    if (bm) {
        if (st.first < 0) st.first = g0 + (__ffs((int)bm) - 1) * NW;
        st.last = g0 + (32 - __clz((int)bm)) * NW - 1;
    }
}

__device__ void ksw_pk_pair(const DpArgs &a, uint32_t pid, const Words &wd, const uint2 *stab, const uint4 *keep,
                            int lane, int qlen, int tlen, const uint32_t *t, int h0, unsigned long long &ncells)
{
    const int e = a.sc.e, oe = a.sc.oe, o = a.sc.o;
    uint16_t *Hh = wd.h16();
    const uint16_t *Eh = wd.e16();
    /* the reference's first row (ksw_kernel_template.h:75-79) */
    for (int w = lane; w < wd.n; w += 32) wd.H[wd.at(w)] = wd.E[wd.at(w)] = make_uint4(0, 0, 0, 0);
    __syncwarp();
    const int v1 = h0 > oe ? h0 - oe : 0;
    for (int j = lane; j <= qlen; j += 32) {
        int h = 0;
        if (j == 0) h = h0;
        else if (j == 1) h = v1;
        else if (v1 - (long long)(j - 2) * e > e) h = v1 - (j - 1) * e;
        if (h) Hh[wd.hw(j)] = (uint16_t)h;
    }
    __syncwarp();
    const int L8 = (qlen >> 3) << 3;
    int mx = h0, max_i = -1, max_j = -1, max_ie = -1, gscore = -1, mo = 0;
    int beg = 0, end = qlen;
    ncells = 0;
    RowConst rc;
    rc.noe = ((uint32_t)-oe & 0xFFFFu) * 0x10001u, rc.ne = ((uint32_t)-e & 0xFFFFu) * 0x10001u;
    rc.cmul = (uint32_t)(max(a.sc.match, 0) + 1), rc.e = e, rc.lane = lane, rc.keep = keep;
    for (int i = 0; i < tlen;) {
        rc.tab = stab[code(__ldg(t + (i >> 3)), i & 7)];
        rc.end = end;
        int h1 = 0;
        if (beg == 0) h1 = max((int)((uint32_t)h0 - (uint32_t)(o + e * (i + 1))), 0);
        RowState st{0, h1, 0, 0, -1, -1};
        int w0 = beg >> 3;
        if (beg < end) {
            ncells += (unsigned long long)(end - beg);
            for (const int wend = (end + 7) >> 3; w0 < wend;) { /* wend: one past the row's last word */
                if (wend - w0 > 32) {
                    if (end >= (w0 + 64) << 3) row_tile<2, true>(wd, rc, w0, st);
                    else row_tile<2, false>(wd, rc, w0, st);
                    w0 += 64;
                } else {
                    if (end == (w0 + 32) << 3) row_tile<1, true>(wd, rc, w0, st);
                    else row_tile<1, false>(wd, rc, w0, st);
                    w0 += 32;
                }
            }
        }
        /* eh[end] = H(end - 1): stored by the last tile, or the value that left it */
        if ((end >> 3) >= w0 && lane == 0) Hh[wd.hw(end)] = (uint16_t)st.hcarry;
        __syncwarp();
        h1 = Hh[wd.hw(end)];
        const int m = st.m;
        if (max(L8, end) == qlen) {
            max_ie = gscore > h1 ? max_ie : i;
            gscore = max(gscore, h1);
        }
        bool leave = false;
        if (m == 0) {
            leave = true;
        } else if (m > mx || (a.zdrop > 0 && mx - m > a.zdrop)) {
            /* the maximum's last column is wanted: one of 16, at eh[column + 1] */
            const int jj = st.mcol + 1 + (lane & 15);
            const unsigned at = __ballot_sync(ALL, jj <= end && Hh[wd.hw(min(jj, end))] == m);
            const int mj = st.mcol + 15 - __clz((int)(at << 16));
            if (m > mx) {
                mx = m, max_i = i, max_j = mj;
                mo = max(mo, abs(mj - i));
            } else {
                leave = mx - m - abs((i - max_i) - (mj - max_j)) * e > a.zdrop;
            }
        }
        if (leave) {
            i = ((i >> 3) + 1) << 3;
        } else {
            /* trimming (ksw_kernel_template.h:188-196): one ballot, lanes 0-15
             * over the two words the entries start in, 16-31 over the two they
             * end in */
            const int jj = lane < 16 ? (st.first << 3) + lane : (st.last << 3) + lane - 24;
            const int x = wd.hw(min(max(jj, 0), end));
            const unsigned bal = __ballot_sync(ALL, st.first >= 0 && jj >= 0 && jj < end && (Hh[x] | Eh[x]) != 0);
            const int nbeg = (bal & 0xFFFFu) ? (st.first << 3) + __ffs((int)(bal & 0xFFFFu)) - 1 : end;
            int lastnz = nbeg - 1;
            if (h1 != 0) lastnz = end;
            else if (bal >> 16) lastnz = (st.last << 3) + 7 - __clz((int)bal);
            beg = nbeg;
            end = lastnz + 2 < qlen ? lastnz + 2 : qlen;
            i++;
        }
        __syncwarp(); /* the reads above come before the next row's stores */
    }
    if (lane == 0) {
        const bool at_max = gscore <= 0 || gscore <= mx - 5;
        if (a.score) a.score[pid] = at_max ? mx : gscore;
        if (a.q_end) a.q_end[pid] = at_max ? max_j + 1 : qlen;
        if (a.t_end) a.t_end[pid] = (at_max ? max_i : max_ie) + 1;
        if (a.max_off) a.max_off[pid] = mo;
    }
    __syncwarp();
}

/* queries of q_lo .. 8 * words - 2 bases (longer ones to `rest` when
 * `handback`, else the next class launch's) */
__global__ void __launch_bounds__(32) ksw_pk_kernel(DpArgs a, const uint32_t *list, int nlist, int words, int q_lo,
                                                    int handback, uint32_t *rest, uint32_t *nrest, uint32_t *wq,
                                                    unsigned long long *cells)
{
    extern __shared__ __align__(16) uint4 ksw_pk_smem[];
    __shared__ uint2 stab[16];
    __shared__ uint4 keep[9];
    const int lane = threadIdx.x;
    build_score_table(stab, a.sc, true);
    if (lane < 9) {
        auto m = [&](int p) { return (lane > p ? 0xFFFFu : 0u) | (lane > p + 4 ? 0xFFFF0000u : 0u); };
        keep[lane] = make_uint4(m(0), m(1), m(2), m(3));
    }
    __syncthreads();
    const int half = words / 2 + 4;
    const Words wd{ksw_pk_smem, ksw_pk_smem + 2 * half, ksw_pk_smem + 4 * half, words, half};
    const uint32_t n = a.n_dev ? min(*a.n_dev, (uint32_t)nlist) : (uint32_t)nlist;
    const long long mpos = max(a.sc.match, 0);
    for (;;) {
        uint32_t idx = 0;
        if (lane == 0) idx = atomicAdd(wq, 1u);
        idx = __shfl_sync(ALL, idx, 0);
        if (idx >= n) break;
        const uint32_t pid = list ? list[idx] : idx;
        const int qlen = (int)a.q_len[pid], tlen = (int)a.t_len[pid];
        if (qlen < q_lo) continue;
        const bool fits = qlen + 2 <= 8 * words;
        if (!fits && !handback) continue;
        const uint32_t h0 = a.seed ? a.seed[pid] : 0u;
        bool ok = fits && ((long long)h0 + mpos * qlen) * (mpos + 1) < 32768;
        const uint32_t *q = a.pq + (a.q_off[pid] >> 3), *t = a.pt + (a.t_off[pid] >> 3);
        if (ok) {
            const int qregs = (qlen + 7) >> 3, tregs = (tlen + 7) >> 3;
            uint32_t bad = 0;
            for (int x = lane; x < qregs + tregs; x += 32) {
                const uint32_t y = x < qregs ? q[x] : t[x - qregs];
#pragma unroll
                for (int k = 0; k < 8; k++) bad |= ~(PLAIN_CODES >> ((y >> (4 * k)) & 15u)) & 1u;
            }
            ok = __all_sync(ALL, bad == 0);
            /* selectors: class byte and its sign, columns k and k + 4 */
            for (int x = lane; ok && x < words; x += 32) {
                const uint32_t y = x < qregs ? q[x] : 0u;
                uint32_t s[4];
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    const uint32_t c0 = class_of((y >> (28 - 4 * p)) & 15u), c1 = class_of((y >> (12 - 4 * p)) & 15u);
                    s[p] = (c0 * 0x11u | 0x80u) | ((c1 * 0x11u | 0x80u) << 8);
                }
                wd.sel[wd.at(x)] = make_uint4(s[0], s[1], s[2], s[3]);
            }
        }
        if (!ok) {
            if (lane == 0) rest[atomicAdd(nrest, 1u)] = pid;
            continue;
        }
        __syncwarp();
        unsigned long long nc = 0;
        ksw_pk_pair(a, pid, wd, stab, keep, lane, qlen, tlen, t, (int)h0, nc);
        if (cells && lane == 0) atomicAdd(cells, nc);
    }
}

} // namespace

bool ksw_pk_scores_ok(const Scores &sc)
{
    return sc.match >= -128 && sc.match <= 127 && sc.mismatch >= 0 && sc.mismatch <= 128 && sc.o >= 0 && sc.e >= 0 &&
           sc.oe > 0 && sc.oe <= 16000;
}

cudaError_t launch_ksw_pk(const DpArgs &a, const uint32_t *list, int nlist, int slots, int q_lo, bool handback,
                          uint32_t *rest, uint32_t *nrest, uint32_t *wq, unsigned long long *cells, cudaStream_t s)
{
    if (nlist <= 0) return cudaSuccess;
    const int words = slots / 8;
    const size_t smem = (size_t)(words / 2 + 4) * 96;
    cudaError_t e = allow_dyn_smem(ksw_pk_kernel);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 148, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ksw_pk_kernel, 32, smem);
    if (e != cudaSuccess) return e;
    const int blocks = std::max(1, std::min(nlist, std::max(per_sm, 1) * sms));
    ksw_pk_kernel<<<blocks, 32, smem, s>>>(a, list, nlist, words, q_lo, handback ? 1 : 0, rest, nrest, wq, cells);
    return cudaGetLastError();
}

} // namespace gb
