/*
 * dp_pk.cuh -- LOCAL, GLOBAL and target-tail SEMI_GLOBAL sweeps with two 8-row
 * bands per lane in the halves of int16x2 registers.  Included by one
 * translation unit per algorithm (dp_pk_local.cu, dp_pk_global.cu,
 * dp_pk_semi.cu); plan and dispatch are in dp_pk.cu.
 *
 * What bounds it.  A cell is a handful of max and add-max operations on the
 * half-rate integer pipe; a 16x2 instruction of that pipe takes the same two
 * issue cycles per warp as a 32-bit one and does two cells.  So the lanes pack
 * two cells per register, and the recurrence is arranged to need few
 * operations per packed cell (5 on that pipe, the score lookup included):
 *
 *   Every value is held with an offset that grows along the block,
 *   value'' = value + c0 + a*(k+1) + b*(bc+1) at row k of the band and column
 *   bc of the 8-column word.  With a = gap extend the vertical gap needs no
 *   decay, E'' = max(E'', M'' - o): one add-max.  b = gap extend (LOCAL,
 *   SEMI_GLOBAL) does the same for F; in GLOBAL b = mismatch - gap extend, so
 *   that the score table is never negative, M'' = D'' + s'' is a plain 32-bit
 *   add (no carry between the halves) and a pad row's selector can give the
 *   mismatch score exactly.  c0 keeps everything non-negative; the offsets
 *   return to their start at each word (F, D: - 8b) and band (H, E: - 8a).
 *
 * Layout.  A pair is swept by a group of G lanes as V = 2G virtual lanes:
 * virtual lane v takes the 8-row bands v, v+V, v+2V, ... one 8-column query
 * word per step, one step behind virtual lane v-1.  The low half of lane L is
 * virtual lane 2L, the high half 2L+1: the low half's outputs of the last step
 * are the high half's inputs of this one, and the high half's travel to lane
 * L+1 by one shuffle per column.  The last virtual lane's outputs reach the
 * first, one round later, through a ring of one word per query column in
 * shared memory.  Against one band per lane this halves the instructions per
 * cell and the shuffles, and keeps one ring per pair (packing two pairs per
 * lane instead doubles the rings and halves the resident warps).
 *
 * W = 2 and 4: the warps of a block share a pair, for pairs that would outlast
 * the rest of the launch.  Warp x takes the bands of every W-th round; the warps run
 * unsynchronised, each
 * handing its last virtual lane's outputs to the next through a fifo of
 * PK_FIFO words with counters, the last to the first through the ring.  The
 * waits are bounded: the warp votes after each, so one lane whose polls run out
 * ends the whole warp's sweep at the same step, and sets a word that the host
 * reports as an error (one lane polling for the warp through a shuffle instead
 * cost 100k LOCAL tracebacks of 50-5,000 bp 5%).  No warp waits in a circle: a
 * round has at least as many steps as the group virtual lanes, and the ring
 * holds a whole one, so the last warp never waits for room.
 *
 * Measured on a B200 (us a batch, before with one pair per thread below 32
 * query words and one band per lane above, after): 300k SEMI_GLOBAL 150 bp with
 * starts 6,960 / 4,710; 200k LOCAL of 50-5,000 bp with starts 51,700 / 27,000;
 * 150k SEMI_GLOBAL of the same lengths 39,400 / 19,000; 100k GLOBAL of
 * 50-1,000 bp with traceback 19,000 / 6,400; 5k GLOBAL 150 bp 460 / 135; 1k
 * LOCAL of 250-2,000 bp 750,000 / 2,950.  Rates on equal lengths of 500: GLOBAL
 * 5.1 T cells/s, SEMI_GLOBAL 4.2, LOCAL 3.6.  A LOCAL step of a warp is about 700 instructions, 500 of
 * them on that pipe (73% busy at two warps a scheduler).
 *
 * H and E cross a band boundary as 16-bit values, as in the reference's short2
 * row buffer; the host only sends pairs here whose values cannot leave 15 bits
 * (pk_fits), so the results are the reference's bit for bit.
 */
#ifndef GB_DP_PK_CUH
#define GB_DP_PK_CUH

#include "dp_core.cuh"
#include "dp_pk.h"

#include <type_traits>

namespace gb {
namespace {

constexpr uint32_t PAD_WORD = 0xEEEEEEEEu; /* eight N codes */

__device__ __forceinline__ int half_of(uint32_t x, bool hi) { return (int)(int16_t)(hi ? x >> 16 : x & 0xFFFFu); }
/* both halves of x with half `hi` replaced by v (16 bits) */
__device__ __forceinline__ uint32_t set_half(uint32_t x, int v, bool hi)
{
    return prmt(x, (uint32_t)v, hi ? 0x5410u : 0x3254u);
}

/* nibble mask (8) of the rows of a word that are not below `valid` */
__device__ __forceinline__ uint32_t pad_nibbles(int valid)
{
    return valid >= 8 ? 0u : valid <= 0 ? 0x88888888u : 0x88888888u >> (4 * valid);
}
/* nibble mask (1) of the word's N codes (14) */
__device__ __forceinline__ uint32_t n_nibbles(uint32_t w)
{
    return ~w & (w >> 1) & (w >> 2) & (w >> 3) & 0x11111111u;
}
/* a word whose first `valid` codes are bases: 1 = some code (pads included) is
 * none of A, C, G, T (1, 3, 7, 4) and N, 2 = some base is N, 4 = some pad is
 * not (the reference's reversal leaves the pads in front of the bases) */
__device__ __forceinline__ uint32_t odd_codes(uint32_t w, int valid)
{
    const uint32_t b1 = w >> 1, b2 = w >> 2, b3 = w >> 3;
    const uint32_t pads = pad_nibbles(valid) >> 3;
    const uint32_t acgt = ~b3 & ((~b2 & w) | (b2 & ~(b1 ^ w))), n = n_nibbles(w);
    return ((~(acgt | n) & 0x11111111u) ? 1u : 0u) | ((n & ~pads) ? 2u : 0u) | ((~n & pads) ? 4u : 0u);
}

/* 2-bit class of the four bases (code >> 1) & 3: A 0, C 1, T 2, G 3 */
constexpr uint32_t PK_REP = 1u | (3u << 4) | (4u << 8) | (7u << 12);

/* tab[c1 << 4 | c2]: the four score bytes of query codes c1 and c2 against the
 * classes, offset a + b included */
__device__ void pk_score_table(uint2 *tab, const Scores &sc, bool n_zero, int ab)
{
    auto row = [&](int r) {
        uint32_t w = 0;
        for (int j = 0; j < 4; j++) {
            const int g = (int)((PK_REP >> (4 * j)) & 15u);
            const int v = ab + ((n_zero && r == 14) ? 0 : (r == g ? sc.match : -sc.mismatch));
            w |= (uint32_t)(v & 0xFF) << (8 * j);
        }
        return w;
    };
    for (int x = threadIdx.x; x < 256; x += blockDim.x) tab[x] = make_uint2(row(x >> 4), row(x & 15));
}

/* The pairs list[0], list[dir], .. (nl of them) on G lanes of W warps each, taken from the zeroed
 * counter `queue`.  smem: the warp's rings (W > 1: the block's).
 * FAST: targets of A, C, G, T and N, scores by one prmt per packed cell (its
 * selector's bytes: the row's class, then that byte's sign).  Otherwise
 * compares, any code. */
template <int G, int W, int ALGO, int START, bool FAST>
__device__ __forceinline__ void pk_pairs(const DpArgs &A, const PkConst &P, const uint2 *tab, uint32_t *pk_smem,
                                         const uint32_t *list, int nl, uint32_t *queue, int ring_cols, int max_q8,
                                         int dir = 1)
{
    constexpr int LANES = G * W;
    constexpr int V = 2 * G;
    constexpr bool LOC = ALGO == LOCAL_, GLO = ALGO == GLOBAL_, SEM = ALGO == SEMI_GLOBAL_;
    constexpr bool TB = START == WITH_TB_;
    const int lane = threadIdx.x & 31, gl = lane & (G - 1), gbase = lane & ~(G - 1);
    const unsigned gmask = G == 32 ? 0xFFFFFFFFu : (((1u << (G & 31)) - 1u) << gbase);
    const int o = A.sc.o, e = A.sc.e, oe = A.sc.oe;
    const bool free_head_t = SEM && (A.head == TARGET_ || A.head == BOTH_);
    const bool zero_rows = SEM && (A.head == QUERY_ || A.head == BOTH_);
    const int wi = W > 1 ? (int)(threadIdx.x >> 5) : 0;
    /* the last warp's outputs to the first: a word per query column; between
     * neighbouring warps of a group: PK_FIFO query words */
    uint32_t *ring = pk_smem + (W > 1 ? 0 : (size_t)(lane / G) * ring_cols);
    uint32_t *fifo = pk_smem + ring_cols; /* warp w's at fifo + w * 8 * PK_FIFO */
    /* W > 1: query words handed on and taken, counted over the rounds; a start
     * pass's first band with a hit; the group's item and results */
    __shared__ volatile int prod[W], cons[W], s_stop;
    __shared__ int s_item, s_key[W], s_res[3];
    auto ran_out = [&]() {
        if (lane == 0) {
            *const_cast<volatile uint32_t *>(A.stuck) = 1u;
            __threadfence_system();
        }
    };
    auto group_any = [&](bool x) -> bool {
        if (W > 1) return __syncthreads_or(x);
        return __ballot_sync(0xFFFFFFFFu, x) & gmask;
    };

    for (;;) {
        unsigned item0 = 0;
        if (W > 1) {
            __syncthreads();
            if (threadIdx.x == 0) s_item = (int)atomicAdd(queue, 1u);
            __syncthreads();
            item0 = (unsigned)s_item;
        } else {
            if (lane == 0) item0 = atomicAdd(queue, (unsigned)(32 / G));
            item0 = __shfl_sync(0xFFFFFFFFu, item0, 0);
        }
        if ((int)item0 >= nl) break;
        const int item = (int)item0 + lane / G;
        const bool listed = item < nl;
        const int i = listed ? (list ? (int)list[dir * item] : item) : 0;
        const int qlen0 = listed ? (int)A.q_len[i] : 0, tlen0 = listed ? (int)A.t_len[i] : 0;
        /* longer than the host's copy of the lengths said: its ring would not hold it.  Never
         * written, as in the one-thread kernel (this only guards memory), and not walked */
        auto too_long = [&]() { return (uint32_t)qlen0 > (uint32_t)max_q8; };
        auto skip = [&]() {
            if (TB && gl == 0 && wi == 0) A.tb_kind[i] = 2;
        };
        const uint32_t *q = A.pq + (listed ? (A.q_off[i] >> 3) : 0);
        const uint32_t *t = A.pt + (listed ? (A.t_off[i] >> 3) : 0);
        bool has = listed, with_n = false;
        if (FAST) {
            uint32_t odd = too_long() ? 1u : 0u, odd_q = 0;
            const int x0 = W > 1 ? (int)threadIdx.x : gl;
            for (int x = x0; 8 * x < tlen0; x += LANES) odd |= odd_codes(t[x], tlen0 - 8 * x);
            bool bad = odd & 1u;
            if (GLO) {
                /* N is an ordinary base: a target N scores as against A, C, G or T unless the
                 * query has N too (with a traceback, either one's N meets the other's pads) */
                for (int x = x0; 8 * x < qlen0; x += LANES) odd_q |= odd_codes(q[x], qlen0 - 8 * x);
                const bool tn = group_any(odd & 2u);
                bad |= TB ? tn || (odd_q & 2u) : tn && (odd_q & 2u);
            } else {
                with_n = W > 1 ? group_any(odd & 6u) : __any_sync(0xFFFFFFFFu, odd & 6u);
            }
            if (group_any(bad)) {
                /* left to compare scoring: short pairs from the list's front, long ones from its end */
                if (too_long()) {
                    skip();
                } else if (listed && gl == 0 && wi == 0) {
                    if (qlen0 >= PK_CMP_LONG) A.defer[A.n - 1 - (int)atomicAdd(A.ndefer + 1, 1u)] = (uint32_t)i;
                    else A.defer[atomicAdd(A.ndefer, 1u)] = (uint32_t)i;
                }
                has = false;
            }
        } else if (too_long()) {
            skip();
            has = false;
        }
        const bool work = has && qlen0 > 0 && tlen0 > 0;
        const int qlen = work ? qlen0 : 0, tlen = work ? tlen0 : 0;
        const int qregs = (qlen + 7) >> 3, tregs = (tlen + 7) >> 3;
        uint32_t *tops = nullptr, *lefts = nullptr;
        if (TB && work) {
            tops = reinterpret_cast<uint32_t *>(A.tb + A.tb_off[i]);
            lefts = tops + (size_t)((tregs + 1) >> 1) * (qregs << 3);
        }
        if (TB && has && gl == 0 && wi == 0) A.tb_kind[i] = 1;
        int score = 0, r_qe = 0, r_te = 0, r_qs = 0, r_ts = 0;

#pragma unroll 1
        for (int pass = 0; pass < (START == WITH_START_ && !GLO ? 2 : 1); pass++) {
            const bool rev = START == WITH_START_ && pass == 1;
            /* the sweep's query words, target bands and first band */
            int qn = qregs, nb = tregs, T0 = 0;
            if (rev && LOC) {
                qn = score > 0 ? min((r_qe >> 3) + 1, qregs) : 0;
                nb = score > 0 ? min((r_te >> 3) + 1, tregs) : 0;
            }
            if (rev && SEM) {
                const int x = tregs - ((r_te >> 3) + 1);
                T0 = max(x > 0 ? x - 1 : x, 0);
                nb = work ? tregs - T0 : 0;
            }
            /* rounds of warp x of the group: it takes bands (r*W + x)*V .. of round r */
            auto rounds_of = [&](int x) { return qn > 0 && nb > x * V ? (nb - x * V + W * V - 1) / (W * V) : 0; };
            const int rounds = rounds_of(wi);
            /* steps of a round: the group's first virtual lane comes to a word of the next
             * round after the last one has done it */
            const int per = rounds_of(0) > 1 ? max(qn, W * V) : qn;
            /* done when the last band's virtual lane is */
            int gend = rounds > 0 ? rounds * per + min(V - 1, nb - 1 - ((rounds - 1) * W + wi) * V) : 0;
            int wend = W > 1 ? gend : (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)gend);
            const bool multi = W == 1 && wend > 0 && __any_sync(0xFFFFFFFFu, rounds > 1);
            /* words the next warp will take from this one, and where */
            const int wanted = W == 1 ? 0 : wi < W - 1 ? rounds_of(wi + 1) * per : (rounds_of(0) - 1) * per;
            int avail = 0, taken = 0;
            if (W > 1) {
                __syncthreads();
                if (lane == 0) prod[wi] = 0, cons[wi] = 0;
                if (threadIdx.x == 0) s_stop = 0x7fffffff, s_res[0] = s_res[1] = s_res[2] = 0;
                __syncthreads();
            }
            const int lastw = (qlen - 1) >> 3, lastb = (qlen - 1) & 7;

            auto qword = [&](int j) -> uint32_t {
                if (j < 0 || j >= qn) return PAD_WORD;
                if (!rev) return __ldg(q + j);
                if (LOC) return nib_rev(__ldg(q + (qn - 1 - j)));
                return rev_window(q, qlen - 8 - (j << 3));
            };
            /* band T's rows: their classes with 8 set on pad and N rows (FAST), or their codes */
            auto tword = [&](int T) -> uint32_t {
                if (T >= nb) return FAST ? 0x88888888u : PAD_WORD;
                uint32_t w, pad = 0;
                if (!rev) {
                    w = __ldg(t + T);
                } else if (LOC) {
                    w = nib_rev(__ldg(t + (nb - 1 - T)));
                } else {
                    w = rev_window(t, tlen - 8 - 8 * (T0 + T)), pad = pad_nibbles(tlen - 8 * (T0 + T));
                }
                return FAST ? (((w >> 1) & 0x33333333u) | pad | (n_nibbles(w) << 3)) : w;
            };

            uint32_t F[8], D[8], sel[8], oH[8], oE[8], xw[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                F[k] = D[k] = oH[k] = oE[k] = (uint32_t)P.c0 * 0x10001u;
                xw[k] = oH[k];
                sel[k] = 0;
            }
            int w = -2 * gl, r = 0, wh = w - 1, rh = 0;
            uint32_t qw = qword(w), qp = PAD_WORD;
            /* the halves' next bands' words, loaded a round ahead of use */
            uint32_t t_lo = tword(wi * V + 2 * gl), t_hi = tword(wi * V + 2 * gl + 1);
            /* LOCAL: key of the best cell so far (4 * H + 3), per half; a start
             * pass looks for the forward score.  SEMI_GLOBAL: best last-column
             * value, in basis (0, lastb) */
            uint32_t thr = LOC ? (rev ? (uint32_t)(4 * score - 1) * 0x10001u : 0x00030003u) : 0u;
            int at_lo = -1, at_hi = -1;     /* LOCAL: band << 16 | word; SEMI_GLOBAL: row */
            uint32_t keys_lo[8], keys_hi[8]; /* LOCAL: that block's column keys, rows 0-3 and 4-7 */
            bool hit_lo = false, hit_hi = false;
            const int sbase = SEM ? P.c0 + P.a + P.b * (lastb + 1) : 0;

            /* NT (LOCAL, SEMI_GLOBAL): rows of N before the end of some target of the warp, which
             * score 0 by a bitwise select per packed cell.  Without it N rows score what the
             * selector gives, 0 or less, which changes nothing when only pads follow them */
            auto sweep = [&](auto nt) {
            constexpr bool NT = decltype(nt)::value;
            uint32_t nrow[8];
#pragma unroll
            for (int k = 0; k < 8; k++) nrow[k] = 0;
            for (int s = 0; s < wend; s++) {
                const int band_lo = (r * W + wi) * V + 2 * gl, band_hi = (rh * W + wi) * V + 2 * gl + 1;
                if (W > 1 && s < rounds * per) { /* wait for the word that lane 0 reads */
                    const int src = wi > 0 ? wi - 1 : W - 1, need = wi > 0 ? s : s - per;
                    bool late = false;
                    for (int spin = 0; need >= avail && !late;) {
                        avail = prod[src];
                        late = ++spin > A.spins;
                    }
                    if (__any_sync(0xFFFFFFFFu, late)) { /* never: the producer's step does not wait on this one */
                        ran_out();
                        wend = s;
                    }
                    __threadfence_block();
                }
                /* next step's query word: in flight during this one (and before the fence that
                 * ends it, which waits for loads) */
                const uint32_t qx = qword(w + 1 == per ? 0 : w + 1);
                const int stop_seen = W > 1 && rev ? s_stop : 0x7fffffff;
                const bool on = s < gend;
                const bool live_lo = on && w >= 0 && band_lo < nb, live_hi = on && wh >= 0 && band_hi < nb;
                /* H and E entering the low half's band at this word's columns */
                uint32_t xin[8];
#pragma unroll
                for (int b = 0; b < 8; b++) xin[b] = __shfl_up_sync(0xFFFFFFFFu, xw[b], 1, G);
                if (gl == 0) {
                    if ((r == 0 && wi == 0) || r >= rounds) { /* past the last round: values no carry can come from */
#pragma unroll
                        for (int b = 0; b < 8; b++) {
                            const int c = (w << 3) + b;
                            int h = 0, ev = 0;
                            if (GLO) h = c == 0 ? 0 : -(o + e * c);
                            if (SEM && !zero_rows) h = c == 0 ? 0 : -(o + e * c), ev = h - oe;
                            if (SEM && zero_rows) ev = -e;
                            const int hb = P.c0 + P.b * (b + 1) + h;
                            const int eb = GLO ? 0 : P.c0 + P.a + P.b * (b + 1) + ev;
                            xin[b] = (uint32_t)hb | ((uint32_t)eb << 16);
                        }
                    } else {
                        const uint4 *rp = reinterpret_cast<const uint4 *>(
                            W > 1 && wi > 0 ? fifo + ((wi - 1) * PK_FIFO + (s & (PK_FIFO - 1))) * 8 : ring + (w << 3));
                        const uint4 x0 = rp[0], x1 = rp[1];
                        xin[0] = x0.x, xin[1] = x0.y, xin[2] = x0.z, xin[3] = x0.w;
                        xin[4] = x1.x, xin[5] = x1.y, xin[6] = x1.z, xin[7] = x1.w;
                    }
                }
                if (W > 1 && wi > 0 && lane == 0) {
                    __threadfence_block();
                    cons[wi] = s + 1;
                }
                if (TB && live_lo && w < qregs) {
                    uint4 *p4 = reinterpret_cast<uint4 *>(tops + (size_t)(band_lo >> 1) * (qregs << 3) + (w << 3));
                    p4[0] = make_uint4(xin[0], xin[1], xin[2], xin[3]);
                    p4[1] = make_uint4(xin[4], xin[5], xin[6], xin[7]);
                }
                /* a half entering a new band: its rows' selectors and left boundary */
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if ((h ? wh : w) == 0) {
                        const int band = h ? band_hi : band_lo;
                        const uint32_t tw = h ? t_hi : t_lo;
                        if (h) t_hi = tword(band + W * V);
                        else t_lo = tword(band + W * V);
                        const int R0 = band < nb ? band << 3 : 0;
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            const uint32_t x = (tw >> (28 - 4 * k)) & 15u;
                            if (FAST) {
                                if (h) sel[k] = (sel[k] & 0x00FFu) | (((x * 0x11u) | 0x80u) + 0x44u) << 8;
                                else sel[k] = (sel[k] & 0xFF00u) | (x * 0x11u) | 0x80u;
                                if (NT) nrow[k] = set_half(nrow[k], x >= 8u ? 0xFFFF : 0, h);
                            } else {
                                sel[k] = set_half(sel[k], (int)x, h);
                            }
                            int dv = 0, fv = 0;
                            const int R = R0 + k, edge = R == 0 ? 0 : -(o + e * R);
                            if (GLO) dv = edge;
                            if (SEM) dv = free_head_t ? 0 : edge, fv = (free_head_t ? 0 : -(o + e * R)) - oe;
                            D[k] = set_half(D[k], P.c0 + P.a * k + dv, h);
                            F[k] = set_half(F[k], GLO ? 0 : P.c0 + P.a * (k + 1) + P.b + fv, h);
                        }
                    }
                    if (TB) {
                        const int ww = h ? wh : w;
                        if ((h ? live_hi : live_lo) && !(ww & 1) && ww < qregs) {
                            const uint32_t m = h ? 0x7632u : 0x5410u;
                            uint4 *p4 = reinterpret_cast<uint4 *>(lefts + (size_t)(ww >> 1) * (tregs << 3) +
                                                                  ((h ? band_hi : band_lo) << 3));
                            p4[0] = make_uint4(prmt(D[0], F[0], m), prmt(D[1], F[1], m), prmt(D[2], F[2], m),
                                               prmt(D[3], F[3], m));
                            p4[1] = make_uint4(prmt(D[4], F[4], m), prmt(D[5], F[5], m), prmt(D[6], F[6], m),
                                               prmt(D[7], F[7], m));
                        }
                    }
                }
                /* the column that ends the pair (SEMI_GLOBAL: every band's; GLOBAL: the last band's) */
                const bool fin_lo = !LOC && live_lo && w == lastw && (SEM || band_lo == nb - 1);
                const bool fin_hi = !LOC && live_hi && wh == lastw && (SEM || band_hi == nb - 1);
                const int finb = (fin_lo || fin_hi) ? lastb : 8;
                uint32_t hc[8];
#pragma unroll
                for (int k = 0; k < 8; k++) hc[k] = 0;

                uint32_t cA[8], cB[8], bk = 0;
                uint2 tl = make_uint2(0, 0), th = make_uint2(0, 0);
#pragma unroll
                for (int b = 0; b < 8; b++) {
                    uint32_t sl = 0, sh = 0, rr = 0, rn = 0;
                    if (FAST) {
                        if (!(b & 1)) {
                            tl = tab[(qw >> (24 - 4 * b)) & 255u];
                            th = tab[(qp >> (24 - 4 * b)) & 255u];
                        }
                        sl = (b & 1) ? tl.y : tl.x;
                        sh = (b & 1) ? th.y : th.x;
                    } else {
                        rr = ((qw >> (28 - 4 * b)) & 15u) | (((qp >> (28 - 4 * b)) & 15u) << 16);
                        rn = __vcmpeq2(rr, 0x000E000Eu);
                    }
                    const uint32_t inH = prmt(xin[b], oH[b], 0x5410u);
                    uint32_t E = prmt(xin[b], oE[b], 0x5432u);
                    uint32_t H[8], key[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        uint32_t Dm, sv = 0;
                        if (FAST) {
                            sv = prmt(sl, sh, sel[k]);
                            if (NT) sv = (sv & ~nrow[k]) | (P.n0 & nrow[k]);
                            Dm = D[k];
                        } else {
                            /* u = 0 for a match, match + mismatch otherwise; N scores 0 outside GLOBAL */
                            uint32_t u = __vminu2((sel[k] ^ rr) * (uint32_t)P.mk, (uint32_t)P.mk * 0x10001u);
                            if (!GLO) {
                                const uint32_t n = rn | __vcmpeq2(sel[k], 0x000E000Eu);
                                u = (u & ~n) | (((uint32_t)A.sc.match * 0x10001u) & n);
                            }
                            Dm = D[k] + P.m1 - u;
                        }
                        if (LOC) {
                            const uint32_t fl = P.fl[k + b];
                            uint32_t M;
                            if (TB) { /* exact values for the traceback */
                                M = FAST ? __vadd2(Dm, sv) : Dm;
                                H[k] = __vmaxs2(__vimax3_s16x2(M, F[k], E), fl);
                            } else { /* an M below 0 raised to 0: no H, and no gap that reaches one, changes */
                                M = FAST ? __viaddmax_s16x2(Dm, sv, fl) : __vmaxs2(Dm, fl);
                                H[k] = __vimax3_s16x2(M, F[k], E);
                            }
                            F[k] = __viaddmax_s16x2(M, P.no, F[k]);
                            E = __viaddmax_s16x2(M, P.no, E);
                            key[k] = mad_lo_u32(H[k], 4u, P.kk[k]);
                        } else if (GLO) {
                            const uint32_t M = Dm + sv;
                            H[k] = __vimax3_s16x2(M, F[k], E);
                            F[k] = __viaddmax_s16x2(F[k], P.be, M + P.tadd);
                            E = __viaddmax_s16x2(M, P.no, E);
                        } else {
                            const uint32_t mf = FAST ? __viaddmax_s16x2(Dm, sv, F[k]) : __vmaxs2(Dm, F[k]);
                            H[k] = __vmaxs2(mf, E);
                            F[k] = __viaddmax_s16x2(H[k], P.no, F[k]);
                            E = __viaddmax_s16x2(mf, P.no, E);
                        }
                    }
                    oH[b] = H[7] + P.ra;
                    oE[b] = E + P.ra;
                    D[0] = inH;
#pragma unroll
                    for (int k = 1; k < 8; k++) D[k] = H[k - 1];
                    if (LOC) {
                        cA[b] = __vmaxs2(__vimax3_s16x2(key[0], key[1], key[2]), key[3]);
                        cB[b] = __vmaxs2(__vimax3_s16x2(key[4], key[5], key[6]), key[7]);
                        bk = __viaddmax_s16x2(__vmaxs2(cA[b], cB[b]), P.kc[b], bk);
                    } else if (b == finb) {
#pragma unroll
                        for (int k = 0; k < 8; k++) hc[k] = H[k];
                    }
                }
#pragma unroll
                for (int k = 0; k < 8; k++) F[k] += P.rb, D[k] += P.rb, xw[k] = prmt(oH[k], oE[k], 0x7632u);
                if (multi) {
                    if (gl == G - 1 && wh >= 0 && on) {
                        uint4 *rp = reinterpret_cast<uint4 *>(ring + (wh << 3));
                        rp[0] = make_uint4(xw[0], xw[1], xw[2], xw[3]);
                        rp[1] = make_uint4(xw[4], xw[5], xw[6], xw[7]);
                    }
                    __syncwarp();
                }
                if (W > 1) {
                    const int x = s - (V - 1); /* the word the last virtual lane has done */
                    if (x >= 0 && x < wanted && on) {
                        if (wi < W - 1) {
                            bool late = false;
                            for (int spin = 0; taken + PK_FIFO <= x && !late;) { /* room in the fifo */
                                taken = cons[wi + 1];
                                late = ++spin > A.spins;
                            }
                            if (__any_sync(0xFFFFFFFFu, late)) {
                                ran_out();
                                wend = s;
                            }
                        }
                        if (gl == G - 1) {
                            uint4 *rp = reinterpret_cast<uint4 *>(
                                wi < W - 1 ? fifo + (wi * PK_FIFO + (x & (PK_FIFO - 1))) * 8 : ring + (wh << 3));
                            rp[0] = make_uint4(xw[0], xw[1], xw[2], xw[3]);
                            rp[1] = make_uint4(xw[4], xw[5], xw[6], xw[7]);
                            __threadfence_block();
                            prod[wi] = x + 1;
                        }
                    }
                }
                bool hit = false;
                if (LOC) {
                    const uint32_t m = __vmaxs2(bk, thr);
                    if (m != thr) {
                        if (live_lo && ((m ^ thr) & 0xFFFFu)) {
                            const int z = P.zero; /* keeps the arrays out of the registers */
#pragma unroll
                            for (int b = 0; b < 8; b++) keys_lo[z + b] = prmt(cA[b], cB[b], 0x5410u);
                            at_lo = (band_lo << 16) | w;
                            thr = set_half(thr, rev ? 0x7FFF : (int)(m | 3u), false);
                            hit = true;
                        }
                        if (live_hi && ((m ^ thr) & 0xFFFF0000u)) {
                            const int z = P.zero;
#pragma unroll
                            for (int b = 0; b < 8; b++) keys_hi[z + b] = prmt(cA[b], cB[b], 0x7632u);
                            at_hi = (band_hi << 16) | wh;
                            thr = set_half(thr, rev ? 0x7FFF : (int)((m >> 16) | 3u), true);
                            hit = true;
                        }
                    }
                } else if (finb < 8) {
                    if (GLO) {
                        const int k = (tlen - 1) & 7;
                        uint32_t v = hc[0];
#pragma unroll
                        for (int x = 1; x < 8; x++) v = x == k ? hc[x] : v;
                        score = half_of(v, fin_hi) - P.c0 - P.a * (k + 1) - P.b * (lastb + 1);
                        at_lo = 1;
                    } else {
                        /* rows in one basis; those past the target out of the running */
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            hc[k] -= (uint32_t)(P.a * k) * 0x10001u;
                            if (((T0 + band_lo) << 3) + k >= tlen) hc[k] &= 0xFFFF0000u;
                            if (((T0 + band_hi) << 3) + k >= tlen) hc[k] &= 0xFFFFu;
                        }
                        uint32_t m = __vimax3_s16x2(hc[0], hc[1], hc[2]);
                        m = __vimax3_s16x2(m, hc[3], hc[4]);
                        m = __vimax3_s16x2(m, hc[5], hc[6]);
                        m = __vmaxs2(m, hc[7]);
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const int v = half_of(m, h);
                            if ((h ? fin_hi && !hit_hi : fin_lo && !hit_lo) && v > half_of(thr, h)) {
                                int row = 0;
#pragma unroll
                                for (int k = 7; k >= 0; k--) row = half_of(hc[k], h) == v ? k : row;
                                row += (T0 + (h ? band_hi : band_lo)) << 3;
                                thr = set_half(thr, v, h);
                                const bool reached = rev && v - sbase >= score;
                                if (h) at_hi = row, hit_hi = reached;
                                else at_lo = row, hit_lo = reached;
                                hit |= reached;
                            }
                        }
                    }
                }
                if (rev) {
                    /* the first band (in sweep order) with a hit decides: the group is done when
                     * the virtual lanes before it have finished the round */
                    const unsigned m = __ballot_sync(0xFFFFFFFFu, hit);
                    if (m) {
                        int fin = 0x7fffffff;
                        if (hit) {
                            int bd = 0x7fffffff;
                            if (LOC) {
                                if (half_of(thr, false) == 0x7FFF && at_lo >= 0) bd = min(bd, at_lo >> 16);
                                if (half_of(thr, true) == 0x7FFF && at_hi >= 0) bd = min(bd, at_hi >> 16);
                            } else {
                                if (hit_lo) bd = min(bd, (at_lo >> 3) - T0);
                                if (hit_hi) bd = min(bd, (at_hi >> 3) - T0);
                            }
                            if (W > 1) atomicMin(const_cast<int *>(&s_stop), bd);
                            else if (bd != 0x7fffffff) fin = (bd / V) * per + per + (bd % V);
                        }
                        if (W == 1) {
#pragma unroll
                            for (int off = G / 2; off > 0; off >>= 1)
                                fin = min(fin, __shfl_xor_sync(0xFFFFFFFFu, fin, off));
                            gend = min(gend, max(fin, s + 1));
                            wend = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)gend);
                        }
                    }
                    if (W > 1 && __any_sync(0xFFFFFFFFu, stop_seen != 0x7fffffff)) {
                        const int bd = (int)__reduce_min_sync(0xFFFFFFFFu, (unsigned)stop_seen);
                        const int R = bd / (W * V), wb = bd / V - R * W, vb = bd % V;
                        int fin = R * per + V; /* the rounds before */
                        if (wi < wb) fin += per;
                        else if (wi == wb) fin = max(fin, R * per + per + vb);
                        gend = min(gend, max(fin, s + 1));
                        wend = min(wend, gend);
                    }
                }
                wh = w, rh = r;
                if (++w == per) w = 0, ++r;
                qp = qw, qw = qx;
            }
            };
            if (FAST && !GLO && with_n) sweep(std::true_type{});
            else sweep(std::false_type{});
            if (W > 1) { /* nobody waits for a warp that is done */
                __syncwarp();
                if (lane == 0) prod[wi] = 0x3fffffff, cons[wi] = 0x3fffffff;
            }

            /* the pair's result from its virtual lanes */
            if (GLO) {
                if (W > 1) {
                    if (at_lo == 1) s_res[0] = score;
                    __syncthreads();
                    score = s_res[0];
                } else {
                    const unsigned own = __ballot_sync(0xFFFFFFFFu, at_lo == 1) & gmask;
                    score = __shfl_sync(0xFFFFFFFFu, score, own ? __ffs((int)own) - 1 : lane);
                    if (!own) score = 0;
                }
            } else {
                unsigned best = 0;
                bool use_hi = false;
                const bool any_hit = SEM && rev && group_any(hit_lo || hit_hi);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int at = h ? at_hi : at_lo;
                    if (at < 0) continue;
                    unsigned kx;
                    if (LOC) {
                        const unsigned hv = rev ? 1u : (unsigned)half_of(thr, h) >> 2;
                        kx = (hv << 16) | (0xFFFFu - (unsigned)(at >> 16));
                    } else if (any_hit) {
                        if (!(h ? hit_hi : hit_lo)) continue;
                        kx = (1u << 16) | (0xFFFFu - (unsigned)at);
                    } else {
                        kx = ((unsigned)half_of(thr, h) << 16) | (0xFFFFu - (unsigned)at);
                    }
                    if (kx > best) best = kx, use_hi = h;
                }
                unsigned all = best;
#pragma unroll
                for (int off = G / 2; off > 0; off >>= 1) all = max(all, __shfl_xor_sync(0xFFFFFFFFu, all, off));
                if (W > 1) {
                    if (lane == 0) s_key[wi] = (int)all;
                    __syncthreads();
#pragma unroll
                    for (int x = 0; x < W; x++) all = max(all, (unsigned)s_key[x]);
                }
                const bool mine = all != 0 && best == all;
                const unsigned own = W > 1 ? all : __ballot_sync(0xFFFFFFFFu, mine) & gmask;
                const int src = W == 1 && own ? __ffs((int)own) - 1 : lane;
                int row = 0, col = 0, val = 0;
                if (LOC && mine) {
                    /* the block's first column reaching the value, its first row */
                    const int word = (use_hi ? at_hi : at_lo) & 0xFFFF, band = (use_hi ? at_hi : at_lo) >> 16;
                    val = rev ? score : half_of(thr, use_hi) >> 2;
                    const int z = P.zero;
                    int bb = 0, kr = 0;
                    for (int b = 7; b >= 0; b--) {
                        const uint32_t x = use_hi ? keys_hi[z + b] : keys_lo[z + b];
                        const int off = 4 * P.b * (b + 1);
                        const int xa = half_of(x, false) - off, xb = half_of(x, true) - off;
                        const bool up = (xa >> 2) >= (xb >> 2);
                        if (((up ? xa : xb) >> 2) >= val) bb = b, kr = up ? 3 - (xa & 3) : 7 - (xb & 3);
                    }
                    row = (band << 3) + kr, col = (word << 3) + bb;
                }
                if (SEM && mine) row = use_hi ? at_hi : at_lo, val = half_of(thr, use_hi) - sbase;
                if (W > 1) {
                    if (mine) s_res[0] = row, s_res[1] = col, s_res[2] = val;
                    __syncthreads();
                    row = s_res[0], col = s_res[1], val = s_res[2];
                } else {
                    row = __shfl_sync(0xFFFFFFFFu, row, src);
                    col = __shfl_sync(0xFFFFFFFFu, col, src);
                    val = __shfl_sync(0xFFFFFFFFu, val, src);
                }
                if (!rev) {
                    score = val, r_te = row, r_qe = LOC ? col : tlen;
                } else if (LOC) {
                    /* reversed coordinates -> what the reference records */
                    if (own) r_ts = (nb << 3) - 1 - ((row >> 3) << 3) + (row & 7), r_qs = (qn << 3) - 1 - col;
                } else if (work) {
                    r_ts = (tlen - 1) - row, r_qs = (qlen - 1) - tlen;
                }
            }
        }

        if (gl == 0 && wi == 0 && has) {
            if (A.score) A.score[i] = score;
            if (!GLO) {
                if (A.q_end) A.q_end[i] = r_qe;
                if (A.t_end) A.t_end[i] = r_te;
                if (START == WITH_START_) {
                    if (A.q_start) A.q_start[i] = r_qs;
                    if (A.t_start) A.t_start[i] = r_ts;
                }
            }
        }
    }
}

/* One launch over every class of pairs, longest first: a warp works through
 * the first class's pairs with that class's lane group, then the next's, so no
 * class has a tail of its own and a batch of mixed lengths fills the chip to
 * its end (launches per class, one after another or on two streams, left
 * 10,000 pairs of 50-1,000 bp at 3.1 ms).  A class of group 32 * W shares each
 * pair among the W warps of the block. */
template <int W, int ALGO, int START, bool FAST>
__global__ void __launch_bounds__(32 * W, 16 / W)
    dp_pk_kernel(const __grid_constant__ DpArgs A, const __grid_constant__ PkConst P,
                 const __grid_constant__ PkClasses C, const uint32_t *list)
{
    extern __shared__ __align__(16) uint32_t pk_smem[];
    __shared__ uint2 tab[FAST ? 256 : 1];
    if (FAST) {
        pk_score_table(tab, A.sc, ALGO != GLOBAL_, P.a + P.b);
        __syncthreads();
    }
    uint32_t *mem = pk_smem + (size_t)(threadIdx.x >> 5) * C.warp_words;
#pragma unroll 1
    for (int c = 0; c < C.n; c++) {
        const PkClass &k = C.k[c];
        const uint32_t *l = list ? list + k.first : nullptr;
        [[maybe_unused]] const int nl = k.n;
        uint32_t *qu = A.queue + c;
        if constexpr (!FAST) { /* what the table-scoring launch left: long pairs, then short ones */
            if (k.group == 32)
                pk_pairs<32, 1, ALGO, START, FAST>(A, P, tab, mem, l + (A.n - 1), (int)A.n_dev[1], qu, k.ring_cols,
                                                    k.max_q8, -1);
            else if (k.many > 0 && (int)A.n_dev[0] >= k.many)
                pk_pairs<1, 1, ALGO, START, FAST>(A, P, tab, mem, l, (int)A.n_dev[0], qu, k.ring_cols, k.max_q8);
            else if (k.many > 0 && 5ll * (int)A.n_dev[0] >= k.many)
                pk_pairs<2, 1, ALGO, START, FAST>(A, P, tab, mem, l, (int)A.n_dev[0], qu, k.ring_cols, k.max_q8);
            else
                pk_pairs<4, 1, ALGO, START, FAST>(A, P, tab, mem, l, (int)A.n_dev[0], qu, k.ring_cols, k.max_q8);
            continue;
        }
        switch (k.group) {
        case 1: pk_pairs<1, 1, ALGO, START, FAST>(A, P, tab, mem, l, nl, qu, k.ring_cols, k.max_q8); break;
        case 2: pk_pairs<2, 1, ALGO, START, FAST>(A, P, tab, mem, l, nl, qu, k.ring_cols, k.max_q8); break;
        case 4: pk_pairs<4, 1, ALGO, START, FAST>(A, P, tab, mem, l, nl, qu, k.ring_cols, k.max_q8); break;
        case 8: pk_pairs<8, 1, ALGO, START, FAST>(A, P, tab, mem, l, nl, qu, k.ring_cols, k.max_q8); break;
        case 16: pk_pairs<16, 1, ALGO, START, FAST>(A, P, tab, mem, l, nl, qu, k.ring_cols, k.max_q8); break;
        case 32: pk_pairs<32, 1, ALGO, START, FAST>(A, P, tab, mem, l, nl, qu, k.ring_cols, k.max_q8); break;
        default:
            if constexpr (W > 1)
                pk_pairs<32, W, ALGO, START, FAST>(A, P, tab, pk_smem, l, nl, qu, k.ring_cols, k.max_q8);
            __syncthreads(); /* the block's rings become its warps' */
        }
    }
}

template <int ALGO, int START> PkKernel pk_variant(PkVariant v)
{
    if (v == PK_CMP) return dp_pk_kernel<1, ALGO, START, false>;
    if (v == PK_W4) return dp_pk_kernel<4, ALGO, START, true>;
    if (v == PK_W2) return dp_pk_kernel<2, ALGO, START, true>;
    return dp_pk_kernel<1, ALGO, START, true>;
}

template <int ALGO> PkKernel pk_kernel(PkVariant v, int start)
{
    if (start == WITH_TB_ && ALGO != SEMI_GLOBAL_)
        return pk_variant<ALGO, ALGO == SEMI_GLOBAL_ ? WITHOUT_START_ : WITH_TB_>(v);
    if (start == WITH_START_ && ALGO != GLOBAL_)
        return pk_variant<ALGO, ALGO == GLOBAL_ ? WITHOUT_START_ : WITH_START_>(v);
    return pk_variant<ALGO, WITHOUT_START_>(v);
}

} // namespace
} // namespace gb

#endif
