/*
 * tb_kernel.cu -- tracebacks into GASAL2's CIGAR bytes.
 *
 * Replaces reference src/kernels/get_tb.h:4-149.  traceback_kernel walks the
 * direction tiles of the one-thread and warp-cooperative kernels, one thread per
 * pair; traceback_points_kernel walks the packed kernels' checkpoints, one thread
 * per pair or eight to the longest.  Output format: one byte per run, (count << 2) | op
 * with op 0 match, 1 mismatch, 2 deletion (consumes target), 3 insertion
 * (consumes query), count <= 63, written last operation first at the pair's
 * query offset of the device query batch; the run count replaces nothing else
 * (n_cigar is written to its own array).  LOCAL starts at the end cell and
 * stops once the operations re-score to the alignment score, reporting the
 * start; GLOBAL starts at (target length, query length) -- one past the last
 * cell, as the reference does -- and flushes leftover target / query bases as
 * 63-long runs.  The state machine (normal mode reads the 2 direction bits,
 * gap mode reads the extend bit of the gap's kind) is the reference's.
 * Target-tail SEMI_GLOBAL (an extension) has its own walk, semi_walk.
 */
#include "gb_internal.h"

namespace gb {

/* Run-length CIGAR writer: runs of one operation up to 63 long, last
 * operation first, bytes past `room` counted but not written. */
struct CigarOut {
    uint8_t *out;
    uint32_t room, n = 0, op = 0;
    int count = 0;
    __device__ __forceinline__ void put(uint32_t o)
    {
        if (count > 0 && count < 63 && o == op) {
            count++;
            return;
        }
        flush();
        op = o, count = 1;
    }
    __device__ __forceinline__ void flush()
    {
        if (count > 0) {
            if (n < room) out[n] = (uint8_t)(op | ((uint32_t)count << 2));
            n++;
        }
        count = 0;
    }
};

/* SEMI_GLOBAL traceback, an extension (the reference instantiates semi-global
 * WITH_TB empty, semiglobal_kernel_template.h:227), for a free target tail:
 * from the end cell (t_end, qlen - 1), an affine state machine over the
 * nibbles of semi_nib -- in H the two low bits give the move (diagonal, or
 * enter E / F at the same cell), in E (deletion) and F (insertion) the
 * cell's own extend bit says whether the gap continues or was opened from H
 * of the cell it came from.  At a free leading edge (target for head TARGET
 * or BOTH, query for QUERY or BOTH) the walk stops; at a closed one the
 * remaining bases become one gap.  Starts: the first aligned target row and
 * query column. */
__device__ uint32_t semi_walk(const uint4 *tb, int q8, int i, int j, int head, uint8_t *out, uint32_t room,
                              int *si, int *sj)
{
    CigarOut c{out, room};
    int state = 0; /* 0 H, 2 E (deletion), 3 F (insertion) */
    while (i >= 0 && j >= 0) {
        const int cell = (((i >> 3) * q8) << 3) + (j << 3) + (i & 7);
        const uint4 tile = tb[cell >> 5];
        const int in_tile = cell & 31, reg = in_tile >> 3;
        const uint32_t word = reg == 0 ? tile.x : (reg == 1 ? tile.y : (reg == 2 ? tile.z : tile.w));
        const uint32_t nib = (word >> (28 - ((in_tile & 7) << 2))) & 15u;
        if (state == 0) {
            const uint32_t src = nib & 3u;
            if (src <= 1) {
                c.put(src);
                i--, j--;
                continue;
            }
            state = (int)src;
        }
        if (state == 2) {
            c.put(2);
            state = (nib & 4u) ? 2 : 0;
            i--;
        } else {
            c.put(3);
            state = (nib & 8u) ? 3 : 0;
            j--;
        }
    }
    const bool free_t = head == TARGET_ || head == BOTH_, free_q = head == QUERY_ || head == BOTH_;
    int ts = i + 1, qs = j + 1;
    if (j < 0 && i >= 0 && !free_t) {
        for (; i >= 0; i--) c.put(2);
        ts = 0;
    }
    if (i < 0 && j >= 0 && !free_q) {
        for (; j >= 0; j--) c.put(3);
        qs = 0;
    }
    c.flush();
    *si = ts, *sj = qs;
    return c.n;
}

__global__ void __launch_bounds__(128) traceback_kernel(TbArgs a)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n || (a.kind && a.kind[p])) return;
    const int qlen = (int)a.q_len[p], tlen = (int)a.t_len[p];
    uint32_t n_ops = 0;
    if (a.algo == SEMI_GLOBAL_) {
        int si = 0, sj = 0;
        if (qlen > 0 && tlen > 0) {
            const uint32_t room = a.q_off[p] < a.cigar_bytes ? a.cigar_bytes - a.q_off[p] : 0u;
            n_ops = semi_walk(a.tb + a.tb_off[p], ((qlen + 7) >> 3) << 3, a.t_end[p], qlen - 1, a.head,
                              a.cigar + a.q_off[p], room, &si, &sj);
        }
        if (a.t_start) a.t_start[p] = si;
        if (a.q_start) a.q_start[p] = sj;
        if (a.n_cigar) a.n_cigar[p] = n_ops;
        return;
    }
    if (qlen > 0 && tlen > 0) {
        const uint4 *tb = a.tb + a.tb_off[p];
        const int q8 = ((qlen + 7) >> 3) << 3;
        int i, j, total = 0;
        if (a.algo == LOCAL_) {
            i = a.t_end[p], j = a.q_end[p], total = a.score[p];
        } else {
            i = tlen, j = qlen;
        }
        uint8_t *out = a.cigar + a.q_off[p];
        const uint32_t room = a.q_off[p] < a.cigar_bytes ? a.cigar_bytes - a.q_off[p] : 0u;
        uint32_t prev_op = 0, op_fill;
        int prev_tile = -1, op_select = 3, op_shift = 0, count = 0, curr = 0;
        uint4 tile = make_uint4(0, 0, 0, 0);
        while (i >= 0 && j >= 0) {
            const int cell = (((i >> 3) * q8) << 3) + (j << 3) + (i & 7);
            const int tile_no = cell >> 5;
            if (tile_no != prev_tile) tile = tb[tile_no];
            prev_tile = tile_no;
            const int in_tile = cell & 31;
            const int reg = in_tile >> 3;
            const uint32_t word = reg == 0 ? tile.x : (reg == 1 ? tile.y : (reg == 2 ? tile.z : tile.w));
            const uint32_t nib = (word >> (28 - ((in_tile & 7) << 2))) & 15u;
            const uint32_t op = (nib >> op_shift) & (uint32_t)op_select;
            op_fill = (op == 0 || op_select == 3) ? op : (uint32_t)op_shift;
            op_select = (op == 0 || (op == 1 && op_select == 3)) ? 3 : 1;
            op_shift = (op == 0 || (op == 1 && op_select == 3)) ? 0 : ((op == 2 || op == 3) ? (int)op : op_shift);
            if (count < 63 && op_fill == prev_op) {
                count++;
            } else {
                if (count > 0) {
                    if (n_ops < room) out[n_ops] = (uint8_t)(prev_op | ((uint32_t)count << 2));
                    n_ops++;
                }
                count = 1;
            }
            if (a.algo == LOCAL_) {
                const bool gap = (op_fill == 2 || op_fill == 3);
                curr += (gap && prev_op != op_fill) ? -a.sc.oe
                                                    : (gap ? -a.sc.e : (op_fill == 1 ? -a.sc.mismatch : a.sc.match));
                if (curr == total) break;
            }
            prev_op = op_fill;
            if (op_fill == 0 || op_fill == 1 || op_fill == 2) i--;
            if (op_fill == 0 || op_fill == 1 || op_fill == 3) j--;
        }
        if (n_ops < room) out[n_ops] = (uint8_t)(prev_op | ((uint32_t)count << 2));
        n_ops++;
        if (a.algo == GLOBAL_) {
            for (; i >= 0; i -= 63, n_ops++)
                if (n_ops < room) out[n_ops] = (uint8_t)(2u | ((uint32_t)min(i + 1, 63) << 2));
            for (; j >= 0; j -= 63, n_ops++)
                if (n_ops < room) out[n_ops] = (uint8_t)(3u | ((uint32_t)min(j + 1, 63) << 2));
        }
        if (a.algo == LOCAL_) {
            if (a.t_start) a.t_start[p] = i;
            if (a.q_start) a.q_start[p] = j;
        }
    } else if (a.algo == LOCAL_) {
        /* an empty query or target: no operations and start 0, like every
         * other result of such a pair (nothing else writes the starts) */
        if (a.t_start) a.t_start[p] = 0;
        if (a.q_start) a.q_start[p] = 0;
    }
    if (a.n_cigar) a.n_cigar[p] = n_ops;
}

/* Traceback from the packed kernels' checkpoints (LOCAL, GLOBAL).  The
 * forward sweep writes no direction code per cell (a dozen integer operations
 * on top of a cell's five to nine): it leaves H and E entering every 16th row
 * and D and F entering every 16th column (0.5 B per cell, as the tiles), and
 * the walk recomputes the 16 x 16 blocks its path crosses, each from its own
 * exact borders -- about 32 cells per base of the path instead of a code for
 * every cell of the matrix.
 *
 * Most pairs take one thread: the warp alternates between recomputing every
 * lane's block and walking every lane to its block's edge, so the lanes stay
 * together.  That is the least work, but a 5,000-base path is 600 blocks of
 * some 5,700 instructions in a row (8.0 of the 16.1 ms of 100k mixed LOCAL
 * pairs).  So the longest pairs -- the first `coop` of the length order -- take
 * 8 lanes each: a lane has two rows of the block and runs one column behind
 * the lane above (that batch, sweep included: 16.7 to 12.4 ms). */
constexpr int TBP_THREADS = 64;

/* the walk's state (the reference's machine, src/kernels/get_tb.h:74-117) */
template <bool LOC> struct PointWalk {
    int i, j, total, curr = 0, count = 0, op_select = 3, op_shift = 0;
    uint32_t n_ops = 0, prev_op = 0, room;
    uint8_t *out;
    bool done;
    __device__ __forceinline__ bool on() const { return !done && i >= 0 && j >= 0; }
    __device__ __forceinline__ void step(uint32_t nib, const Scores &sc)
    {
        const uint32_t op = (nib >> op_shift) & (uint32_t)op_select;
        const uint32_t op_fill = (op == 0 || op_select == 3) ? op : (uint32_t)op_shift;
        const bool normal = op == 0 || (op == 1 && op_select == 3);
        op_shift = normal ? 0 : ((op == 2 || op == 3) ? (int)op : op_shift);
        op_select = normal ? 3 : 1;
        if (count < 63 && op_fill == prev_op) {
            count++;
        } else {
            if (count > 0) {
                if (n_ops < room) out[n_ops] = (uint8_t)(prev_op | ((uint32_t)count << 2));
                n_ops++;
            }
            count = 1;
        }
        if (LOC) {
            const bool gap = (op_fill == 2 || op_fill == 3);
            curr += (gap && prev_op != op_fill) ? -sc.oe : (gap ? -sc.e : (op_fill == 1 ? -sc.mismatch : sc.match));
            if (curr == total) {
                done = true;
                return;
            }
        }
        prev_op = op_fill;
        if (op_fill != 3) i--;
        if (op_fill != 2) j--;
    }
    __device__ __forceinline__ void finish()
    {
        if (n_ops < room) out[n_ops] = (uint8_t)(prev_op | ((uint32_t)count << 2));
        n_ops++;
        if constexpr (!LOC) {
            for (; i >= 0; i -= 63, n_ops++)
                if (n_ops < room) out[n_ops] = (uint8_t)(2u | ((uint32_t)min(i + 1, 63) << 2));
            for (; j >= 0; j -= 63, n_ops++)
                if (n_ops < room) out[n_ops] = (uint8_t)(3u | ((uint32_t)min(j + 1, 63) << 2));
        }
    }
};

/* one cell of a recomputed block: its direction nibble, H to `h` */
template <bool LOC>
__device__ __forceinline__ uint32_t point_cell(int diag, int &F, int &E, uint32_t qc, uint32_t tc, const Scores &sc, int &h)
{
    int s = qc == tc ? sc.match : -sc.mismatch;
    if (LOC && (qc == 14u || tc == 14u)) s = 0;
    const int M = diag + s;
    int H = max(max(M, F), E);
    if (LOC) H = max(H, 0);
    uint32_t d = (H == M) ? (M >= diag ? 0u : 1u) : (H == F ? 3u : 2u);
    const int t0 = M - sc.oe;
    d |= t0 > F - sc.e ? 0u : 8u;
    d |= t0 > E - sc.e ? 0u : 4u;
    F = max(F - sc.e, t0);
    E = max(E - sc.e, t0);
    h = H;
    return d;
}

template <bool LOC> __global__ void __launch_bounds__(TBP_THREADS) traceback_points_kernel(TbArgs a, int coop)
{
    constexpr int CL = 8; /* lanes of a cooperative pair */
    __shared__ uint2 nibs[16][TBP_THREADS];
    const int coop_blocks = (coop * CL + TBP_THREADS - 1) / TBP_THREADS;
    const bool shared_walk = (int)blockIdx.x < coop_blocks;
    const int tid = threadIdx.x, lane = tid & 31, gl = lane & (CL - 1);
    const int slot = shared_walk ? ((int)blockIdx.x * TBP_THREADS + tid) / CL
                                 : coop + ((int)blockIdx.x - coop_blocks) * TBP_THREADS + tid;
    const int col = shared_walk ? tid / CL : tid; /* this pair's column of nibs */
    int p = 0;
    bool have = slot < (shared_walk ? coop : a.n);
    if (have) {
        p = a.order ? (int)a.order[slot] : slot;
        have = a.kind[p] == 1;
    }
    int qlen = 0, tlen = 0;
    if (have) qlen = (int)a.q_len[p], tlen = (int)a.t_len[p];
    const bool real = have && qlen > 0 && tlen > 0;
    const int qregs = (qlen + 7) >> 3, tregs = (tlen + 7) >> 3, q8 = qregs << 3, t8 = tregs << 3;
    const uint32_t *tops = nullptr, *lefts = nullptr, *qw = nullptr, *tw = nullptr;
    PointWalk<LOC> w;
    w.i = w.j = -1, w.total = 0, w.room = 0, w.out = nullptr, w.done = !real;
    if (real) {
        tops = reinterpret_cast<const uint32_t *>(a.tb + a.tb_off[p]);
        lefts = tops + (size_t)((tregs + 1) >> 1) * q8;
        qw = a.pq + (a.q_off[p] >> 3), tw = a.pt + (a.t_off[p] >> 3);
        if (LOC) w.i = a.t_end[p], w.j = a.q_end[p], w.total = a.score[p];
        else w.i = tlen, w.j = qlen;
        w.out = a.cigar + a.q_off[p];
        w.room = a.q_off[p] < a.cigar_bytes ? a.cigar_bytes - a.q_off[p] : 0u;
        if (shared_walk && gl != 0) w.room = 0; /* every lane walks, the first writes */
    }
    const Scores sc = a.sc;
    while (__any_sync(0xFFFFFFFFu, w.on())) {
        const bool on = w.on();
        const int bi = w.i >> 4, bj = w.j >> 4;
        const bool in = on && w.i < t8 && w.j < q8;
        /* recompute the block's rows down to the walk's */
        if (__any_sync(0xFFFFFFFFu, in)) {
            const int rows = in ? (w.i & 15) + 1 : 0;
            uint32_t qa = 0, qb = 0;
            const bool two = in && 2 * bj + 1 < qregs;
            if (in) qa = qw[2 * bj];
            if (two) qb = qw[2 * bj + 1];
            if (shared_walk) {
                /* lane gl: rows 2gl and 2gl + 1, column s - gl at step s */
                const int r0 = 2 * gl;
                int diag0 = 0, diag1 = 0, F0 = 0, F1 = 0;
                uint32_t t0 = 0, t1 = 0, top0 = 0, top1 = 0;
                if (in) {
                    const uint2 tp = gl < 4 || two
                                         ? *reinterpret_cast<const uint2 *>(tops + (size_t)bi * q8 + (bj << 4) + 2 * gl)
                                         : make_uint2(0, 0);
                    top0 = tp.x, top1 = tp.y;
                    if ((bi << 4) + r0 < t8) {
                        const uint2 l = *reinterpret_cast<const uint2 *>(lefts + (size_t)bj * t8 + (bi << 4) + r0);
                        const int off = a.c0 + a.pa * (r0 & 7);
                        diag0 = (int)(l.x & 0xFFFFu) - off, F0 = (int)(l.x >> 16) - off - a.pa - a.pb;
                        diag1 = (int)(l.y & 0xFFFFu) - off - a.pa, F1 = (int)(l.y >> 16) - off - 2 * a.pa - a.pb;
                        const uint32_t x = tw[2 * bi + (r0 >> 3)];
                        t0 = (x >> (28 - 4 * (r0 & 7))) & 15u, t1 = (x >> (24 - 4 * (r0 & 7))) & 15u;
                    }
                }
                uint32_t n0l = 0, n0h = 0, n1l = 0, n1h = 0;
                int hb = 0, eb = 0; /* H and E leaving this lane's rows at its last column */
                for (int s = 0; s < 16 + CL - 1; s++) {
                    const int c = s - gl;
                    /* the row above, column c: the lane above's last step, or the block's top */
                    const uint32_t tx = __shfl_sync(0xFFFFFFFFu, top0, (lane & ~(CL - 1)) + ((s >> 1) & (CL - 1)));
                    const uint32_t ty = __shfl_sync(0xFFFFFFFFu, top1, (lane & ~(CL - 1)) + ((s >> 1) & (CL - 1)));
                    int hu = __shfl_up_sync(0xFFFFFFFFu, hb, 1, CL), E = __shfl_up_sync(0xFFFFFFFFu, eb, 1, CL);
                    if (gl == 0) {
                        const uint32_t x = (s & 1) ? ty : tx;
                        const int off = a.c0 + a.pb * ((s & 7) + 1);
                        hu = (int)(x & 0xFFFFu) - off, E = (int)(x >> 16) - off - a.pa;
                    }
                    if (c >= 0 && c < 16) {
                        const uint32_t qc = ((c < 8 ? qa : qb) >> (28 - 4 * (c & 7))) & 15u;
                        int h0, h1;
                        const uint32_t d0 = point_cell<LOC>(diag0, F0, E, qc, t0, sc, h0);
                        const uint32_t d1 = point_cell<LOC>(diag1, F1, E, qc, t1, sc, h1);
                        diag0 = hu, diag1 = h0, hb = h1, eb = E;
                        const uint32_t sh = 4 * (c & 7);
                        if (c < 8) n0l |= d0 << sh, n1l |= d1 << sh;
                        else n0h |= d0 << sh, n1h |= d1 << sh;
                    }
                }
                nibs[r0][col] = make_uint2(n0l, n0h);
                nibs[r0 + 1][col] = make_uint2(n1l, n1h);
                __syncwarp();
            } else {
                int Hup[16], E[16];
                if (in) {
                    const uint4 *t4 = reinterpret_cast<const uint4 *>(tops + (size_t)bi * q8 + (bj << 4));
#pragma unroll
                    for (int g = 0; g < 4; g++) {
                        const uint4 v = g < 2 || two ? t4[g] : make_uint4(0, 0, 0, 0);
                        const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const int c = 4 * g + u, off = a.c0 + a.pb * ((c & 7) + 1);
                            Hup[c] = (int)(x[u] & 0xFFFFu) - off;
                            E[c] = (int)(x[u] >> 16) - off - a.pa;
                        }
                    }
                }
                const uint32_t *lf = lefts + (size_t)bj * t8 + (bi << 4);
                for (int r = 0; r < 16; r++) {
                    if (!__any_sync(0xFFFFFFFFu, r < rows)) break;
                    if (r < rows) {
                        const uint32_t l = lf[r];
                        const int off = a.c0 + a.pa * (r & 7);
                        int diag = (int)(l & 0xFFFFu) - off, F = (int)(l >> 16) - off - a.pa - a.pb;
                        const uint32_t tc = (tw[2 * bi + (r >> 3)] >> (28 - 4 * (r & 7))) & 15u;
                        uint32_t lo = 0, hi = 0;
#pragma unroll
                        for (int c = 0; c < 16; c++) {
                            const uint32_t qc = ((c < 8 ? qa : qb) >> (28 - 4 * (c & 7))) & 15u;
                            int H;
                            const uint32_t d = point_cell<LOC>(diag, F, E[c], qc, tc, sc, H);
                            if (c < 8) lo |= d << (4 * c);
                            else hi |= d << (4 * (c - 8));
                            diag = Hup[c];
                            Hup[c] = H;
                        }
                        nibs[r][col] = make_uint2(lo, hi);
                    }
                }
            }
        }
        /* walk to the block's edge; a cell past the matrix (GLOBAL's first)
         * reads 0, and the block that its successor lies in comes next */
        bool go = on;
        while (go) {
            uint32_t nib = 0;
            if (in) {
                const uint2 x = nibs[w.i & 15][col];
                nib = ((w.j & 8 ? x.y : x.x) >> (4 * (w.j & 7))) & 15u;
            }
            w.step(nib, sc);
            go = in && w.on() && (w.i >> 4) == bi && (w.j >> 4) == bj;
        }
        __syncwarp();
    }
    if (!have || (shared_walk && gl != 0)) return;
    if (real) w.finish();
    if (LOC) {
        if (a.t_start) a.t_start[p] = real ? w.i : 0;
        if (a.q_start) a.q_start[p] = real ? w.j : 0;
    }
    if (a.n_cigar) a.n_cigar[p] = w.n_ops;
}

cudaError_t launch_traceback_points(const TbArgs &a, int coop, cudaStream_t s)
{
    if (a.n <= 0) return cudaSuccess;
    coop = coop < a.n ? coop : a.n;
    const int blocks = (coop * 8 + TBP_THREADS - 1) / TBP_THREADS + (a.n - coop + TBP_THREADS - 1) / TBP_THREADS;
    if (a.algo == LOCAL_) traceback_points_kernel<true><<<blocks, TBP_THREADS, 0, s>>>(a, coop);
    else traceback_points_kernel<false><<<blocks, TBP_THREADS, 0, s>>>(a, coop);
    return cudaGetLastError();
}

cudaError_t launch_traceback(const TbArgs &a, cudaStream_t s)
{
    if (a.n <= 0) return cudaSuccess;
    traceback_kernel<<<(a.n + 127) / 128, 128, 0, s>>>(a);
    return cudaGetLastError();
}

} // namespace gb
