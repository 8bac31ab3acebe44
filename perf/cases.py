"""Timed cases of the alignment path: batches of sequence pairs through the
library's public entry points, from a handful of pairs to the mixed production
batch.

A case is a plain dict:
  shape   which generator workload the pairs come from (gasal_b200.workloads):
          0 short reads 100-150 bp, 1 150 bp reads on 150-300 bp windows (half
          flagged reverse-complement), 2 uneven 50-1000 bp, 3 seed extensions
          250-2000 bp, 4 production mix (log-normal, 50-5000 bp)
  algo, start, second, rc, zdrop, scores   the launch options
  n       pairs in the batch
  api     "dev": gb_align_dev on a batch already in device memory;
          "storage": the host staging + gasal_aln_async loop on host buffers
"""
import numpy as np
import torch

from gasal_b200 import lib as gl
from gasal_b200 import workloads as W
from gasal_b200.capi import (OUT_FIELDS, GLOBAL, KSW, LOCAL, SEMI_GLOBAL, TARGET, WITHOUT_START, WITH_START, WITH_TB,
                             Outputs, Params, has_cigar)

ALGOS = {"local": LOCAL, "global": GLOBAL, "semi": SEMI_GLOBAL, "ksw": KSW}
STARTS = {"none": WITHOUT_START, "start": WITH_START, "tb": WITH_TB}
# match, mismatch, gap open, gap extend: the library's defaults, and the other set its tests use
SCORES = {"default": (1, 4, 6, 1), "m2x3o5e2": (2, 3, 5, 2)}
# integer operations a DP cell cannot do without, per algorithm (+4 for a direction code)
CELL_OPS = {"local": 11, "global": 9, "semi": 10, "ksw": 13}


def _case(name, shape, algo, start, n, **kw):
    c = {"name": name, "shape": shape, "algo": algo, "start": start, "n": n, "second": 0, "rc": 0, "zdrop": 0,
         "scores": "default", "api": "dev"}
    c.update(kw)
    return c


def listed():
    return [
        # one read's candidate windows checked on their own: latency and launches
        _case("local_64", 0, "local", "start", 64),
        # the short-read set at its full size through the host staging loop GASAL2 callers run
        _case("local_20k_storage", 0, "local", "none", 20000, api="storage"),
        # a per-stream batch of the size a read mapper hands over (scores only)
        _case("global_5k", 1, "global", "start", 5000, rc=1),
        # read against window with the second-best hit for a mapping quality, half reverse-complemented
        _case("local_second_100k", 1, "local", "start", 100001, second=1, rc=1),
        # glocal read mapping, a large batch of equal short reads
        _case("semi_300k", 1, "semi", "start", 300000, rc=1),
        # few long reads: the work must spread within the pairs
        _case("local_long_1k", 3, "local", "start", 1000),
        # end-to-end alignments with CIGARs, uneven lengths
        _case("global_tb_100k", 2, "global", "tb", 100000),
        # seed extension of long reads
        _case("ksw_50k", 3, "ksw", "none", 50000),
        # the production mix's four launches
        _case("local_mix_200k", 4, "local", "start", 200000),
        _case("local_tb_mix_100k", 4, "local", "tb", 100000),
        _case("semi_mix_150k", 4, "semi", "start", 150000),
        _case("ksw_mix_200k", 4, "ksw", "none", 200000, zdrop=100),
    ]


# algorithm, start, shapes, and the most pairs a drawn batch of each shape has
_KINDS = [("local", "none"), ("local", "start"), ("local", "start"), ("local", "tb"), ("global", "start"),
          ("global", "tb"), ("semi", "start"), ("semi", "start"), ("ksw", "none"), ("ksw", "none")]
_MOST = {0: 300000, 1: 300000, 2: 100000, 3: 12000, 4: 90000}


def draw(rng):
    algo, start = _KINDS[rng.randrange(len(_KINDS))]
    shape = rng.choice((3, 4) if algo == "ksw" else (0, 1, 2, 3, 4))
    n = int(round(32 * (_MOST[shape] / 32) ** rng.random()))
    c = _case("", shape, algo, start, n)
    del c["name"]
    if algo in ("local", "semi") and start != "tb" and shape < 3:
        c["second"] = int(rng.random() < 0.3)
    c["rc"] = int(shape == 1)
    if algo == "ksw":
        c["zdrop"] = rng.choice((0, 100))
    c["scores"] = "m2x3o5e2" if rng.random() < 0.2 else "default"
    if shape == 0 and n <= 50000:
        c["api"] = rng.choice(("dev", "storage"))
    return c


def _params(case):
    m, x, o, e = SCORES[case["scores"]]
    return Params(algo=ALGOS[case["algo"]], start_pos=STARTS[case["start"]], second_best=case["second"], head=TARGET,
                  tail=TARGET, reverse_complement=case["rc"], zdrop=case["zdrop"], match=m, mismatch=x, gap_open=o,
                  gap_extend=e)


def _batch(case, seed):
    return W.generate(case["shape"], case["n"], seed)[0]


def _cigar_room(case):
    mean, most = {0: (130, 152), 1: (152, 152), 2: (325, 1000), 3: (1130, 2000), 4: (350, 5000)}[case["shape"]]
    return int(1.2 * mean * case["n"]) + 20 * most


def prepare(case, seed):
    p, b = _params(case), _batch(case, seed)
    if case["api"] == "storage":
        longest_q = max(int(b.q_len.max()), (b.q.shape[0] + b.n - 1) // b.n)
        longest_t = max(int(b.t_len.max()), (b.t.shape[0] + b.n - 1) // b.n)
        return {"p": p, "b": b, "streams": gl.Streams(1, longest_q, longest_t, b.n, p)}
    dev = torch.device("cuda", torch.cuda.current_device())

    def up(a, dtype=None):
        return torch.from_numpy(np.ascontiguousarray(a).view(dtype or a.dtype)).to(dev)

    t = {"q": up(b.q), "t": up(b.t), "pq": torch.zeros(b.q.shape[0] // 8, dtype=torch.int32, device=dev),
         "pt": torch.zeros(b.t.shape[0] // 8, dtype=torch.int32, device=dev)}
    for k in ("q_off", "t_off", "q_len", "t_len"):
        t[k] = up(getattr(b, k), np.int32)
    for k in ("q_op", "t_op"):
        if getattr(b, k) is not None:
            t[k] = up(getattr(b, k))
    if b.seed is not None:
        t["seed"] = up(b.seed, np.int32)
    outs = {k: torch.zeros(b.n, dtype=torch.int32, device=dev) for k in Outputs.fields_for(None, p)}
    if has_cigar(p):
        # a buffer with room for any batch of this many pairs, as a caller that reuses it has
        outs["cigar"] = torch.zeros(_cigar_room(case), dtype=torch.uint8, device=dev)
        outs["n_cigar"] = torch.zeros(b.n, dtype=torch.int32, device=dev)
    m = {"q_bytes": b.q.shape[0], "t_bytes": b.t.shape[0]}
    m.update({k: v.data_ptr() for k, v in t.items()})
    m.update({"out_" + k: v.data_ptr() for k, v in outs.items()})
    return {"p": p, "b": b, "t": t, "outs": outs, "m": m}


def run(state):
    p, b = state["p"], state["b"]
    if "streams" in state:
        s = state["streams"]
        qb, tb = s.fill_bulk(0, b)
        s.aln_async(0, qb, tb, b.n)
        s.wait(0)
        return s.results(0, b.n, b)
    gl.align_dev(p, state["m"], b.q_len, b.t_len, torch.cuda.current_stream().cuda_stream)
    return state["outs"]


def work(case):
    """Every base and pair entry read once, every result written once; one
    DP over the whole matrix (ksw: what trimming leaves is data dependent)."""
    b = _lengths(case)
    p = _params(case)
    outs = len(Outputs.fields_for(None, p)) + (1 if has_cigar(p) else 0)
    cells = int(W.pair_cells(case["shape"], case["n"], 0).sum())
    ops = CELL_OPS[case["algo"]] + (4 if case["start"] == "tb" else 0)
    return {"bytes": b + case["n"] * (16 + 4 * outs), "flops": cells * ops}


def _lengths(case):
    b = _batch(case, 0)
    return int(b.q_len.sum()) + int(b.t_len.sum())


def exact(case, seed):
    """The scores of small LOCAL and GLOBAL batches by a plain 64-bit DP over
    all pairs at once (gaps open from an aligned pair only, N scores 0 in
    LOCAL); every other output is a position in, or a path through, the same
    matrix."""
    if case["algo"] not in ("local", "global") or case["rc"] or case["shape"] != 0:
        return None
    p, b = _params(case), _batch(case, seed)
    if b.n * int(b.q_len.max()) * int(b.t_len.max()) > 5e8:
        return None
    m, x, o, e = SCORES[case["scores"]]
    local = case["algo"] == "local"
    nq, nt, n = int(b.q_len.max()), int(b.t_len.max()), b.n

    def grid(buf, off, ln, width):
        a = np.zeros((width, n), np.uint8)
        for j in range(width):
            live = j < ln
            a[j, live] = buf[off[live].astype(np.int64) + j]
        return a

    q, t = grid(b.q, b.q_off, b.q_len, nq), grid(b.t, b.t_off, b.t_len, nt)
    low = np.int64(-1 << 40)
    score = np.zeros(n, np.int64)
    edge = lambda k: np.int64(0 if local or k == 0 else -(o + e * (k - 1)))  # boundary cell k steps from the corner
    H = np.stack([np.full(n, edge(j)) for j in range(nq + 1)])
    E = np.full((nq + 1, n), low)
    if not local:
        H[1] = 0
        for j in range(2, nq + 1):
            H[j] = -(o + e * (j - 1))
    for i in range(nt):
        diag = np.zeros(n, np.int64) if local or i == 0 else np.full(n, np.int64(-(o + e * i)))
        F = np.full(n, low)
        for j in range(nq):
            s = np.where(q[j] == t[i], m, -x).astype(np.int64)
            if local:
                s[(q[j] == 0x4E) | (t[i] == 0x4E)] = 0
            M = diag + s
            best = np.maximum(np.maximum(M, F), E[j + 1])
            if local:
                best = np.maximum(best, 0)
                live = (i < b.t_len) & (j < b.q_len)
                score = np.where(live, np.maximum(score, best), score)
            else:
                last = (i == b.t_len - 1) & (j == b.q_len - 1)
                score = np.where(last, best, score)
            F = np.maximum(F - e, M - o - e)
            E[j + 1] = np.maximum(E[j + 1] - e, M - o - e)
            diag = H[j + 1].copy()
            H[j + 1] = best
    names = list(Outputs.fields_for(None, p)) + (["n_cigar", "cigar"] if has_cigar(p) else [])
    return {k: score if k == "score" else None for k in names}
