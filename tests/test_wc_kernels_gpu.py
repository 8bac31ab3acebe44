"""The kernels behind the packed ones: score sets just outside the packed range
(mismatch 61, or GLOBAL with mismatch < gap extend) on batches of 2,048+ pairs
run the warp-cooperative kernels without a second best -- table and compare
scoring, direction tiles, start passes -- and the one-thread kernel beside
them; and the checkpoint walk with one thread to every pair."""
import os
import subprocess
import sys

import numpy as np
import pytest

from gasal_b200 import lib as gl
from gasal_b200.capi import Batch, Params, KSW, LOCAL, GLOBAL, SEMI_GLOBAL, WITH_START, WITH_TB, NONE, QUERY, TARGET, BOTH
from oracle.bindings import oracle_align

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)
FAR = dict(match=2, mismatch=61, gap_open=6, gap_extend=1)
LOW = dict(match=2, mismatch=1, gap_open=4, gap_extend=2)
MODES = [Params(algo=LOCAL, **FAR), Params(algo=LOCAL, start_pos=WITH_START, **FAR),
         Params(algo=LOCAL, start_pos=WITH_TB, **FAR), Params(algo=GLOBAL, **LOW),
         Params(algo=GLOBAL, start_pos=WITH_TB, **LOW)] + \
        [Params(algo=SEMI_GLOBAL, head=h, tail=TARGET, start_pos=s, **FAR) for h, s in
         ((NONE, 0), (QUERY, WITH_START), (TARGET, WITH_START), (BOTH, 0))]


def _batch(rng, odd):
    """2,090 pairs: short ones, queries around 32 and 127 words, targets of a
    few bases, and (odd) a fifth with other codes than A, C, G, T."""
    lens = np.concatenate([rng.integers(20, 249, 700), rng.integers(249, 420, 1300),
                           [249, 256, 257, 1008, 1009, 1016, 1017, 1500], rng.integers(1009, 1300, 82)])
    qs, ts = [], []
    for k, n in enumerate(int(x) for x in rng.permutation(lens)):
        q = ACGT[rng.integers(0, 4, n)]
        t = q.copy()
        m = rng.random(n) < 0.04
        t[m] = ACGT[rng.integers(0, 4, int(m.sum()))]
        c = int(rng.integers(0, n))
        t = np.concatenate([t[:c], ACGT[rng.integers(0, 4, int(rng.integers(0, 4)))], t[c:]])
        if k % 50 == 7:
            t = t[:int(rng.integers(1, 9))]
        if odd and k % 5 == 0:
            q[int(rng.integers(0, n))] = ord("R") if k % 2 else ord("N")
            t[int(rng.integers(0, len(t)))] = ord("N") if k % 3 else ord("Y")
        qs.append(q.tobytes())
        ts.append(t.tobytes())
    return Batch.from_seqs(qs, ts)


@pytest.mark.parametrize("group", [0, 8, 16, 32, 64])
@pytest.mark.parametrize("odd", [False, True], ids=["acgt", "other"])
@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
def test_wc_kernels_without_second_best(p, odd, group):
    b = _batch(np.random.default_rng(group + 2 * p.algo + odd), odd)
    saved = gl.get_tuning()
    try:
        gl.set_tuning(wc_group=group, wc_min_qregs=group or 32)
        got = gl.align(p, b).as_dict(p)
    finally:
        gl.set_tuning(**saved)
    exp = oracle_align(p, b).as_dict(p)
    if "cigar" in exp and np.any(exp["n_cigar"] > (b.q_len + 7) // 8 * 8):
        got.pop("cigar"), exp.pop("cigar")  # a CIGAR longer than its slot runs into the next pair's
    for k, v in exp.items():
        bad = np.nonzero(got[k] != v)[0]
        assert not len(bad), f"{p.key()} {k}: {len(bad)} differ, first {bad[:5]} (q {b.q_len[bad[:5]]})"


WALKS = """
import os, sys
sys.path[:0] = [sys.argv[1], os.path.join(sys.argv[1], "tests")]
import test_packed_gpu as T
from gasal_b200.capi import WITH_TB
for p in T.MODES:
    if p.start_pos == WITH_TB:
        T.test_edges_of_words_bands_and_rounds(p, 0)
        for odd in (b"N", b"NR", b"Nn", b"RYK"):
            T.test_other_codes(p, odd)
        for sc in T.SCORES:
            T.test_score_sets(p, sc)
        T.test_mixed_lengths_in_order(p)
        T.test_few_long_pairs(p, 9)
"""


@pytest.mark.parametrize("coop", [-1, 0, 40])
def test_checkpoint_walks_by_lanes_per_pair(coop):
    """The traceback tests of the packed kernels with one thread to every pair,
    to all but the queries of 127+ words, and with 40 pairs on 8 lanes."""
    r = subprocess.run([sys.executable, "-c", WALKS, ROOT], env=dict(os.environ, GASAL_B200_TB_COOP=str(coop)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("n", [3, 60, 2100])
def test_ksw_batches_of_short_queries_only(n):
    """Queries of at most 31 words alone: the lane groups take the whole list,
    ordered or not, and hand seeds beyond 16 bits to the one-thread kernel."""
    rng = np.random.default_rng(n)
    qs = [ACGT[rng.integers(0, 4, int(k))] for k in rng.integers(1, 249, n)]
    ts = [np.concatenate([q[:int(rng.integers(0, len(q) + 1))], ACGT[rng.integers(0, 4, int(rng.integers(0, 60)))]])
          for q in qs]
    b = Batch.from_seqs([q.tobytes() for q in qs], [t.tobytes() for t in ts])
    b.seed = rng.integers(0, 100, n).astype(np.uint32)
    b.seed[::3] = 33000
    p = Params(algo=KSW, zdrop=50)
    got, exp = gl.align(p, b).as_dict(p), oracle_align(p, b).as_dict(p)
    for k, v in exp.items():
        bad = np.nonzero(got[k] != v)[0]
        assert not len(bad), f"{k}: {len(bad)} differ, first {bad[:5]} (q {b.q_len[bad[:5]]})"
