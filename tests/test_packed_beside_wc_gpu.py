"""Batches whose long pairs leave the packed kernels' range and run
warp-cooperative beside them, and a warp-cooperative threshold above the 127
words at which the length order stops sorting by query length: every pair is
swept by a launch whose buffers were sized for it.  Against the oracle."""
import numpy as np
import pytest

from gasal_b200 import lib as gl
from gasal_b200.capi import Batch, Params, LOCAL, GLOBAL, SEMI_GLOBAL, WITH_START, WITH_TB, TARGET, QUERY
from oracle.bindings import oracle_align

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)
BIG = dict(match=16, mismatch=8, gap_open=12, gap_extend=2)  # 1,024 matches are beyond 15 bits, 160 are not
MODES = [Params(algo=LOCAL, start_pos=WITH_START, **BIG), Params(algo=LOCAL, start_pos=WITH_TB, **BIG),
         Params(algo=GLOBAL, **BIG), Params(algo=GLOBAL, start_pos=WITH_TB, **BIG),
         Params(algo=SEMI_GLOBAL, head=TARGET, tail=TARGET, start_pos=WITH_START, **BIG),
         Params(algo=SEMI_GLOBAL, head=QUERY, tail=TARGET, **BIG),
         # no packed kernel at all
         Params(algo=LOCAL, start_pos=WITH_START, second_best=1),
         Params(algo=SEMI_GLOBAL, head=TARGET, tail=TARGET, start_pos=WITH_START, second_best=1)]


def _batch(rng):
    """2,100 short pairs; queries of 127 to 199 words, one of them with the
    batch's longest target, and of 200 words and more."""
    sizes = [(int(n), int(n) + int(d)) for n, d in zip(rng.integers(40, 161, 2100), rng.integers(-8, 30, 2100))]
    sizes += [(1009, 6500), (1040, 1100), (1592, 1600), (1599, 900), (1600, 1700), (1750, 1760), (1024, 1030),
              (1100, 3000)]
    qs, ts = [], []
    for q, t in sizes:
        s = ACGT[rng.integers(0, 4, q)]
        x = np.concatenate([s, ACGT[rng.integers(0, 4, max(0, t - q))]])[:t]
        m = rng.random(len(x)) < 0.06
        x[m] = ACGT[rng.integers(0, 4, int(m.sum()))]
        qs.append(s.tobytes())
        ts.append(x.tobytes())
    o = rng.permutation(len(qs))
    return Batch.from_seqs([qs[k] for k in o], [ts[k] for k in o])


@pytest.mark.parametrize("words", [32, 200])
@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
def test_long_pairs_beside_the_packed_ones(p, words):
    b = _batch(np.random.default_rng(words + p.algo))
    saved = gl.get_tuning()
    try:
        gl.set_tuning(wc_min_qregs=words)
        got = gl.align(p, b).as_dict(p)
    finally:
        gl.set_tuning(**saved)
    exp = oracle_align(p, b).as_dict(p)
    if "cigar" in exp and np.any(exp["n_cigar"] > (b.q_len + 7) // 8 * 8):
        got.pop("cigar"), exp.pop("cigar")  # a CIGAR longer than its slot runs into the next pair's
    for k, v in exp.items():
        bad = np.nonzero(got[k] != v)[0]
        assert not len(bad), f"{p.key()} {k}: {len(bad)} differ, first {bad[:5]} (q {b.q_len[bad[:5]]})"
