"""The packed kernels at the edges of the values they accept: the longest pairs
whose scores stay within 15 bits and the first that do not, bytes after a
sequence's end that are bases (LOCAL scores them, as the reference does), and
the lowest values of GLOBAL and SEMI_GLOBAL; and as many pairs with other codes as
make compare scoring take two lanes each, or one.  Against the oracle."""
from dataclasses import replace

import numpy as np
import pytest

from gasal_b200 import lib as gl
from gasal_b200.capi import Batch, Params, LOCAL, GLOBAL, SEMI_GLOBAL, WITH_START, WITH_TB, TARGET, NONE, QUERY
from oracle.bindings import oracle_align

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)
MODES = [Params(algo=LOCAL), Params(algo=LOCAL, start_pos=WITH_START), Params(algo=LOCAL, start_pos=WITH_TB),
         Params(algo=GLOBAL), Params(algo=GLOBAL, start_pos=WITH_TB)] + \
        [Params(algo=SEMI_GLOBAL, head=h, tail=TARGET, start_pos=WITH_START) for h in (NONE, QUERY, TARGET)]


def _check(p, b, what):
    got, exp = gl.align(p, b).as_dict(p), oracle_align(p, b).as_dict(p)
    if "cigar" in exp and np.any(exp["n_cigar"] > (b.q_len + 7) // 8 * 8):
        got.pop("cigar"), exp.pop("cigar")  # a CIGAR longer than its slot runs into the next pair's
    for k, v in exp.items():
        bad = np.nonzero(got[k] != v)[0]
        assert not len(bad), f"{what} {k}: {len(bad)} differ, first {bad[:5]}: {got[k][bad[:5]]} want {v[bad[:5]]}"


def _equal_pairs(rng, n):
    """Pairs of equal sequences of n bases whose bytes up to the next multiple
    of 8 go on with equal bases too."""
    seqs = [ACGT[rng.integers(0, 4, (n + 7) // 8 * 8)] for _ in range(3)]
    b = Batch.from_seqs([s.tobytes() for s in seqs], [s.tobytes() for s in seqs])
    b.q_len[:] = n
    b.t_len[:] = n
    return b


@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
@pytest.mark.parametrize("match,lengths", [(50, range(153, 169)), (16, range(497, 514)), (59, range(265, 283)),
                                           (13, (617, 624, 625, 632))], ids=lambda v: v if isinstance(v, int) else "")
def test_highest_scores(p, match, lengths):
    """match * length crosses 8,183 (LOCAL) or about 16,200 (the others) among
    the lengths, by the bases counted or by those after the end."""
    rng = np.random.default_rng(match)
    for n in lengths:
        _check(replace(p, match=match), _equal_pairs(rng, n), f"{p.key()} match {match} length {n}")


@pytest.mark.parametrize("n", [8176, 8177])
def test_highest_scores_of_long_pairs(n):
    p = Params(algo=LOCAL)
    _check(p, _equal_pairs(np.random.default_rng(n), n), f"length {n}")


@pytest.mark.parametrize("p", [m for m in MODES if m.algo != LOCAL], ids=lambda p: p.key())
@pytest.mark.parametrize("e", [10, 2])
def test_lowest_scores(p, e):
    """Sequences with no base in common: gaps over all of both, down to the
    lowest value accepted and below it."""
    sc = dict(match=1, mismatch=10, gap_open=6, gap_extend=e)
    for t in {10: (990, 1008, 1013, 1016, 1017, 1030), 2: (6900, 7100, 7300, 7500, 7700)}[e]:
        for q in (1, 8, 500, 512, 513, 900):
            b = Batch.from_seqs([b"A" * q, b"C" * q], [b"C" * t, b"G" * t])
            _check(replace(p, **sc), b, f"{p.key()} {q} x {t}")


@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
@pytest.mark.parametrize("n,longest", [(8200, 128), (40400, 128), (40400, 129)])
def test_many_pairs_of_other_codes(p, n, longest):
    """Pairs whose targets hold R, a fifth of 272 on each of 148 SMs and as many
    as that, queries of 1 to 128 bases, or one of 129."""
    rng = np.random.default_rng(longest)
    w = 136
    q = ACGT[rng.integers(0, 4, (n, w))]
    t = q.copy()
    m = rng.random((n, w)) < 0.05
    t[m] = ACGT[rng.integers(0, 4, int(m.sum()))]
    t[:, 0] = ord("R")
    q[::7, 2] = ord("N")
    t[::5, 3] = ord("N")
    off = np.arange(n, dtype=np.uint32) * np.uint32(w)
    ql = rng.integers(1, 129, n).astype(np.uint32)
    tl = np.minimum(ql + rng.integers(0, 9, n).astype(np.uint32), 136)
    tl[::9] = rng.integers(1, 137, len(tl[::9]))
    ql[5] = longest
    for x, ln in ((q, ql), (t, tl)):
        x[np.arange(w)[None, :] >= ln[:, None]] = ord("N")
    _check(p, Batch(q.reshape(-1), t.reshape(-1), off, off.copy(), ql, tl), p.key())
