"""The packed (two 8-row bands per lane, int16x2) kernels against the oracle,
bit for bit: sizes at the edges of words, bands, lane groups and rounds, codes
that take the N select or the compare-scoring kernel, score sets at the edge
of what the packed kernels accept, and the checkpoint traceback."""
from dataclasses import replace

import numpy as np
import pytest

from gasal_b200 import lib as gl
from gasal_b200.capi import (Batch, Params, LOCAL, GLOBAL, SEMI_GLOBAL, WITH_START, WITH_TB, NONE, QUERY, TARGET, BOTH)
from oracle.bindings import oracle_align

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)
MODES = [Params(algo=LOCAL), Params(algo=LOCAL, start_pos=WITH_START), Params(algo=LOCAL, start_pos=WITH_TB),
         Params(algo=GLOBAL), Params(algo=GLOBAL, start_pos=WITH_TB)] + \
        [Params(algo=SEMI_GLOBAL, head=h, tail=TARGET, start_pos=s) for h in (NONE, QUERY, TARGET, BOTH)
         for s in (0, WITH_START)]


@pytest.fixture(autouse=True)
def _settings():
    gl.set_reference_max_query_len(2048)
    yield
    gl.set_tuning(wc_group=0)


def _pair(rng, qlen, tlen, related=True, odd=b""):
    q = ACGT[rng.integers(0, 4, qlen)]
    if related:  # the query with 5% substitutions and one gap, inside (or cut to) the target
        s = q.copy()
        m = rng.random(qlen) < 0.05
        s[m] = ACGT[rng.integers(0, 4, int(m.sum()))]
        c = qlen // 2
        s = np.concatenate([s[:c], ACGT[rng.integers(0, 4, 3)], s[c:]])
        lead = max(0, (tlen - len(s)) // 2)
        t = np.concatenate([ACGT[rng.integers(0, 4, lead)], s, ACGT[rng.integers(0, 4, max(tlen, 1))]])[:tlen]
    else:
        t = ACGT[rng.integers(0, 4, tlen)]
    t = t.copy()
    for seq in (q, t):
        for c in odd:
            if len(seq):
                seq[rng.integers(0, len(seq), max(1, len(seq) // 40))] = c
    return q.tobytes(), t.tobytes()


def _batch(rng, sizes, **kw):
    pairs = [_pair(rng, q, t, related=k % 3 != 2, **kw) for k, (q, t) in enumerate(sizes)]
    return Batch.from_seqs([q for q, _ in pairs], [t for _, t in pairs])


def _check(p, b):
    got, exp = gl.align(p, b).as_dict(p), oracle_align(p, b).as_dict(p)
    if "cigar" in exp:
        # a CIGAR longer than its query slot runs into the next pair's (undefined in the reference)
        room = (b.q_len + 7) & ~np.uint32(7)
        if np.any(exp["n_cigar"] > room):
            got.pop("cigar"), exp.pop("cigar")
    for k, v in exp.items():
        bad = np.nonzero(got[k] != v)[0]
        assert not len(bad), f"{p.key()} {k}: {len(bad)} differ, first {bad[:5]}: {got[k][bad[:5]]} want {v[bad[:5]]}"


@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
@pytest.mark.parametrize("group", [0, 8, 16, 32, 64])
def test_edges_of_words_bands_and_rounds(p, group):
    """Query words and target bands one below, at and one above the virtual
    lanes of every group, and single bases."""
    rng = np.random.default_rng(group + 100 * p.algo + p.start_pos)
    words = (1, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33)
    sizes = [(8 * w - int(rng.integers(0, 8)), 8 * n - int(rng.integers(0, 8)))
             for w in words for n in (1, 4, 5, 8, 9, 16, 17, 32, 33, 65)]
    sizes += [(1, 1), (1, 30), (30, 1), (8, 8), (9, 16), (520, 1100), (1023, 1030), (1017, 2100)]
    gl.set_tuning(wc_group=group)
    _check(p, _batch(rng, sizes))


@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
@pytest.mark.parametrize("odd", [b"N", b"NR", b"Nn", b"RYK"], ids=["N", "N+R", "N+n", "IUPAC"])
def test_other_codes(p, odd):
    rng = np.random.default_rng(len(odd) + 7 * p.algo)
    sizes = [(int(q), int(q) + int(d)) for q, d in zip(rng.integers(5, 300, 90), rng.integers(-4, 60, 90))]
    _check(p, _batch(rng, sizes + [(511, 530), (512, 520), (1300, 1200), (900, 2100), (2000, 2050)], odd=odd))


SCORES = [dict(match=2, mismatch=3, gap_open=5, gap_extend=2), dict(match=1, mismatch=1, gap_open=0, gap_extend=1),
          dict(match=5, mismatch=4, gap_open=10, gap_extend=0), dict(match=60, mismatch=60, gap_open=100, gap_extend=30),
          dict(match=0, mismatch=0, gap_open=0, gap_extend=0), dict(match=61, mismatch=4, gap_open=6, gap_extend=1),
          dict(match=1, mismatch=0, gap_open=3, gap_extend=2)]


@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
@pytest.mark.parametrize("sc", SCORES, ids=lambda s: "x".join(str(v) for v in s.values()))
def test_score_sets(p, sc):
    rng = np.random.default_rng(sum(sc.values()) + p.algo)
    sizes = [(int(a), int(b)) for a, b in zip(rng.integers(1, 260, 100), rng.integers(1, 300, 100))]
    _check(replace(p, **sc), _batch(rng, sizes))


@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
def test_mixed_lengths_in_order(p):
    """A batch large enough for the length order: every class, empty
    sequences among them."""
    rng = np.random.default_rng(5 + p.algo)
    q = np.exp(rng.normal(5.0, 0.9, 2200)).astype(int).clip(1, 1500)
    sizes = [(int(a), int(a) + int(d)) for a, d in zip(q, rng.integers(0, 40, 2200))]
    b = _batch(rng, sizes)
    if p.algo == LOCAL:  # (the other modes' results on empty sequences are this library's own: 0)
        b.q_len[[3, 700]] = 0
        b.t_len[[4, 700]] = 0
    _check(p, b)


@pytest.mark.parametrize("p", [m for m in MODES if m.algo == LOCAL], ids=lambda p: p.key())
def test_scores_beyond_the_packed_range(p):
    """match 10 on 1,100-base queries: those leave the packed LOCAL range and
    run warp-cooperative beside the packed classes; at match 7 they fit."""
    rng = np.random.default_rng(9)
    sizes = [(int(a), int(a) + 12) for a in rng.integers(40, 160, 2100)] + [(1100, 1130), (1017, 1016), (1150, 1300)]
    b = _batch(rng, sizes)
    for match in (7, 10):
        _check(replace(p, match=match, mismatch=8, gap_open=12, gap_extend=2), b)


@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
@pytest.mark.parametrize("n", [1, 9, 40])
def test_few_long_pairs(p, n):
    """Too few pairs to fill the GPU: several warps share a pair, one round
    and more, among them queries narrower than the handover between warps
    and targets that end in each of the group's warps."""
    rng = np.random.default_rng(n + 10 * p.algo)
    tl = [9000, 530, 1030, 2100, 4200, 600, 3000, 8200, 70]
    sizes = [(int(rng.integers(1, 2500)) if k % 4 else 100 + k, tl[k % len(tl)] - int(rng.integers(0, 8)))
             for k in range(n)]
    sizes[0] = (2300, 9000)
    _check(p, _batch(rng, sizes))
