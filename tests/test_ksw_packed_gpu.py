"""The packed ksw row kernel against the oracle, bit for bit: query lengths at
the edges of words, of one- and two-word tiles and of the length classes,
seeds at the edge of what it takes (larger ones go to the 32-bit kernels),
other codes, z-drop."""
import numpy as np
import pytest

from gasal_b200 import lib as gl
from gasal_b200.capi import Batch, Params, KSW
from oracle.bindings import oracle_align

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)
LENGTHS = (249, 255, 256, 257, 263, 264, 511, 512, 513, 519, 520, 767, 768, 1023, 1025, 2040, 2046, 2047, 2050, 4103,
           8190, 8191)


def _batch(rng, lens, h0, odd=b"", err=0.06, low=1):
    qs, ts = [], []
    for k, n in enumerate(lens):
        q = ACGT[rng.integers(0, 4, n)]
        t = q.copy()
        if k % 5 == 4:
            t = ACGT[rng.integers(0, 4, int(rng.integers(low, n + 40)))]
        else:
            m = rng.random(n) < err
            t[m] = ACGT[rng.integers(0, 4, int(m.sum()))]
            for _ in range(int(rng.integers(0, 4))):
                c = int(rng.integers(0, len(t)))
                t = np.delete(t, np.arange(c, min(len(t), c + 3))) if rng.random() < 0.5 else \
                    np.insert(t, c, ACGT[rng.integers(0, 4, 3)])
        for s in (q, t):
            for c in odd:
                if len(s):
                    s[rng.integers(0, len(s), max(1, len(s) // 60))] = c
        qs.append(q.tobytes())
        ts.append(t.tobytes())
    b = Batch.from_seqs(qs, ts)
    b.seed = np.asarray([h0[k % len(h0)] for k in range(len(lens))], dtype=np.uint32)
    return b


def _check(p, b):
    got, exp = gl.align(p, b).as_dict(p), oracle_align(p, b).as_dict(p)
    for k, v in exp.items():
        bad = np.nonzero(got[k] != v)[0]
        assert not len(bad), f"{p.key()} {k}: {len(bad)} differ, first {bad[:5]} (q {b.q_len[bad[:5]]}): " \
                             f"{got[k][bad[:5]]} want {v[bad[:5]]}"


@pytest.mark.parametrize("zdrop", [0, 100, 12])
@pytest.mark.parametrize("sc", [dict(), dict(match=3, mismatch=2, gap_open=5, gap_extend=2),
                                dict(match=2, mismatch=5, gap_open=0, gap_extend=1)], ids=["bwa", "m3", "o0"])
def test_tile_and_class_edges(zdrop, sc):
    rng = np.random.default_rng(zdrop + len(sc))
    lens = [n for n in LENGTHS for _ in range(3)]
    _check(Params(algo=KSW, zdrop=zdrop, **sc), _batch(rng, lens, (20, 60, 300, 7, 0)))


@pytest.mark.parametrize("h0", [5, 1500, 15800, 16200, 30000])
def test_seeds(h0):
    """Seeds with which the largest value times match + 1 fits 15 bits, is at
    its edge (16,383) and does not."""
    rng = np.random.default_rng(h0)
    _check(Params(algo=KSW, zdrop=100), _batch(rng, [int(n) for n in rng.integers(249, 600, 40)], (h0, h0 + 37)))


@pytest.mark.parametrize("odd", [b"N", b"NR"])
def test_other_codes(odd):
    rng = np.random.default_rng(len(odd))
    _check(Params(algo=KSW), _batch(rng, [int(n) for n in rng.integers(250, 1500, 60)], (40,), odd=odd))


def test_in_length_order():
    """A batch large enough for the length order, both lane-group and row
    kernels, high error rates (ranges that split and vanish)."""
    rng = np.random.default_rng(4)
    lens = np.exp(rng.normal(5.6, 0.7, 2100)).astype(int).clip(30, 2500)
    _check(Params(algo=KSW, zdrop=100), _batch(rng, [int(n) for n in lens], (20, 45, 60), err=0.2))
