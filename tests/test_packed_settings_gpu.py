"""Settings around the packed kernels: every lane group that can be forced gives
the oracle's results, the warp-cooperative kernels' lane group leaves packed
batches alone, the autotuner tries only what the batch's route uses, and a
storage's graph is replayed for batches that differ in nothing the launches
depend on; and what the host spends on a large batch of short pairs."""
import os
import subprocess
import sys
import time

import numpy as np
import pytest

from gasal_b200 import lib as gl
from gasal_b200 import workloads as W
from gasal_b200.capi import Batch, Params, LOCAL, SEMI_GLOBAL, WITH_START, TARGET
from oracle.bindings import oracle_align

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SEMI = Params(algo=SEMI_GLOBAL, start_pos=WITH_START, head=TARGET, tail=TARGET)


def _device(torch, p, b):
    dev = torch.device("cuda", 0)

    def up(a, dt=None):
        return torch.from_numpy(np.ascontiguousarray(a).view(dt or a.dtype)).to(dev)
    keep = {"q": up(b.q), "t": up(b.t), "pq": torch.zeros(b.q.shape[0] // 8, dtype=torch.int32, device=dev),
            "pt": torch.zeros(b.t.shape[0] // 8, dtype=torch.int32, device=dev)}
    for k in ("q_off", "t_off", "q_len", "t_len"):
        keep[k] = up(getattr(b, k), np.int32)
    outs = {k: torch.zeros(b.n, dtype=torch.int32, device=dev) for k in ("score", "q_end", "t_end", "q_start", "t_start")}
    m = {"q_bytes": b.q.shape[0], "t_bytes": b.t.shape[0]}
    m.update({k: v.data_ptr() for k, v in keep.items()})
    m.update({"out_" + k: v.data_ptr() for k, v in outs.items()})
    return m, keep, outs


FORCED = """
import os, sys
sys.path[:0] = [sys.argv[1], os.path.join(sys.argv[1], "tests")]
import test_packed_gpu as T
for p in T.MODES:
    T.test_edges_of_words_bands_and_rounds(p, 0)
    T.test_few_long_pairs(p, 9)
    T.test_mixed_lengths_in_order(p)
"""


@pytest.mark.parametrize("group", [1, 2, 4, 8, 16, 32, 64, 128])
def test_forced_lane_groups(group):
    """The edge shapes, a few long pairs and the ordered mix of the packed
    kernels' tests on at least `group` lanes per pair."""
    r = subprocess.run([sys.executable, "-c", FORCED, ROOT], env=dict(os.environ, GASAL_B200_PK_GROUP=str(group)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_warp_cooperative_group_leaves_short_reads_alone():
    """100,000 short reads take the same time with any wc_group (while it
    forced the packed kernels' lanes too, 32 cost them six times as much)."""
    torch = pytest.importorskip("torch")
    b = W.workload0(100000, seed=5)
    m, keep, outs = _device(torch, SEMI, b)
    s = torch.cuda.current_stream().cuda_stream
    ms = {}
    saved = gl.get_tuning()
    try:
        for g in (0, 32):
            gl.set_tuning(wc_group=g)
            for _ in range(3):
                gl.align_dev(SEMI, m, b.q_len, b.t_len, s)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(10):
                gl.align_dev(SEMI, m, b.q_len, b.t_len, s)
            e1.record()
            torch.cuda.synchronize()
            ms[g] = e0.elapsed_time(e1)
    finally:
        gl.set_tuning(**saved)
    assert ms[32] < 2 * ms[0], ms


def test_autotune_of_a_packed_batch_keeps_the_settings():
    torch = pytest.importorskip("torch")
    p = Params(algo=LOCAL, start_pos=WITH_START)
    b = W.workload2(3000, seed=6)
    m, keep, outs = _device(torch, p, b)
    saved = gl.get_tuning()
    try:
        best = gl.autotune(p, m, b.q_len, b.t_len, torch.cuda.current_stream().cuda_stream, reps=1)
        torch.cuda.synchronize()
        assert best["ms"] > 0
        assert gl.get_tuning() == saved
        for k, v in oracle_align(p, b).as_dict(p).items():
            assert np.array_equal(outs[k].cpu().numpy(), v), k
    finally:
        gl.set_tuning(**saved)

def test_graph_replayed_for_an_unordered_batch_of_other_lengths():
    """Fewer pairs than the length order takes, of nearly equal lengths: one
    launch whatever their classes, so the same bytes and pairs replay the
    graph."""
    rng = np.random.default_rng(7)
    p = Params(algo=LOCAL, start_pos=WITH_START)

    def batch(lens):
        q = [rng.choice(np.frombuffer(b"ACGT", np.uint8), n).tobytes() for n in lens]
        return Batch.from_seqs(q, [(x + b"ACGTTGCA" * 20)[:160] for x in q])
    a, b = batch([120] * 50 + [128] * 50), batch([112] + [120] * 48 + [128] * 51)
    assert a.q.shape == b.q.shape and a.t.shape == b.t.shape
    gl.set_graphs(True)
    with gl.Streams(1, 160, 160, 100, p) as st:
        seen = []
        for x in (a, b):
            s0 = gl.graph_stats()
            qi, ti = st.fill_fast(0, x)
            st.aln_async(0, qi, ti, x.n)
            st.wait(0)
            got = st.results(0, x.n, x)
            for k, v in oracle_align(p, x).as_dict(p).items():
                assert np.array_equal(got[k], v), k
            seen.append({k: v - s0[k] for k, v in gl.graph_stats().items()})
    assert seen[0]["instantiated"] == 1 and seen[1]["relaunched"] == 1, seen


def test_host_time_of_many_short_pairs():
    """Planning 300,000 pairs of one class costs the host no more than twice the
    plain form's (a look at each pair cost four times as much and set the time
    of the call)."""
    torch = pytest.importorskip("torch")
    p = Params(algo=LOCAL)
    rng = np.random.default_rng(8)
    n, w = 300000, 40
    seqs = rng.choice(np.frombuffer(b"ACGT", np.uint8), n * w)
    off, ln = np.arange(n, dtype=np.uint32) * np.uint32(w), np.full(n, w, np.uint32)
    b = Batch(seqs, seqs.copy(), off, off.copy(), ln, ln.copy())
    m, keep, outs = _device(torch, p, b)
    s = torch.cuda.current_stream().cuda_stream
    saved, best = gl.get_tuning(), {}
    try:
        for persistent in (1, 0):
            gl.set_tuning(persistent=persistent)
            ts = []
            for _ in range(12):
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                gl.align_dev(p, m, b.q_len, b.t_len, s)
                ts.append(time.perf_counter() - t0)
            best[persistent] = min(ts[2:])
    finally:
        gl.set_tuning(**saved)
    assert best[1] < 2 * best[0], best


def test_many_short_queries_of_other_codes_keep_the_plain_forms_time():
    """100,000 pairs of 20-base queries whose targets hold R: compare scoring
    on four lanes each took twice the plain form's time."""
    torch = pytest.importorskip("torch")
    p = Params(algo=LOCAL)
    rng = np.random.default_rng(9)
    n, q, t = 100000, 24, 1000
    qs, ts = (rng.choice(np.frombuffer(b"ACGT", np.uint8), (n, w)) for w in (q, t))
    ts[:, 0] = ord("R")
    off = np.arange(n, dtype=np.uint32)
    b = Batch(qs.reshape(-1), ts.reshape(-1), off * np.uint32(q), off * np.uint32(t), np.full(n, 20, np.uint32),
              np.full(n, t, np.uint32))
    m, keep, outs = _device(torch, p, b)
    s = torch.cuda.current_stream().cuda_stream
    saved, ms = gl.get_tuning(), {}
    try:
        for persistent in (1, 0):
            gl.set_tuning(persistent=persistent)
            for _ in range(3):
                gl.align_dev(p, m, b.q_len, b.t_len, s)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(5):
                gl.align_dev(p, m, b.q_len, b.t_len, s)
            e1.record()
            torch.cuda.synchronize()
            ms[persistent] = e0.elapsed_time(e1)
    finally:
        gl.set_tuning(**saved)
    assert ms[1] < 1.4 * ms[0], ms
