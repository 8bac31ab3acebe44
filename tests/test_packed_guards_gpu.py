"""The packed kernels' guards: a query longer than the host copy of the lengths
is left unwritten, the others are right; a wait between the warps of a pair that
runs out ends the sweep and is reported, and the next batch is right again."""
import os
import subprocess
import sys

import numpy as np
import pytest

from gasal_b200 import lib as gl
from gasal_b200.capi import Batch, Params, LOCAL, GLOBAL, SEMI_GLOBAL, WITH_START, WITH_TB, TARGET
from oracle.bindings import oracle_align

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)
FIELDS = ("score", "q_end", "t_end", "q_start", "t_start", "n_cigar")


def device_batch(torch, b):
    dev = torch.device("cuda", 0)

    def up(a, dt=None):
        return torch.from_numpy(np.ascontiguousarray(a).view(dt or a.dtype)).to(dev)
    keep = {"q": up(b.q), "t": up(b.t), "pq": torch.zeros(b.q.shape[0] // 8, dtype=torch.int32, device=dev),
            "pt": torch.zeros(b.t.shape[0] // 8, dtype=torch.int32, device=dev)}
    for k in ("q_off", "t_off", "q_len", "t_len"):
        keep[k] = up(getattr(b, k), np.int32)
    outs = {k: torch.full((b.n,), -7, dtype=torch.int32, device=dev) for k in FIELDS}
    outs["cigar"] = torch.zeros(b.q.shape[0], dtype=torch.uint8, device=dev)
    m = {"q_bytes": b.q.shape[0], "t_bytes": b.t.shape[0]}
    m.update({k: v.data_ptr() for k, v in keep.items()})
    m.update({"out_" + k: v.data_ptr() for k, v in outs.items()})
    return m, keep, outs


@pytest.mark.parametrize("p", [Params(algo=LOCAL, start_pos=WITH_START), Params(algo=LOCAL, start_pos=WITH_TB),
                               Params(algo=GLOBAL), Params(algo=GLOBAL, start_pos=WITH_TB),
                               Params(algo=SEMI_GLOBAL, head=TARGET, tail=TARGET, start_pos=WITH_START)],
                         ids=lambda p: p.key())
@pytest.mark.parametrize("odd", [b"", b"R"], ids=["table", "compare"])
def test_query_longer_than_the_host_lengths(p, odd):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(p.algo)
    lens = [100] * 40
    lens[17] = 2000
    q = [ACGT[rng.integers(0, 4, n)].tobytes() for n in lens]
    b = Batch.from_seqs(q, [odd + x[len(odd):] for x in q])
    m, keep, outs = device_batch(torch, b)
    h_q_len = b.q_len.copy()
    h_q_len[17] = 100
    gl.align_dev(p, m, h_q_len, b.t_len, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    others = np.arange(b.n) != 17
    for k, v in oracle_align(p, b).as_dict(p).items():
        if k == "cigar":
            continue
        got = outs[k].cpu().numpy()
        assert np.array_equal(got[others].astype(np.int64), v[others].astype(np.int64)), k
        assert got[17] == -7, k


WAITS = r"""
import os, sys
sys.path[:0] = [sys.argv[1], os.path.join(sys.argv[1], "tests")]
import numpy as np, torch
from gasal_b200 import lib as gl
from gasal_b200.capi import Batch, Params, LOCAL, GLOBAL, SEMI_GLOBAL, WITH_START, WITH_TB, TARGET
from oracle.bindings import oracle_align
from test_packed_guards_gpu import device_batch, ACGT

rng = np.random.default_rng(3)
def batch(n, lens):
    q = [ACGT[rng.integers(0, 4, lens)].tobytes() for _ in range(n)]
    return Batch.from_seqs(q, q)
few_long, short = batch(2, 4000), batch(200, 100)
s = torch.cuda.current_stream().cuda_stream
for p in (Params(algo=LOCAL, start_pos=WITH_START), Params(algo=LOCAL, start_pos=WITH_TB), Params(algo=GLOBAL),
          Params(algo=SEMI_GLOBAL, head=TARGET, tail=TARGET, start_pos=WITH_START)):
    def dev(b):
        m, keep, outs = device_batch(torch, b)
        gl.align_dev(p, m, b.q_len, b.t_len, s)
        torch.cuda.synchronize()
        return {k: v.cpu().numpy() for k, v in outs.items()}
    def right(b):
        got = dev(b)
        for k, v in oracle_align(p, b).as_dict(p).items():
            if k != "cigar":
                assert np.array_equal(got[k].astype(np.int64), v.astype(np.int64)), (p.key(), k)
    right(short)
    dev(few_long)            # accepted: the wait runs out on the device
    try:
        right(short)
        sys.exit("the next call did not report it")
    except gl.GasalError:
        pass
    right(short)             # reported once
    dev(few_long)
    try:
        gl.release_workspaces()
        sys.exit("release did not report it")
    except gl.GasalError:
        pass
    right(short)
    try:
        gl.align(p, few_long)
        sys.exit("gb_align did not report it")
    except gl.GasalError:
        pass
    with gl.Streams(1, 4000, 4000, 200, p) as st:
        for b, ok in ((few_long, False), (short, True)):
            qi, ti = st.fill(0, b)
            st.aln_async(0, qi, ti, b.n)
            try:
                st.wait(0)
                assert ok, "gasal_is_aln_async_done did not report it"
            except gl.GasalError:
                assert not ok
print("REPORTED")
"""


def test_wait_that_runs_out_is_reported():
    """With no poll allowed, the first wait of a pair swept by several warps
    runs out; every entry point reports it and works again afterwards."""
    r = subprocess.run([sys.executable, "-c", WAITS, ROOT], env=dict(os.environ, GASAL_B200_WAIT_SPINS="0"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "REPORTED" in r.stdout, (r.stdout[-500:], r.stderr[-2000:])
