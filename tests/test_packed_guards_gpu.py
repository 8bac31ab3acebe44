"""What the packed kernels do when the host's word does not hold: a query longer
than the host copy of the lengths is left unwritten, the others are right."""
import os

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
