"""Inputs that are packed already (Parameters::isPacked): one query buffer holds
the 4-bit words and receives the CIGARs, so a traceback must not read a word
that a CIGAR has been written over.  Every operation byte, run count, score and
LOCAL start against the oracle, in one chunk and in several, through the C++
API and through gb_align_dev with the CIGAR buffer laid over the words."""
import os
import struct
import subprocess

import numpy as np
import pytest

from gasal_b200 import lib as gl
from gasal_b200 import workloads as W
from gasal_b200.capi import Params, LOCAL, GLOBAL, SEMI_GLOBAL, WITH_TB, TARGET
from oracle.bindings import oracle_align

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MODES = [Params(algo=LOCAL, start_pos=WITH_TB), Params(algo=GLOBAL, start_pos=WITH_TB),
         # mismatch < gap extend: GLOBAL tracebacks from direction tiles
         Params(algo=GLOBAL, start_pos=WITH_TB, mismatch=1, gap_open=3, gap_extend=2),
         Params(algo=SEMI_GLOBAL, start_pos=WITH_TB, head=TARGET, tail=TARGET)]

CALLER = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "gasal_header.h"
#include "gasal_b200_capi.h"

int main(int argc, char **argv)
{
    if (argc < 3) return 2;
    FILE *f = fopen(argv[1], "rb");
    int32_t h[11]; /* n, query and target bytes, algo, head, tail, scores, traceback budget in MB */
    if (!f || fread(h, 4, 11, f) != 11) return 2;
    const int n = h[0], qb = h[1], tb = h[2];
    std::vector<uint32_t> meta(4 * (size_t)n);
    std::vector<char> q(qb / 2), t(tb / 2);
    if (fread(meta.data(), 4, meta.size(), f) != meta.size() || fread(q.data(), 1, q.size(), f) != q.size() ||
        fread(t.data(), 1, t.size(), f) != t.size()) return 2;
    fclose(f);
    gb_set_tb_budget_mb(h[10]);
    gasal_subst_scores sc{};
    sc.match = h[6], sc.mismatch = h[7], sc.gap_open = h[8], sc.gap_extend = h[9];
    gasal_copy_subst_scores(&sc);
    Parameters p(0, nullptr);
    p.algo = (algo_type)h[3], p.start_pos = WITH_TB, p.isPacked = true;
    p.semiglobal_skipping_head = (data_source)h[4], p.semiglobal_skipping_tail = (data_source)h[5];
    gasal_gpu_storage_v v = gasal_init_gpu_storage_v(1);
    gasal_init_streams(&v, qb / n + 16, tb / n + 16, n, &p);
    gasal_gpu_storage_t *s = &v.a[0];
    FILE *o = fopen(argv[2], "wb");
    for (int rep = 0; rep < 2; rep++) { /* the second run replays the captured batch */
        gasal_host_batch_fill(s, 0, q.data(), (uint32_t)q.size(), QUERY);
        gasal_host_batch_fill(s, 0, t.data(), (uint32_t)t.size(), TARGET);
        memcpy(s->host_query_batch_offsets, &meta[0], 4 * n);
        memcpy(s->host_target_batch_offsets, &meta[n], 4 * n);
        memcpy(s->host_query_batch_lens, &meta[2 * n], 4 * n);
        memcpy(s->host_target_batch_lens, &meta[3 * n], 4 * n);
        gasal_aln_async(s, qb, tb, n, &p);
        while (gasal_is_aln_async_done(s) == -1) {}
        const gasal_res_t *r = s->host_res;
        fwrite(r->aln_score, 4, n, o);
        fwrite(r->n_cigar_ops, 4, n, o);
        std::vector<int32_t> zero(n);
        fwrite(r->query_batch_start ? r->query_batch_start : zero.data(), 4, n, o);
        fwrite(r->target_batch_start ? r->target_batch_start : zero.data(), 4, n, o);
        fwrite(r->cigar, 1, qb, o);
    }
    fclose(o);
    gasal_destroy_streams(&v, &p);
    gasal_destroy_gpu_storage_v(&v);
    return 0;
}
"""


def _pack(a):
    """ASCII -> 4-bit codes, the first of 8 in the top bits of a 32-bit word."""
    c = (a & 15).astype(np.uint32).reshape(-1, 8)
    w = np.zeros(c.shape[0], dtype=np.uint32)
    for k in range(8):
        w |= c[:, k] << np.uint32(28 - 4 * k)
    return w


def _ops(cigar, off, n):
    keep = np.zeros(len(cigar), dtype=bool)
    for o, k in zip(off.astype(np.int64), n.astype(np.int64)):
        keep[o:o + k] = True
    return cigar[keep]


def _compare(got, exp, b, what):
    for k, v in exp.items():
        if k == "cigar":
            assert np.array_equal(_ops(got[k], b.q_off, exp["n_cigar"]), _ops(v, b.q_off, exp["n_cigar"])), what + " cigar"
        elif k in got:
            bad = np.nonzero(np.asarray(got[k]).astype(np.int64) != v.astype(np.int64))[0]
            assert not len(bad), f"{what} {k}: {len(bad)} differ, first {bad[:5]}"


@pytest.fixture(scope="module")
def caller(tmp_path_factory):
    d = tmp_path_factory.mktemp("packed")
    src, exe = str(d / "caller.cpp"), str(d / "caller")
    with open(src, "w") as f:
        f.write(CALLER)
    so = os.path.dirname(gl.LIB_PATH)
    subprocess.run(["g++", "-O1", "-I", os.path.join(ROOT, "include"), "-I/usr/local/cuda/include", src, "-o", exe,
                    gl.LIB_PATH, "-L/usr/local/cuda/lib64", "-lcudart", f"-Wl,-rpath,{so}",
                    "-Wl,-rpath,/usr/local/cuda/lib64"], check=True)
    return exe


@pytest.mark.parametrize("mb", [98304, 1], ids=["one_chunk", "chunks"])
@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
def test_is_packed_storage(caller, tmp_path, p, mb):
    b = W.workload2(900, seed=31)
    exp = oracle_align(p, b).as_dict(p)
    nq, nt = int(b.q.shape[0]), int(b.t.shape[0])
    with open(tmp_path / "in", "wb") as f:
        f.write(struct.pack("<11i", b.n, nq, nt, p.algo, p.head, p.tail, p.match, p.mismatch, p.gap_open, p.gap_extend,
                            mb))
        for a in (b.q_off, b.t_off, b.q_len, b.t_len, _pack(b.q), _pack(b.t)):
            f.write(np.ascontiguousarray(a, dtype=np.uint32).tobytes())
    subprocess.run([caller, str(tmp_path / "in"), str(tmp_path / "out")], check=True, timeout=300)
    out = np.fromfile(tmp_path / "out", dtype=np.uint8)
    one = 16 * b.n + nq
    assert len(out) == 2 * one
    for rep in range(2):
        x = out[rep * one:(rep + 1) * one]
        words = x[:16 * b.n].view(np.int32).reshape(4, b.n)
        got = dict(score=words[0], n_cigar=words[1], cigar=x[16 * b.n:])
        if p.algo != GLOBAL:
            got.update(q_start=words[2], t_start=words[3])
        _compare(got, exp, b, f"{p.key()} run {rep}")


@pytest.mark.parametrize("mb", [98304, 1], ids=["one_chunk", "chunks"])
@pytest.mark.parametrize("over", ["q", "t"])
@pytest.mark.parametrize("p", MODES, ids=lambda p: p.key())
def test_cigar_buffer_over_the_words(p, over, mb):
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda", 0)
    b = W.workload2(900, seed=32)
    exp = oracle_align(p, b).as_dict(p)

    def up(a, dt=None):
        return torch.from_numpy(np.ascontiguousarray(a).view(dt or a.dtype)).to(dev)
    nq, nt = int(b.q.shape[0]), int(b.t.shape[0])
    keep = {"q": up(b.q), "t": up(b.t), "pq": torch.zeros(nq, dtype=torch.uint8, device=dev),
            "pt": torch.zeros(max(nq, nt), dtype=torch.uint8, device=dev)}
    for k in ("q_off", "t_off", "q_len", "t_len"):
        keep[k] = up(getattr(b, k), np.int32)
    outs = {k: torch.zeros(b.n, dtype=torch.int32, device=dev) for k in ("score", "q_end", "t_end", "q_start", "t_start",
                                                                         "n_cigar")}
    m = {"q_bytes": nq, "t_bytes": nt}
    m.update({k: v.data_ptr() for k, v in keep.items()})
    m.update({"out_" + k: v.data_ptr() for k, v in outs.items()})
    m["out_cigar"] = m["p" + over]
    gl.set_tb_budget_mb(mb)
    try:
        gl.align_dev(p, m, b.q_len, b.t_len, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    finally:
        gl.set_tb_budget_mb(98304)
    got = {k: v.cpu().numpy() for k, v in outs.items()}
    got["cigar"] = keep["p" + over].cpu().numpy()[:nq]
    _compare(got, exp, b, p.key())
