"""The bounded wait between the strips of a job.  With the limit cut to a few cycles the wait runs
out: the call fails with the reason through the batch API, device buffers and the request queue (no
fault, no hang: the strips run to their end and the launch ends), the jobs concerned carry status
-3 without a CIGAR, and with the default limit back the same engine aligns the batch exactly."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from protlocus_b200 import lib as L
from protlocus_b200 import workload as W
from protlocus_b200.abi import NS_F_CIGAR, Options

pytestmark = pytest.mark.gpu

INT32_MIN = -(1 << 31)


def _jobs(rng, n):
    jobs = []
    for _ in range(n):
        aa = W.random_protein(rng, int(rng.integers(40, 120))).encode()
        nt = W.build_gene(rng, aa.decode(), divergence=0.2, n_frameshift=1, intron_lengths=[90]).encode()
        nt += W.random_dna(rng, 3000).encode()
        jobs += [(nt, aa), (W.revcomp(nt), aa)]
    jobs.append((nt[:150], aa))  # a single strip: waits for nothing
    return jobs


def _device(lib, eng, opt, jobs):
    """Return code, and (score, n_cigar, status) of every job, through device buffers."""
    tab, nt, aa, at = (L.SpliceJob * len(jobs))(), b"", b"", {}
    for q, (n, a) in enumerate(jobs):
        if a not in at:  # both strands' jobs name one copy of the protein: they can pair
            at[a] = len(aa)
            aa += a
        tab[q].nt_off, tab[q].aa_off, tab[q].ss_off, tab[q].nl, tab[q].al = len(nt), at[a], -1, len(n), len(a)
        nt += n
    d_nt, d_aa = (torch.from_numpy(np.frombuffer(x, np.uint8).copy()).cuda() for x in (nt, aa))
    cap = sum(len(n) + len(a) + 8 for n, a in jobs)
    cig = torch.zeros(cap, dtype=torch.int32, device="cuda")
    res = torch.zeros(len(jobs) * C.sizeof(L.SpliceResult), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    rc = lib.pl_splice_batch_device(eng.h, opt.ptr, tab, len(jobs), d_nt.data_ptr(), d_aa.data_ptr(), None, res.data_ptr(),
                                    cig.data_ptr(), cap, None, None)
    out = (L.SpliceResult * len(jobs)).from_buffer_copy(res.cpu().numpy().tobytes())
    return rc, [(r.score, r.n_cigar, r.status) for r in out]


@pytest.mark.parametrize("pairing", [0, 2])
def test_wait_between_strips_runs_out_cleanly(pairing):
    import oracle_lib as O
    lib = L.load()
    opt = Options(flag=NS_F_CIGAR)
    jobs = _jobs(np.random.default_rng(5 + pairing), 12)
    want = [O.run("gs_auto", nt, aa, opt) for nt, aa in jobs]
    assert L.gpu_init(0)
    eng = L.Engine(0)
    try:
        eng.set_pairing(pairing)
        for _ in range(3):  # the launch sequence is captured and replayed by then
            assert [g[:2] for g in eng.align_host(opt, jobs)] == [(w[0], w[3]) for w in want]
        try:
            assert lib.pl_debug_strip_wait(4) == 1
            with pytest.raises(RuntimeError, match="wait between the strips"):
                eng.align_host(opt, jobs)
            rc, got = _device(lib, eng, opt, jobs)
            assert rc == 0 and "wait between the strips" in L.error()
            assert not L.gpu_global(*jobs[0], opt)[0]
            assert b"wait between the strips" in lib.ns_gpu_error()
        finally:
            lib.pl_debug_strip_wait(0)
        assert any(s == -3 for _, _, s in got) and got[-1][2] == 0
        for (score, n, status), w in zip(got, want):
            assert status in (0, -3)
            assert (score, n) == ((INT32_MIN, 0) if status else (w[0], len(w[3])))
        assert [g[:2] for g in eng.align_host(opt, jobs)] == [(w[0], w[3]) for w in want]
        rc, got = _device(lib, eng, opt, jobs)
        assert rc == 1 and [g[:2] for g in got] == [(w[0], len(w[3])) for w in want]
        ok, score, _, _, cig = L.gpu_global(*jobs[0], opt)
        assert ok and (score, cig) == (want[0][0], want[0][3])
    finally:
        eng.close()
