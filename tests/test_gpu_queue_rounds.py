"""The request queue's batches when callers send one request at a time: a lone caller's requests run
one by one, several callers' together; every answer equals the checker's (the scores and CIGARs are
whole numbers)."""
import ctypes as C
import threading

import pytest

from protlocus_b200 import lib as L
from protlocus_b200.abi import NS_F_CIGAR, NsRst, Options

pytestmark = pytest.mark.gpu

NT, AA, ROUNDS = b"ATGAAAACTTGGCCGATTTGA", b"MKQTWPI", 6


@pytest.mark.parametrize("callers", [1, 2, 7, 130])
def test_one_request_at_a_time(oracle, callers):
    lib = L.load()
    assert L.gpu_init(0)
    opt = Options.nasw_defaults(flag=NS_F_CIGAR, go=3, ge=1, io=100, fs=100, sp_model=0)
    want = [oracle.run("gs16b", NT[k:], AA, opt) for k in range(ROUNDS)]
    out = [[None] * ROUNDS for _ in range(callers)]

    def caller(q):
        for k in range(ROUNDS):
            out[q][k] = L.gpu_global(NT[k:], AA, opt)

    l0 = lib.ns_gpu_launch_count()
    threads = [threading.Thread(target=caller, args=(q,)) for q in range(callers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for row in out:
        for k, (ok, score, ntl, aal, cig) in enumerate(row):
            assert ok and (score, ntl, aal, cig) == want[k]
    n = lib.ns_gpu_launch_count() - l0
    assert n == ROUNDS if callers == 1 else (callers * ROUNDS + 127) // 128 <= n <= callers * ROUNDS


def test_requests_sent_ahead_are_collected(oracle):
    lib = L.load()
    assert L.gpu_init(0)
    opt = Options.nasw_defaults(flag=NS_F_CIGAR, go=3, ge=1, io=100, fs=100, sp_model=0)
    want = oracle.run("gs16b", NT, AA, opt)
    for _ in range(9):  # the last batches were single requests
        assert L.gpu_global(NT, AA, opt)[0]
    l0 = lib.ns_gpu_launch_count()
    reqs = [lib.ns_gpu_submit(None, NT, len(NT), AA, len(AA), opt.ptr, None) for _ in range(5)]
    libc = C.CDLL(None)
    libc.free.argtypes = [C.c_void_p]
    for rq in reqs:
        r = NsRst()
        assert lib.ns_gpu_wait(rq, C.byref(r))
        assert (r.score, r.nt_len, r.aa_len, [r.cigar[k] for k in range(r.n_cigar)]) == want
        libc.free(C.cast(r.cigar, C.c_void_p))
    assert 1 <= lib.ns_gpu_launch_count() - l0 < 5
