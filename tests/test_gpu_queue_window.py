"""The request queue's collection rule.  A lone caller, who sends one request and waits, is served at
once: a tiny request's answer takes less than the 2 ms for which the queue would otherwise wait for
others.  Callers that come together, round after round, share their batches."""
import threading
import time

import pytest

from protlocus_b200 import lib as L
from protlocus_b200.abi import NS_F_CIGAR, Options

pytestmark = pytest.mark.gpu

NT, AA = b"ATGAAAACTTGGCCGATTTGA", b"MKQTWPI"


def _opt():
    return Options.nasw_defaults(flag=NS_F_CIGAR, go=3, ge=1, io=100, fs=100, sp_model=0)


def test_lone_caller_waits_for_nobody(oracle):
    assert L.gpu_init(0)
    opt, took = _opt(), []
    want = oracle.run("gs16b", NT, AA, opt)
    for _ in range(60):
        t0 = time.perf_counter()
        ok, score, ntl, aal, cig = L.gpu_global(NT, AA, opt)
        took.append(time.perf_counter() - t0)
        assert ok and (score, ntl, aal, cig) == want
    # the first requests follow whatever the queue served before; with the window each takes at least 2 ms
    assert sorted(took[20:])[20] < 0.002, sorted(took[20:])[20]


@pytest.mark.parametrize("callers", [2, 7, 40])
def test_callers_in_step_share_batches(callers):
    lib = L.load()
    assert L.gpu_init(0)
    opt, rounds, warm = _opt(), 30, 10
    gate = threading.Barrier(callers)
    count, bad = [], []

    def caller(q):
        for k in range(rounds):
            if gate.wait() == 0 and k >= warm:
                count.append(lib.ns_gpu_launch_count())
            gate.wait()
            if not L.gpu_global(NT, AA, opt)[0]:
                bad.append((q, k))

    threads = [threading.Thread(target=caller, args=(q,)) for q in range(callers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    # one batch a round once the queue has seen the callers together; at most two on average where a
    # thread is late beyond the window
    n, per = lib.ns_gpu_launch_count() - count[0], rounds - warm
    assert per <= n <= 2 * per, (n, per)
