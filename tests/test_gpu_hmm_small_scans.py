"""Scans of few regions: they spread over the SMs, so that as many regions as SMs take about as long
as one, and a profile's scores are the same on either side of the number of regions at which its
kernel changes (four per SM: the 32-bit kernel of profiles with more than five columns a lane, else
two regions a warp), alone and beside other profiles.  Scores against the restatement."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from protlocus_b200 import hmm as H
from protlocus_b200 import lib as L

pytestmark = pytest.mark.gpu


def _tables(rng, m):
    emit = rng.integers(-14, 3, (m, 20)).astype(np.int16)
    emit[np.arange(m), rng.integers(0, 20, m)] = 4
    trans = -rng.integers(0, 12, (m, 7)).astype(np.int16)
    trans[:, 0] = -rng.integers(0, 2, m)
    return emit, trans


@pytest.mark.parametrize("m", [100, 250, 300, 400, 800])
def test_regions_spread_over_the_sms(m):
    rng = np.random.default_rng(m)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    prof = L.HmmProfile(*_tables(rng, m), H.codon_alpha())
    region = rng.integers(0, 4, 6000).astype(np.uint8)
    eng = L.Engine(0)
    try:
        ms = {}
        for n in (1, sms):
            for _ in range(5):
                eng.set_timing(True)
                eng.hmm_score(prof, [region] * n)
                ms[n] = min(ms.get(n, 1e9), eng.times()["dp_ms"])
    finally:
        eng.close()
        prof.close()
    # a region has its scheduler to itself either way; with eight regions an SM it took 1.3 to 1.6 times as long
    assert ms[sms] < 1.2 * ms[1], ms


@pytest.mark.parametrize("m", [30, 161, 192, 193, 256, 385, 700])
@pytest.mark.parametrize("edge", [1, 4])
def test_kernels_agree(oracle, m, edge):
    rng = np.random.default_rng(m)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ca = H.codon_alpha()
    emit, trans = _tables(rng, m)
    prof, other = L.HmmProfile(emit, trans, ca), L.HmmProfile(*_tables(rng, 90), ca)
    kinds = [rng.integers(0, 5, int(k)).astype(np.uint8) for k in rng.choice([3, 50, 301, 700], 12)]
    want = [oracle.port_hmm(m, emit, trans, ca, r) for r in kinds]
    eng = L.Engine(0)
    try:
        for n in (1, 2, edge * sms - 1, edge * sms, edge * sms + 1, edge * sms // 2, edge * sms // 2 + 1):
            regions = (kinds * (n // 12 + 1))[:n]
            expect = (want * (n // 12 + 1))[:n]
            assert list(eng.hmm_score(prof, regions)) == expect, n
            assert list(eng.hmm_score_many([other, prof], regions)[1]) == expect, n
    finally:
        eng.close()
        prof.close()
        other.close()
