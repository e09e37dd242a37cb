"""The hand-off between the strips of a job on different warps, under load: hundreds of strips of a
few columns each, where a column's entry is taken as soon as it is written, run again and again on
one engine (the ring holds the entries of the run before until it is cleared).  Scores and CIGARs
are whole numbers: every run equals the oracle's."""
import numpy as np
import pytest

from protlocus_b200 import lib as L
from protlocus_b200 import workload as W
from protlocus_b200.abi import NS_F_CIGAR, Options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("al", [1, 3, 17, 33, 60])
@pytest.mark.parametrize("pairing", [0, 2])
def test_repeated_batches(al, pairing):
    import oracle_lib as O
    rng = np.random.default_rng(al)
    opt = Options(flag=NS_F_CIGAR)
    jobs = []
    for q in range(24):
        aa = W.random_protein(rng, al).encode()
        gene = W.build_gene(rng, aa.decode(), divergence=0.2, n_frameshift=1 if al > 8 else 0, intron_lengths=[]).encode()
        nt = (gene + W.random_dna(rng, 5000).encode())[:int(rng.integers(1500, 5000))]
        jobs += [(nt, aa), (W.revcomp(nt), aa)]
    want = [O.run("gs_auto", nt, aa, opt) for nt, aa in jobs]
    eng = L.Engine(0)
    try:
        eng.set_tuning(0, 0.7)  # 8 rows a lane: strips of 256 rows
        eng.set_pairing(pairing)
        for _ in range(8):
            got = eng.align_host(opt, jobs)
            assert eng.last_plan()["coop"] > 0  # shared strips
            assert [g[:2] for g in got] == [(w[0], w[3]) for w in want]
    finally:
        eng.close()
