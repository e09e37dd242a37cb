"""Which jobs share their strips: few jobs (every strip on a warp of its own), jobs of very different
sizes (the large ones), and not thousands of about a warp's share each, whose strips would cost more
than the jobs whole.  Scores and CIGARs against the oracle either way."""
import numpy as np
import pytest

from protlocus_b200 import lib as L
from protlocus_b200 import workload as W
from protlocus_b200.abi import NS_F_CIGAR, Options

pytestmark = pytest.mark.gpu


def _jobs(rng, n, al, nl):
    """n jobs of some al residues against some nl bases: 40 different ones, over and over."""
    jobs = []
    for _ in range(40):
        aa = W.random_protein(rng, int(rng.integers(al * 7 // 10, al * 13 // 10 + 1))).encode()
        gene = W.build_gene(rng, aa.decode(), divergence=0.2, n_frameshift=1, intron_lengths=[]).encode()
        nt = (gene + W.random_dna(rng, nl * 13 // 10).encode())[:int(rng.integers(nl * 7 // 10, nl * 13 // 10 + 1))]
        jobs.append((nt, aa))
    return (jobs * (n // 40 + 1))[:n]


@pytest.mark.parametrize("n,al,nl,shared", [
    (40, 20, 600, "all"), (300, 150, 1000, "all"), (2400, 150, 4000, "all"),
    (5000, 20, 600, "none"), (5000, 40, 1000, "none"), (5000, 80, 600, "none"), (12000, 150, 600, "none")])
def test_rule(n, al, nl, shared):
    import oracle_lib as O
    rng = np.random.default_rng(n + al)
    opt = Options(flag=NS_F_CIGAR)
    jobs = _jobs(rng, n, al, nl)
    big = (jobs[0][0] + W.random_dna(rng, 60000).encode(), W.random_protein(rng, 400).encode())
    eng = L.Engine(0)
    try:
        eng.set_pairing(0)
        got = eng.align_host(opt, jobs)
        coop = eng.last_plan()["coop"]
        assert coop == (n if shared == "all" else 0), coop
        mixed = eng.align_host(opt, jobs + [big])  # a job far above the others
        assert eng.last_plan()["coop"] >= 1
    finally:
        eng.close()
    want = [O.run("gs_auto", nt, aa, opt) for nt, aa in jobs[:40] + [big]]
    for q in range(n):
        w = want[q % 40]
        assert got[q][:2] == (w[0], w[3]) and mixed[q][:2] == (w[0], w[3]), q
    assert mixed[-1][:2] == (want[-1][0], want[-1][3])
