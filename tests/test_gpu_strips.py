"""Shared strips of the global spliced DP: the strips of one job run on different warps, so the
sizes that matter are the strip edges (256 and 512 rows at 8 rows per lane, 128 and 256 at 4),
proteins shorter and longer than a warp, and batches of a few jobs (every strip shared) and of
many (some jobs whole on one warp).  Scores and CIGARs against the oracle."""
import numpy as np
import pytest

from protlocus_b200 import lib as L
from protlocus_b200 import workload as W
from protlocus_b200.abi import NS_F_CIGAR, Options

pytestmark = pytest.mark.gpu

ROWS = [1, 127, 128, 129, 255, 256, 257, 511, 512, 513, 769, 2049]


@pytest.mark.parametrize("r4_rows", [0, 1 << 30])
@pytest.mark.parametrize("al", [1, 2, 31, 32, 33, 65, 260])
@pytest.mark.parametrize("pairing", [0, 2])
def test_strip_edges(r4_rows, al, pairing):
    import oracle_lib as O
    rng = np.random.default_rng(1000 * al + pairing)
    opt = Options(flag=NS_F_CIGAR)
    jobs = []
    for nr in ROWS:
        nl = nr + 2
        aa = W.random_protein(rng, al).encode()
        gene = W.build_gene(rng, aa.decode(), divergence=0.2, n_frameshift=1 if al > 8 else 0,
                            intron_lengths=[60] if al > 30 else []).encode()
        nt = (gene + W.random_dna(rng, nl).encode())[:nl]
        jobs += [(nt, aa), (W.revcomp(nt), aa)]
    eng = L.Engine(0)
    try:
        eng.set_tuning(r4_rows, 0.7)
        eng.set_pairing(pairing)
        for batch in (jobs, jobs[-2:], jobs * 40):  # few strips, one locus, more jobs than strips a warp
            got = eng.align_host(opt, batch)
            for (nt, aa), (s, c, _w) in zip(batch[:len(jobs)], got):
                want = O.run("gs_auto", nt, aa, opt)
                assert (s, c) == (want[0], want[3]), (len(nt), len(aa))
            assert [g[:2] for g in got[:len(jobs)]] * (len(batch) // len(jobs) or 1) == [g[:2] for g in got]
    finally:
        eng.close()


@pytest.mark.parametrize("match", [60, 127])
def test_strip_edges_wide(match):
    """The 32-bit and the doubly clamped width over several strips of few jobs."""
    import oracle_lib as O
    rng = np.random.default_rng(match)
    mat = np.full((22, 22), -4, np.int8)
    np.fill_diagonal(mat, match)
    opt = Options(flag=NS_F_CIGAR, matrix=mat)
    jobs = []
    for al in (230, 255, 300, 520, 545):
        aa = W.random_protein(rng, al).encode()
        nt = (W.reverse_translate(rng, aa.decode()) + W.random_dna(rng, 300)).encode()
        jobs += [(nt[:3 * al + int(rng.integers(0, 300))], aa)]
    eng = L.Engine(0)
    try:
        got = eng.align_host(opt, jobs)
        for (nt, aa), (s, c, _w) in zip(jobs, got):
            want = O.run("gs_auto", nt, aa, opt)
            assert (s, c) == (want[0], want[3]), (len(nt), len(aa))
    finally:
        eng.close()
