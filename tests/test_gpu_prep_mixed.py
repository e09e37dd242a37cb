"""The preparation of a batch of many short windows and one very long one: as fast as the two apart
would be, give or take (its grid was jobs x chunks of the longest window: 40 million CTAs here), with
the results of every kind of job against the oracle."""
import numpy as np
import pytest

from protlocus_b200 import lib as L
from protlocus_b200 import workload as W
from protlocus_b200.abi import NS_F_CIGAR, Options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 40, 20000])
def test_one_long_window_among_many(n):
    import oracle_lib as O
    rng = np.random.default_rng(n)
    opt = Options(flag=NS_F_CIGAR)
    aa = b"MKQTWPIACDEFGHIKLMNP"
    kinds = [(W.random_dna(rng, int(k)).encode(), aa) for k in rng.integers(60, 300, 40)]
    small = (kinds * (n // 40 + 1))[:n]
    gene = W.build_gene(rng, aa.decode(), divergence=0.1, n_frameshift=1, intron_lengths=[90])
    long = (W.random_dna(rng, 3_000_000) + gene + W.random_dna(rng, 1_000_000)).encode()
    eng = L.Engine(0)
    try:
        ms = []
        for batch in (small, small + [(long, aa)]):
            best = None
            for _ in range(3):
                eng.set_timing(True)
                got = eng.align_host(opt, batch)
                t = eng.times()["prep_ms"]
                best = t if best is None or t < best else best
            ms.append(best)
    finally:
        eng.close()
    # 4 million positions are some 20 MB in and out; with eight CTAs to a job 245 chunks in a row of a
    # few microseconds each: some 1 ms.  The grid of before took 20 ms for 20,000 jobs
    assert ms[1] < ms[0] + 4.0, ms
    for q in list(range(min(n, 40))) + [n]:
        nt, p = (small + [(long, aa)])[q]
        w = O.run("gs_auto", nt, p, opt)
        assert got[q][:2] == (w[0], w[3]), q
