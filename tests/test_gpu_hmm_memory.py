"""The profile scan's scratch memory and streams: profiles of one tile (up to 256 columns) hand
nothing from tile to tile and take no edge memory, and a set of profiles of one and several tiles
in any order, over more and fewer profiles than streams, on a fresh engine and again on the same,
scores as its profiles alone."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from protlocus_b200 import hmm as H
from protlocus_b200 import lib as L

pytestmark = pytest.mark.gpu


def _profile(rng, m):
    emit = rng.integers(-14, 3, (m, 20)).astype(np.int16)
    emit[np.arange(m), rng.integers(0, 20, m)] = 4
    trans = -rng.integers(0, 12, (m, 7)).astype(np.int16)
    return L.HmmProfile(emit, trans, H.codon_alpha())


def test_one_tile_takes_no_edge_memory():
    rng = np.random.default_rng(1)
    regions = [rng.integers(0, 4, 30000).astype(np.uint8) for _ in range(600)]
    profs = [_profile(rng, m) for m in (40, 64, 65, 96, 128, 160, 192, 224, 255, 256)]
    used = []
    for _ in range(2):  # the context's own memory (the kernels' code and stacks, streams) comes with the first engine
        eng = L.Engine(0)
        try:
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            eng.hmm_score_many(profs, regions)
            used.append(free - torch.cuda.mem_get_info()[0])
        finally:
            eng.close()
    # the bases (18 MB), their rows (6 MB) and six small arrays, each rounded up to 2 MB; the edges of
    # 600 regions' warps would be 90 MB a stream
    assert used[1] <= 48 << 20, [u >> 20 for u in used]


@pytest.mark.parametrize("lens", [[300], [900, 100], [100, 900], [30, 257, 256, 1100, 70, 513, 200, 800, 1200, 90, 520, 40]])
def test_tiles_in_any_order(lens):
    rng = np.random.default_rng(len(lens))
    profs = [_profile(rng, m) for m in lens]
    regions = [rng.integers(0, 5, int(k)).astype(np.uint8) for k in rng.choice([0, 2, 3, 50, 301, 2000, 6000], 61)]
    eng, one = L.Engine(0), L.Engine(0)
    try:
        want = [one.hmm_score(p, regions) for p in profs]
        for q in (np.arange(len(profs)), np.arange(len(profs))[::-1], rng.permutation(len(profs))):
            got = eng.hmm_score_many([profs[k] for k in q], regions)
            assert [list(x) for x in got] == [list(want[k]) for k in q]
    finally:
        eng.close()
        one.close()
        for p in profs:
            p.close()
