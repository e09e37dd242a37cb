"""The seeding's in-shared-memory sort against the restatement: proteins with 0 anchors, around the
class sizes (2048 << c anchors), past the largest (the segmented sort), and index blocks that
spread evenly, cluster in a few buckets of more than 12 and of more than 128 keys, all fall on
one block, use the ids' whole 32 bits, or come in descending order in their buckets."""
import numpy as np
import pytest

from protlocus_b200 import lib as L

pytestmark = pytest.mark.gpu

AA = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", np.uint8)


def _index(rng, mean_occ, blocks):
    n_bucket = 1 << 23
    cnt = rng.poisson(mean_occ, n_bucket).astype(np.int64)
    ki = np.zeros(n_bucket, np.int64)
    ki[1:] = np.cumsum(cnt[:-1])
    return ki, np.ascontiguousarray(blocks(int(cnt.sum())), np.uint32)


KINDS = {
    "spread": lambda r: lambda n: r.integers(0, 781250, n),
    "full_range": lambda r: lambda n: r.integers(0, 1 << 32, n, dtype=np.uint64),
    "clusters": lambda r: lambda n: np.where(r.random(n) < 0.3, 5000 + r.integers(0, 40, n), r.integers(0, 781250, n)),
    "small_clusters": lambda r: lambda n: r.integers(0, 60, n) * 13000 + r.integers(0, 3, n),
    "one_block": lambda r: lambda n: np.full(n, 77),
    "few_blocks": lambda r: lambda n: r.integers(0, 5, n),
    "descending": lambda r: lambda n: np.sort(r.integers(0, 781250, n))[::-1],
}


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("mean_occ", [1.5, 8.0])
def test_sorted_anchors(kind, mean_occ):
    import oracle_lib as O
    rng = np.random.default_rng(len(kind) + int(mean_occ))
    ki, kb = _index(rng, mean_occ, KINDS[kind](rng))
    per = mean_occ / 2  # anchors a residue (every other k-mer is a seed)
    lens = [0, 3, 7, 30, 200]
    for c in range(4):  # around the classes' sizes, so both sides of each edge are met
        lens += [int((2048 << c) / per * f) for f in (0.9, 0.97, 1.0, 1.03, 1.1)]
    lens += [int(30000 / per)]
    prots = [AA[rng.integers(0, 20, n)].tobytes() for n in lens]
    eng = L.Engine(0)
    idx = L.SeedIndex(ki, kb, 6, 1)
    try:
        got = L.seed_anchors(eng, idx, prots, 20000)
        sizes = []
        for p, a in zip(prots, got):
            want = O.seed_anchors(ki, kb, 6, 1, 20000, p, use_ref=False)
            assert np.array_equal(a, want), (kind, len(p), len(a), len(want))
            sizes.append(len(a))
        assert max(sizes) > 16384 and min(sizes) == 0
        assert [len(x) for x in L.seed_anchors(eng, idx, prots[:4], 20000)] == sizes[:4]
    finally:
        idx.close()
        eng.close()
