"""The candidate features' scan and chain at their edges, against the restatement: windows of 1
to 40 bases and around the 16-position groups and a warp's 512 positions, at every alignment of
the window in its buffer, with Ns at random and at the ends; anchor counts around 32, 256 (the
rank sort's limit) and towards 1024, chains with equal scores."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from protlocus_b200 import lib as L
from protlocus_b200 import prefilter as P
from protlocus_b200 import workload as W
from protlocus_b200.abi import make_tables

pytestmark = pytest.mark.gpu


def _check(cands):
    """cands: (window bytes, protein bytes, padding before the window)"""
    import pf_ref
    nt, aa, jobs = [], [], np.zeros(len(cands), P.JOB_DTYPE)
    pn = pa = 0
    for q, (w, a, pad) in enumerate(cands):
        nt += [b"T" * pad, w]
        jobs[q] = (pn + pad, pa, -1, len(w), len(a))
        aa.append(a)
        pn, pa = pn + pad + len(w), pa + len(a)
    eng = L.Engine(0)
    try:
        pipe = P.Pipeline(eng, {"nt": np.frombuffer(b"".join(nt), np.uint8), "aa": np.frombuffer(b"".join(aa), np.uint8),
                                "jobs": jobs})
        feats, chain = pipe.features()
        torch.cuda.synchronize()
        F, ch = feats.float().cpu().numpy(), chain.cpu().numpy()
    finally:
        eng.close()
    tabs = make_tables()
    count = []
    for q, (w, a, _) in enumerate(cands):
        want, wchain, na, _len = pf_ref.features(w, a, *tabs)
        assert np.array_equal(F[q, :512], want[:512]), (q, len(w), len(a))
        assert list(ch[q]) == wchain, (q, len(w), na, list(ch[q]), wchain)
        # scalars: within one bf16 ulp (device log2f may differ from numpy's by an ulp)
        assert np.allclose(F[q, 512:], want[512:], rtol=2 ** -7, atol=1e-6), (q, F[q, 512:532], want[512:532])
        count.append(na)
    return count


def _window(rng, prot, n):
    gene = W.build_gene(rng, prot, divergence=0.1, n_frameshift=1 if len(prot) > 20 else 0,
                        intron_lengths=[70] if len(prot) > 40 else [])
    left = int(rng.integers(0, max(1, n // 3)))
    s = np.frombuffer((W.random_dna(rng, left) + gene + W.random_dna(rng, n)).encode()[:n], np.uint8).copy()
    s[rng.random(n) < 0.01] = ord("N")
    return s.tobytes()


@pytest.mark.parametrize("lo,hi,step", [(1, 41, 1), (500, 530, 1), (1015, 1040, 3), (4090, 4115, 3), (8180, 8200, 7)])
def test_window_edges(lo, hi, step):
    rng = np.random.default_rng(lo)
    cands = []
    for n in range(lo, hi, step):
        for pad in rng.choice(16, 4, replace=False):
            prot = W.random_protein(rng, int(rng.choice([1, 4, 5, 6, 30, 200, 420])))
            w = _window(rng, prot, n)
            if n > 3 and pad % 2:
                w = b"N" + w[1:-1] + b"N"
            cands.append((w, prot.encode(), int(pad)))
    _check(cands)


def test_anchor_counts():
    rng = np.random.default_rng(4)
    cands = []
    for al in (31, 36, 37, 68, 250, 258, 262, 300, 520, 700, 990):  # an undiverged copy: an anchor per residue
        prot = W.random_protein(rng, al)
        cands.append(((W.random_dna(rng, 100) + W.reverse_translate(rng, prot) + W.random_dna(rng, 100)).encode(),
                      prot.encode(), int(rng.integers(0, 16))))
    unit = W.random_protein(rng, 40)  # repeats: many anchors share a protein position
    cands.append((W.reverse_translate(rng, unit * 12).encode(), unit.encode(), 3))
    cands.append((W.reverse_translate(rng, unit * 3).encode(), (unit * 9).encode(), 5))
    count = _check(cands)
    assert max(count) > 900 and any(256 < c < 300 for c in count) and any(c <= 32 for c in count), count
