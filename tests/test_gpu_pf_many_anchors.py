"""Candidates with more anchors than the feature kernel keeps: the window's first 1024 anchors by
position make the chain, the same ones in every run.  The windows hold copies of a part of the
protein and, past the 1024th anchor, the whole of it, so that a later anchor kept in the place of
an earlier one gives a longer chain."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from protlocus_b200 import lib as L
from protlocus_b200 import prefilter as P
from protlocus_b200 import workload as W
from protlocus_b200.abi import make_tables

pytestmark = pytest.mark.gpu


def _window(rng, prot, copies, tail):
    part = prot[:len(prot) // 2]
    s = [W.random_dna(rng, int(rng.integers(0, 40)))]
    s += [W.reverse_translate(rng, part) + "G" * int(rng.integers(0, 3)) for _ in range(copies)]
    w = np.frombuffer("".join(s).encode(), np.uint8).copy()
    w[rng.random(len(w)) < 0.002] = ord("N")
    return w.tobytes() + W.reverse_translate(rng, prot).encode() + W.random_dna(rng, tail).encode()


def _head(pf_ref, w, a, tabs):
    """The shortest start of the window that holds its first 1024 anchors, and its features."""
    lo, hi, got = 0, len(w), None
    while hi - lo > 1:
        mid = (lo + hi) // 2
        try:
            f = pf_ref.features(w[:mid], a, *tabs)
        except AssertionError:  # more than 1024
            hi = mid
            continue
        lo, hi, got = (lo, mid, f) if f[2] == 1024 else (mid, hi, got)
    return got


@pytest.mark.parametrize("al,copies,tail", [(40, 90, 0), (61, 130, 517), (120, 60, 3000)])
def test_first_anchors_kept(al, copies, tail):
    import pf_ref
    rng = np.random.default_rng(al)
    tabs = make_tables()
    prot = W.random_protein(rng, al)
    wins = [_window(rng, prot, copies + q, tail) for q in range(6)]
    nt, jobs, pn = [], np.zeros(len(wins), P.JOB_DTYPE), 0
    for q, w in enumerate(wins):  # every alignment of the window matters little here: six of them
        nt += [b"T" * (q + 1), w]
        jobs[q] = (pn + q + 1, 0, -1, len(w), al)
        pn += q + 1 + len(w)
    eng = L.Engine(0)
    try:
        pipe = P.Pipeline(eng, {"nt": np.frombuffer(b"".join(nt), np.uint8), "aa": np.frombuffer(prot.encode(), np.uint8),
                                "jobs": jobs})
        runs = []
        for _ in range(3):
            feats, chain = pipe.features()
            torch.cuda.synchronize()
            runs.append((feats.float().cpu().numpy(), chain.cpu().numpy()))
    finally:
        eng.close()
    for F, ch in runs[1:]:
        assert np.array_equal(F, runs[0][0]) and np.array_equal(ch, runs[0][1])
    F, ch = runs[0]
    for q, w in enumerate(wins):
        want, wchain, na, length = _head(pf_ref, w, prot.encode(), tabs)
        assert na == 1024
        assert F[q, 531] == 1.0  # more anchors than kept
        assert list(ch[q]) == wchain, (q, list(ch[q]), wchain)
        assert F[q, 516] == pytest.approx(want[516], rel=2 ** -7)  # log2 of the chain's length, one bf16 ulp
        assert F[q, 523] == want[523] and F[q, 528] == want[528]  # frame changes, length / anchors kept
