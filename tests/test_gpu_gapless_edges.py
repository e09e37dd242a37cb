"""The gapless scorer where its wide reads end: contigs of a few bases at either end of the genome,
odd genome lengths, anchors on the first and past the last block, both strands, runs of N, block
widths that are no multiple of a lane's eight deltas, the compiled k-mer lengths and others, and
a genome that starts at any byte of its device buffer.  Against the C restatement."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from protlocus_b200 import lib as L
from protlocus_b200 import workload as W
from protlocus_b200.abi import BLOSUM62, make_tables, set_stop_sc

pytestmark = pytest.mark.gpu

MAT = set_stop_sc(BLOSUM62, 23)
CODON = make_tables()[2]


def _case(rng, bases, contigs, n, al, width, kmer):
    g = rng.integers(0, 4, bases).astype(np.uint8)
    for _ in range(4):
        a = int(rng.integers(0, bases))
        g[a:a + int(rng.integers(1, 30))] = 4
    lens = np.full(contigs, 40 if bases < 4000 else 400)
    lens[0], lens[-1] = int(rng.integers(1, 9)), int(rng.integers(1, 40))
    lens[contigs // 2] = bases - lens.sum() + lens[contigs // 2]
    off = np.concatenate([[0], np.cumsum(lens[:-1])])
    q = rng.integers(0, 22, 6 * al).astype(np.uint8)
    cand, anc = np.zeros(n, W.GAPLESS_CAND_DTYPE), np.zeros(5 * n, W.GAPLESS_ANCHOR_DTYPE)
    for k in range(n):
        c = int(rng.choice([0, contigs // 2, contigs - 1, int(rng.integers(0, contigs))]))
        t_off, t_len = int(off[c]), int(lens[c])
        if k % 37 == 0:  # spans that reach outside the genome read as missing bases
            t_off, t_len = t_off - 50, t_len + 120
        cand[k] = (t_off, t_len, int(rng.integers(0, 6)) * al, al, 5 * k, 5, int(rng.integers(0, 2)))
        tb = rng.integers(-1, t_len // width + 2, 5) * width
        anc["target_block"][5 * k:5 * k + 5] = tb
        anc["query_end"][5 * k:5 * k + 5] = rng.integers(0, al + 1, 5)
    for k in range(0, n, 3):  # true matches: the query's residues spelled out under an anchor
        c = cand[k]
        a = anc[5 * k]
        L_ = int(c["target_length"])
        pos = int(max(a["target_block"], 0)) + int(rng.integers(0, width))
        qe = int(a["query_end"])
        for r in range(max(0, qe - 25), min(al, qe + 25)):
            e = pos + 3 * (r - qe)
            cod = np.nonzero(CODON == q[c["query_offset"] + r])[0]
            if len(cod) == 0 or e - 2 < 0 or e >= L_:
                continue
            v = int(rng.choice(cod))
            for i, b in enumerate((v >> 4, v >> 2 & 3, v & 3)):
                p = e - 2 + i
                at = int(c["target_offset"]) + (L_ - 1 - p if c["reverse"] else p)
                if 0 <= at < bases:
                    g[at] = 3 - b if c["reverse"] else b
    return {"packed": W.pack_nt4(g), "bases": bases, "queries": q, "candidates": cand, "anchors": anc,
            "block_width": width, "kmer": kmer}


def _want(oracle, w, *args):
    """The restatement's scores.  It reads the genome unchecked, so it gets a copy with 128 Ns on
    either side: what lies outside the genome reads as missing."""
    g = np.stack([w["packed"] & 15, w["packed"] >> 4], axis=1).reshape(-1)[:w["bases"]]
    c = w["candidates"].copy()
    c["target_offset"] += 128
    n = np.full(128, 4, np.uint8)
    return oracle.port_gapless(dict(w, packed=W.pack_nt4(np.concatenate([n, g, n, n[:2]])), candidates=c), *args)


@pytest.mark.parametrize("bases,width,kmer", [(700, 256, 6), (701, 256, 6), (5003, 256, 6), (90011, 256, 6),
                                              (5001, 1, 6), (5002, 7, 5), (20007, 100, 7), (20001, 513, 6), (20003, 256, 1),
                                              (20005, 256, 4), (60001, 1024, 8), (60003, 8192, 6), (20009, 250, 64)])
def test_edges(oracle, bases, width, kmer):
    rng = np.random.default_rng(bases + width + kmer)
    w = _case(rng, bases, 5, 1500, 90, width, kmer)
    eng = L.Engine(0)
    try:
        want = _want(oracle, w, width, kmer, 30, MAT, CODON)
        got = eng.gapless_score(w, width, kmer, 30, MAT, CODON)
        bad = np.nonzero(got != want)[0]
        assert bad.size == 0, (bad[:5], got[bad[:5]], want[bad[:5]])
        assert (want > 60).any() or width < 8 or kmer > 40
        # the genome at an odd byte of a device buffer: no aligned words
        for shift in (1, 2):
            d = {k: torch.from_numpy(w[k].view(np.uint8).reshape(-1).copy()).cuda() for k in ("queries", "candidates", "anchors")}
            buf = torch.zeros(w["packed"].size + 8, dtype=torch.uint8, device="cuda")
            buf[shift:shift + w["packed"].size] = torch.from_numpy(w["packed"]).cuda()
            sc = torch.zeros(len(w["candidates"]), dtype=torch.int32, device="cuda")
            mat, codon = np.ascontiguousarray(MAT, np.int8), np.ascontiguousarray(CODON, np.uint8)
            torch.cuda.synchronize()
            assert eng.lib.pl_gapless_score_device(
                eng.h, buf.data_ptr() + shift, bases, d["queries"].data_ptr(), w["queries"].size, d["candidates"].data_ptr(),
                len(w["candidates"]), d["anchors"].data_ptr(), len(w["anchors"]), width, kmer, 30, mat.ctypes.data, 22,
                codon.ctypes.data, sc.data_ptr(), None), L.error()
            assert (sc.cpu().numpy() == want).all()
    finally:
        eng.close()
