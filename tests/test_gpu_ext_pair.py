"""Extension requests that run two to a warp in 16-bit halves, at the edges of what a pair accepts:
proteins of one short of the smallest to a few segments, halves whose segment lengths, padded columns
and strips differ, both orientations and stripe widths, tracks, x-drops that end one half early, odd
batches, and requests that must not pair (short proteins, position-specific scores, a negative
end bonus).  Every answer (whole numbers) equals the unpaired kernel's and the checker's.
"""
import numpy as np
import pytest

from protlocus_b200 import lib as L
from protlocus_b200 import workload as W
from protlocus_b200.abi import NS_F_EXT_LEFT, NS_F_EXT_RIGHT, Options

pytestmark = pytest.mark.gpu

ALS = (30, 31, 32, 33, 47, 48, 49, 63, 64, 65, 100, 127, 128, 129, 160)
WINDOWS = (3, 4, 60, 257, 258, 259, 513, 514, 515, 900, 1300)


def _requests(rng, n, odd_kinds):
    aas = b"ACDEFGHIKLMNPQRSTVWY"
    out = []
    for q in range(n):
        al = int(rng.choice(ALS))
        nl = int(rng.choice(WINDOWS))
        if q % 3:  # a gene, so that the scores climb before the x-drop ends them
            nt, aa = W.single_locus(seed=9000 + q, al=al, window=max(nl, 3 * al + 40), n_intron=q % 2)
            nt = nt[:max(3, nl)] if q % 4 == 1 else nt
        else:
            nt, aa = bytes(rng.choice(list(b"ACGTN"), size=nl)), bytes(rng.choice(list(aas), size=al))
        r = {"nt": nt, "aa": aa, "flag": NS_F_EXT_LEFT if q & 1 else NS_F_EXT_RIGHT, "width": 16 if (q >> 1) & 1 else 8}
        if q % 5 == 2:
            r["ss"] = W.random_ss(rng, len(nt))
        if odd_kinds and q % 11 == 5:
            r["pssm"] = rng.integers(-6, 10, size=(len(aa), 22)).astype(np.int8)
        out.append(r)
    return out


@pytest.mark.parametrize("n,odd_kinds,opt", [
    (2, False, Options()), (3, False, Options()), (129, True, Options()), (128, False, Options(xdrop=20, end_bonus=0)),
    (97, True, Options(xdrop=10 ** 6, end_bonus=5)), (64, False, Options(end_bonus=65535)),
    (64, True, Options(end_bonus=-3)), (65, False, Options(go=0, ge=0, io=0, fs=0)),
    (64, False, Options(go=200, ge=56, io=256, fs=256, stop_pen=100))])
def test_pairs_equal_singles(oracle, n, odd_kinds, opt):
    reqs = _requests(np.random.default_rng(n), n, odd_kinds)
    e = L.Engine(0)
    e.set_pairing(2)
    paired = e.ext_host(opt, reqs)
    e.set_pairing(False)
    single = e.ext_host(opt, reqs)
    e.close()
    assert paired == single
    for r, g in zip(reqs, paired):
        o = opt.with_flag(r["flag"])
        if r.get("pssm") is not None:
            o = o.with_pssm(r["pssm"])
        s, ntl, aal, _ = oracle.port_run("gs16b", r["nt"], r["aa"], o, r.get("ss"), avx2=r["width"] == 16)
        assert g == (s, ntl, aal), (len(r["nt"]), len(r["aa"]))
