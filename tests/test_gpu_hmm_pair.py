"""The paired 16-bit profile DP (two regions per warp) against the restatement: profile lengths
at the edges of a lane's columns and of the tiles, odd numbers of regions and regions of very
different lengths in one batch, and tables at the edge of the 16-bit range -- the largest
emission the paired kernel admits, one above it, scores at int16's lowest value, and a positive
transition (both sent to the 32-bit kernel)."""
import numpy as np
import pytest

from protlocus_b200 import hmm as H
from protlocus_b200 import lib as L

pytestmark = pytest.mark.gpu


def _tables(rng, m, emax=4):
    emit = rng.integers(-14, emax + 1, (m, 20)).astype(np.int16)
    emit[rng.random((m, 20)) < 0.02] = -32768
    emit[np.arange(m), rng.integers(0, 20, m)] = emax
    trans = -rng.integers(0, 12, (m, 7)).astype(np.int16)
    trans[:, [0, 3, 5]] = -rng.integers(0, 2, (m, 3)).astype(np.int16)
    trans[rng.random((m, 7)) < 0.02] = -32768
    return emit, trans


def _regions(rng, emit, n):
    ca = H.codon_alpha()
    by = [np.nonzero(ca == a)[0] for a in range(20)]
    out = []
    for q in range(n):
        L_ = int(rng.choice([0, 2, 3, 5, 9, 12, 13, 48, 49, 300, 301, 302, 1200, 2000]))
        s = rng.integers(0, 5 if q % 5 == 0 else 4, L_).astype(np.uint8)
        k = min(L_ // 3, len(emit))
        if q % 2 and k > 2:  # the profile's own best residues, so that states grow along the diagonal
            a = int(rng.integers(0, len(emit) - k + 1))
            cod = np.array([rng.choice(by[r]) for r in emit[a:a + k].argmax(axis=1)])
            s[:3 * k] = np.stack([cod >> 4, cod >> 2 & 3, cod & 3], axis=1).reshape(-1)
        out.append(s)
    return out


def _check(engine, oracle, m, emit, trans, n=37):
    rng = np.random.default_rng(m)
    ca = H.codon_alpha()
    regions = _regions(rng, emit, n)
    prof = L.HmmProfile(emit, trans, ca)
    got = engine.hmm_score(prof, regions)
    want = [oracle.port_hmm(m, emit, trans, ca, r) for r in regions]
    assert got == want, (m, [k for k in range(n) if got[k] != want[k]][:5])
    assert list(engine.hmm_score_many([prof, prof], regions)[1]) == want
    prof.close()
    return want


@pytest.fixture(scope="module")
def engine():
    e = L.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("m", [1, 2, 31, 33, 63, 64, 65, 96, 127, 129, 255, 256, 257, 320, 321, 511, 513, 800, 1025,
                               2048, 2049])
def test_profile_lengths(engine, oracle, m):
    emit, trans = _tables(np.random.default_rng(m), m)
    _check(engine, oracle, m, emit, trans)


@pytest.mark.parametrize("m,emax", [(80, 203), (80, 204), (200, 81), (500, 32), (500, 33), (16, 991), (1, 10921),
                                    (1, 10922), (300, 32767)])
def test_edge_of_the_16_bit_range(engine, oracle, m, emax):
    emit, trans = _tables(np.random.default_rng(m), m, emax)
    trans[:, [0, 3, 5]] = 0
    best = max(_check(engine, oracle, m, emit, trans, 61))
    assert best >= min(m, 600) * emax // 3


def test_positive_transition(engine, oracle):
    emit, trans = _tables(np.random.default_rng(9), 70)
    trans[33, 0] = 5
    _check(engine, oracle, 70, emit, trans)
