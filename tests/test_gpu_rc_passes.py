"""The recheck's logsum term at every float of its range, and the warps' passes at the edges of
their blocks and rings: rows of 1 column to a few more than the rings hold, peptides of 1 residue
on, groups whose lanes start at different steps and that hold 1 to 32 peptides.  The checker
restates rc_score (recheck.c:283-440) in float32 with the host's expf, log1pf and logf; the bit
score without null2 has to be equal.  The bias ends in double-precision exp, log and log1p of the
device, rounded to float: one unit in its last place, which the bit score inherits.
"""
import ctypes as C

import numpy as np
import pytest

from protlocus_b200 import lib as L

pytestmark = pytest.mark.gpu

f32 = np.float32
NEG = f32(-1e30)
LN2 = f32(0.69314718055994531)
MM, IM, DM, BM, MI, II, MD, DD = range(8)

libm = C.CDLL("libm.so.6")
for fn in ("expf", "log1pf", "logf"):
    getattr(libm, fn).restype = C.c_float
    getattr(libm, fn).argtypes = [C.c_float]


def test_log1pexp_every_float():
    lib = L.load()
    hi, chunk = 0x42480000 + 1, 1 << 27  # bit patterns of 0 .. 50
    a, b = np.empty(chunk, f32), np.empty(chunk, f32)
    for lo in range(0, hi, chunk):
        n = min(chunk, hi - lo)
        assert lib.pl_rc_mathf_eval(0, 6, lo, 1, n, a.ctypes.data) == 1
        assert lib.pl_rc_mathf_eval(0, 7, lo, 1, n, b.ctypes.data) == 1
        bad = a[:n].view(np.uint32) != b[:n].view(np.uint32)
        assert not bad.any(), hex(lo + int(np.argmax(bad)))


def _ls(a, b):
    mx, mn = (a, b) if a > b else (b, a)
    d = f32(mn - mx)
    if mn <= NEG or d < f32(-50):
        return mx
    return f32(mx + f32(libm.log1pf(libm.expf(d))))


def _score(msc, tsc, x, null2):
    M, n = len(msc), len(x)
    p1 = f32(f32(n) / f32(n + 1))
    null1 = f32(f32(f32(n) * f32(libm.logf(p1))) + f32(libm.logf(f32(f32(1) - p1))))
    pm = f32(f32(3) / f32(n + 3))
    move, loop, lE = f32(libm.logf(pm)), f32(libm.logf(f32(f32(1) - pm))), f32(-LN2)
    t = [[f32(v) for v in r] for r in tsc]
    F = [([NEG] * (M + 1), [NEG] * (M + 1))]
    D = [NEG] * (M + 1)
    xN, xB, xJ, xC = f32(0), move, NEG, NEG
    S = [(xN, xJ, xC)]
    for i in range(1, n + 1):
        pM, pI = F[-1]
        m, ins, d = [NEG] * (M + 1), [NEG] * (M + 1), [NEG] * (M + 1)
        E = NEG
        for k in range(1, M + 1):
            r = t[k - 1]
            s = _ls(_ls(f32(pM[k - 1] + r[MM]), f32(pI[k - 1] + r[IM])), _ls(f32(xB + r[BM]), f32(D[k - 1] + r[DM])))
            m[k] = f32(s + f32(msc[k - 1][x[i - 1]]))
            if k < M:
                ins[k] = _ls(f32(pM[k] + r[MI]), f32(pI[k] + r[II]))
            if k > 1:
                d[k] = _ls(f32(m[k - 1] + t[k - 2][MD]), f32(d[k - 1] + t[k - 2][DD]))
            E = _ls(E, _ls(m[k], d[k]))
        xJ, xC = _ls(f32(xJ + loop), f32(E + lE)), _ls(f32(xC + loop), f32(E + lE))
        xN = f32(xN + loop)
        xB = _ls(f32(xN + move), f32(xJ + move))
        F.append((m, ins))
        S.append((xN, xJ, xC))
        D = d
    tot = f32(xC + move)
    bias = f32(0)
    if null2:
        bias = _bias(msc, t, x, F, S, move, loop, lE, tot)
    return f32(f32(f32(tot - null1) - bias) / LN2), f32(bias / LN2)


def _bias(msc, t, x, F, S, move, loop, lE, tot):
    M, n = len(msc), len(x)
    logL = f32(libm.logf(f32(n)))
    bC, bJ, bN = move, NEG, NEG
    bE = f32(bC + lE)
    m, ins, d = [NEG] * (M + 2), [NEG] * (M + 2), [NEG] * (M + 2)
    m[M] = d[M] = bE
    for k in range(M - 1, 0, -1):
        m[k], d[k] = _ls(bE, f32(d[k + 1] + t[k - 1][MD])), _ls(bE, f32(d[k + 1] + t[k - 1][DD]))
    B, T = {n: (m, ins)}, {n: (bN, bJ, bC)}
    for i in range(n - 1, 0, -1):
        pm, pi = m, ins
        e = lambda k: f32(msc[k - 1][x[i]])
        bB = NEG
        for k in range(1, M + 1):
            bB = _ls(bB, f32(f32(pm[k] + t[k - 1][BM]) + e(k)))
        bJ, bC, bN = _ls(f32(bJ + loop), f32(bB + move)), f32(bC + loop), _ls(f32(bN + loop), f32(bB + move))
        bE = _ls(f32(bJ + lE), f32(bC + lE))
        m, ins, d = [NEG] * (M + 2), [NEG] * (M + 2), [NEG] * (M + 2)
        m[M] = d[M] = bE
        for k in range(M - 1, 0, -1):
            n1 = f32(pm[k + 1] + e(k + 1))
            d[k] = _ls(f32(n1 + t[k][DM]), _ls(f32(d[k + 1] + t[k - 1][DD]), bE))
            m[k] = _ls(_ls(f32(n1 + t[k][MM]), f32(pi[k] + t[k - 1][MI])), _ls(bE, f32(d[k + 1] + t[k - 1][MD])))
            ins[k] = _ls(f32(n1 + t[k][IM]), f32(pi[k] + t[k - 1][II]))
        B[i], T[i] = (m, ins), (bN, bJ, bC)
    um, ui, us = [NEG] * (M + 1), [NEG] * (M + 1), [NEG] * 3
    for i in range(1, n + 1):
        for k in range(1, M + 1):
            um[k] = _ls(um[k], f32(F[i][0][k] + B[i][0][k]))
            if k < M:
                ui[k] = _ls(ui[k], f32(F[i][1][k] + B[i][1][k]))
        us = [_ls(us[j], f32(f32(S[i - 1][j] + T[i][j]) + loop)) for j in range(3)]
    xfac = f32(f32(_ls(_ls(us[0], us[1]), us[2]) - tot) - logL)
    li = NEG
    for k in range(1, M):
        li = _ls(li, f32(f32(ui[k] - tot) - logL))
    v = [_ls(xfac, li)] * 20
    for k in range(1, M + 1):
        u = f32(f32(um[k] - tot) - logL)
        v = [_ls(v[c], f32(u + f32(msc[k - 1][c]))) for c in range(20)]
    lx = f32(np.log(np.exp(np.array(v, np.float64)).sum() / 20.0))
    a = np.log(1.0 / 256.0) + float(sum(float(v[c]) if c < 20 else float(lx) for c in x))
    return f32(a + np.log1p(np.exp(-a)) if a > 0 else np.log1p(np.exp(a)))


def _profile(rng, M):
    msc = rng.normal(-0.5, 1.2, (M, 21)).astype(f32)
    p = rng.dirichlet([8, 1, 1], M)
    q, r = rng.uniform(0.2, 0.8, M), rng.uniform(0.2, 0.8, M)
    cols = [p[:, 0], q, r, np.full(M, 2.0 / (M * (M + 1.0))), p[:, 1], 1 - q, p[:, 2], 1 - r]
    return msc, np.log(np.stack(cols, axis=1)).astype(f32)


@pytest.mark.parametrize("null2", [False, True])
@pytest.mark.parametrize("M,lens", [(1, (1, 2, 5)), (2, (3, 1)), (3, (4, 2, 1)), (15, (6,)), (16, (1,)), (17, (5, 2)),
                                    (31, (3,)), (32, (4, 1)), (33, (2, 7)), (34, (3, 3)), (49, (5, 4, 1)), (66, (6, 2))])
def test_passes_at_their_edges(M, lens, null2):
    rng = np.random.default_rng(100 * M + len(lens))
    msc, tsc = _profile(rng, M)
    seqs = [rng.integers(0, 21, n).astype(np.uint8) for n in lens]
    want = [_score(msc, tsc, s, null2) for s in seqs]
    prof, eng = L.RcProfile(msc, tsc), L.Engine(0)
    for n in (1, len(seqs), 32, 40):  # peptides: one lane, a few, a full group, a group and a part
        pick = [int(q) for q in rng.integers(0, len(seqs), n)]
        bits, bias = eng.rc_score([prof], [(0, seqs[q]) for q in pick], null2)
        for j, q in enumerate(pick):
            wb, ws = want[q]
            if not null2:
                assert (bits[j], bias[j]) == (wb, f32(0)), (M, n, q)
                continue
            ulp = float(np.spacing(abs(ws))) * 2  # one unit in the bias in nats, one in its division
            assert abs(float(bias[j]) - float(ws)) <= ulp, (M, n, q)
            assert abs(float(bits[j]) - float(wb)) <= ulp + 2 * float(np.spacing(abs(wb))), (M, n, q)
    eng.close()
    prof.close()
