"""The chaining DP's precomputed score rows (the 32 predecessors before an anchor) and the walk past
them: f, p and v of every anchor against the restatement, on queries of 0, 1, 31-34 and more
anchors, windows much longer than a row (large max_skip), the best anchor so far inside and
outside the row, and more queries than one launch's warps."""
import ctypes as C

import numpy as np
import pytest

import chain_ref as CR
from protlocus_b200 import lib as L
from protlocus_b200.abi import chain_opt, chain_opt_struct

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _query(rng, n, blocks, qlen):
    a = (rng.integers(0, blocks, 2 * n + 4).astype(np.uint64) << np.uint64(32)) | rng.integers(0, qlen, 2 * n + 4).astype(np.uint64)
    return np.unique(a)[:n] if n else np.zeros(0, np.uint64)


@pytest.mark.parametrize("opt", [
    chain_opt("main"), chain_opt("pre"), dict(chain_opt("main"), max_skip=400),
    dict(chain_opt("main"), max_skip=400, max_iter=40), dict(chain_opt("main"), max_skip=1),
    dict(chain_opt("main", max_intron=4000, bbit=0, kmer=5), max_skip=60),
    dict(chain_opt("main"), is_spliced=0, bw=3000, max_dist_x=5000, max_skip=100)],
    ids=["main", "pre", "wide", "wide_iter", "skip1", "nucleotide", "unspliced"])
def test_fill(opt):
    rng = np.random.default_rng(opt["max_skip"] + opt["bbit"])
    scale = 1 if opt["bbit"] else 256
    qs = [_query(rng, n, b * scale, q) for n in (0, 1, 2, 31, 32, 33, 34, 64, 65, 200, 400)
          for b, q in ((60, 300), (400, 900), (6, 200))]
    qs += [_query(rng, int(rng.integers(1, 20)), 300 * scale, 400) for _ in range(60)]
    eng = L.Engine(0)
    try:
        off, n, a = L.chain_pack(qs)
        d_a = torch.from_numpy(a.view(np.int64).copy()).cuda()
        d_f, d_p, d_v = (torch.full((len(a),), -7, dtype=torch.int32, device="cuda") for _ in range(3))
        o = chain_opt_struct(opt)
        torch.cuda.synchronize()
        assert eng.lib.pl_chain_fill_device(eng.h, C.byref(o), len(qs), off.ctypes.data, n.ctypes.data, d_a.data_ptr(),
                                            len(a), d_f.data_ptr(), d_p.data_ptr(), d_v.data_ptr(), None), L.error()
        f, p, v = d_f.cpu().numpy(), d_p.cpu().numpy(), d_v.cpu().numpy()
    finally:
        eng.close()
    linked = 0
    for q, x in enumerate(qs):
        wf, wp, wv = CR.fill(x, opt)
        s = slice(int(off[q]), int(off[q]) + len(x))
        assert np.array_equal(f[s], wf) and np.array_equal(p[s], wp) and np.array_equal(v[s], wv), (q, len(x))
        linked += int((wp >= 0).sum())
    assert linked > 50
