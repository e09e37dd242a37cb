"""The chaining DP past the anchors whose score rows are held at once (4 M): a single query longer
than that, and batches whose queries go on over several launches.  The queries are copies of short
ones, further along the genome than a chain reaches, so that every copy's f, p and v are the short
one's (p counted from the copy's first anchor), which the restatement gives.  The scratch memory of
a call stays at 16 bytes an anchor and the 512 MB of rows."""
import ctypes as C

import numpy as np
import pytest

import chain_ref as CR
from protlocus_b200 import lib as L
from protlocus_b200.abi import chain_opt, chain_opt_struct

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROWS = 4 << 20  # anchors


def _short(rng, n, blocks):
    a = (rng.integers(0, blocks, 2 * n + 4).astype(np.uint64) << np.uint64(32)) | rng.integers(0, 300, 2 * n + 4).astype(np.uint64)
    return np.unique(a)[:n]


@pytest.mark.parametrize("copies,queries,blocks", [(90000, 1, 300), (1200, 60, 40), (1, 140000, 40), (40, 2000, 40)])
def test_fill_over_launches(copies, queries, blocks):
    rng = np.random.default_rng(copies)
    opt = chain_opt("main", max_intron=4000)
    base = [_short(rng, int(m), blocks) for m in rng.integers(70, 90, 8)]
    step = (1 << 17) // 256  # blocks between copies: past max_dist_x
    want = [CR.fill(x, opt) for x in base]
    qs, ref = [], []
    for q in range(queries):
        pick = rng.integers(0, 8, max(1, copies - int(rng.integers(0, 1 + copies // 8))))
        lens = np.array([len(base[k]) for k in pick])
        at = np.repeat(np.arange(len(pick), dtype=np.uint64) * np.uint64(step), lens)
        qs.append(np.concatenate([base[k] for k in pick]) + (at << np.uint64(32)))
        ref.append((pick, lens))
    n = np.array([len(x) for x in qs], np.int32)
    off = np.concatenate([[0], np.cumsum(n[:-1], dtype=np.int64)]).astype(np.int64)
    a = np.concatenate(qs)
    assert len(a) > ROWS
    d_a = torch.from_numpy(a.view(np.int64)).cuda()
    d_f, d_p, d_v = (torch.full((len(a),), -7, dtype=torch.int32, device="cuda") for _ in range(3))
    o = chain_opt_struct(opt)
    eng = L.Engine(0)
    try:
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        assert eng.lib.pl_chain_fill_device(eng.h, C.byref(o), len(qs), off.ctypes.data, n.ctypes.data, d_a.data_ptr(),
                                            len(a), d_f.data_ptr(), d_p.data_ptr(), d_v.data_ptr(), None), L.error()
        used = free - torch.cuda.mem_get_info()[0]
    finally:
        eng.close()
    f, p, v = d_f.cpu().numpy(), d_p.cpu().numpy(), d_v.cpu().numpy()
    for q, (pick, lens) in enumerate(ref):
        s = slice(int(off[q]), int(off[q]) + int(n[q]))
        first = np.repeat(np.concatenate([[0], np.cumsum(lens[:-1])]), lens)
        wf, wp, wv = (np.concatenate([want[k][x] for k in pick]) for x in range(3))
        assert np.array_equal(f[s], wf) and np.array_equal(v[s], wv), q
        assert np.array_equal(p[s], np.where(wp >= 0, wp + first, -1)), q
    # off, n, order, state and row0 of a query: 40 bytes; 64 MB for the allocator's granularity
    assert used <= 128 * ROWS + 16 * len(a) + 40 * len(qs) + (64 << 20), used >> 20
