"""The work that programs have this framework do, as timed cases.

Every case is one call (or the calls that belong together) of a public entry point on
synthetic data of the shapes of the benchmark workloads: the mapper's stages from seeding
to the exact spliced DP, the profile-HMM paths, and the learned prefilter in both
directions.  `listed()` gives one case of each kind, the smallest a single alignment and
the largest the batched global DP of 8192 jobs; `draw()` gives cases of the same kinds
over their whole ranges, down to a handful of jobs.

All generators draw whole batches at once (one protein string, one nucleotide array), so
a state is made in about a second.  Operation counts in `work()` are integer lane
operations per DP cell for the DPs (the counts bench.py reports against) and floating
point operations elsewhere.
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import os

import numpy as np
import torch

from protlocus_b200 import hmm as H
from protlocus_b200 import lib as L
from protlocus_b200 import prefilter as P
from protlocus_b200 import workload as W
from protlocus_b200.abi import (BLOSUM62, CODE1, NS_F_CIGAR, NS_F_EXT_LEFT, NS_F_EXT_RIGHT, NS_S_GENERIC,
                                NS_S_MAMMAL, Options, chain_opt, chain_opt_struct, make_tables)

JOB = P.JOB_DTYPE
EXT_JOB = np.dtype([("nt_off", "<i8"), ("aa_off", "<i8"), ("ss_off", "<i8"), ("pssm_off", "<i8"),
                    ("nl", "<i4"), ("al", "<i4"), ("flag", "<i4"), ("width", "<i4")])
NT = np.frombuffer(b"ACGT", np.uint8)
COMP = np.zeros(256, np.uint8)
COMP[np.frombuffer(b"ACGT", np.uint8)] = np.frombuffer(b"TGCA", np.uint8)


def listed():
    return [
        # one protein against one 20 kb window through the request API: the latency a single caller sees
        {"name": "splice_locus", "kind": "splice_locus", "al": 500, "window": 20000, "model": "generic"},
        # a queue's worth of short gap-filling alignments of one mapping thread pool, host buffers, one strand
        {"name": "splice_queue", "kind": "splice_host", "n": 96, "al": 80, "al_max": 150, "win_min": 300,
         "win_max": 3000, "tracks": False, "model": "generic"},
        # the batched workload: 4096 loci searched on both strands, 1-50 kb windows, device buffers
        {"name": "splice_strands", "kind": "splice_strands", "pairs": 4096, "al": 350, "win_max": 50000},
        # loci whose strand is known, with splice-score tracks (a species model), host buffers
        {"name": "splice_tracks", "kind": "splice_host", "n": 509, "al": 350, "al_max": 2500, "win_min": 1000,
         "win_max": 50000, "tracks": True, "model": "mammal"},
        # terminal extensions, both directions mixed, a whole batch on the device
        {"name": "ext_batch", "kind": "ext", "n": 65536, "win_max": 256, "tracks": False},
        # gapless ranking of coarse chains: 8 anchors per candidate on a 100 Mb genome
        {"name": "gapless", "kind": "gapless", "n": 131072, "anchors": 8, "genome": 100_000_000, "genes": 10000},
        # profile search: many profiles against a six-frame genome slice
        {"name": "hmm_scan", "kind": "hmm", "profiles": 64, "slice": 2_000_000, "region": 12000, "m_max": 800},
        # recheck of reported peptides against their profiles, with the composition bias correction
        {"name": "recheck", "kind": "recheck", "profiles": 96, "n": 4000, "len_max": 600, "m_max": 800, "null2": True},
        # seeding of a protein set against a 100 Mb genome's index, the anchors left on the device
        {"name": "seed", "kind": "seed", "n": 10000, "al": 350, "max_occ": 20000},
        # chaining of the seed anchors of a protein set, host buffers
        {"name": "chain", "kind": "chain", "n": 10000, "al": 350},
        # the learned selection of candidates (features, network, decision)
        {"name": "pf_select", "kind": "pf_select", "proteins": 2048, "al": 350},
        # its training: Adam steps of 4096 rows
        {"name": "pf_train", "kind": "pf_train", "batch": 4096, "steps": 16, "rows": 40960},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["splice_locus", "splice_host", "splice_host", "splice_strands", "ext", "gapless", "hmm",
                       "recheck", "seed", "chain", "pf_select", "pf_train"])
    if kind == "splice_locus":
        return {"kind": kind, "al": _log(rng, 20, 1500), "window": _log(rng, 700, 50000),
                "model": rng.choice(["generic", "mammal"])}
    if kind == "splice_host":
        short = rng.random() < 0.5
        return {"kind": kind, "n": _log(rng, 3, 128) if short else _log(rng, 8, 768), "al": 80 if short else 350,
                "al_max": 150 if short else 2500, "win_min": 300 if short else 1000,
                "win_max": 3000 if short else _log(rng, 4000, 50000), "tracks": rng.random() < 0.5,
                "model": rng.choice(["generic", "mammal"])}
    if kind == "splice_strands":
        return {"kind": kind, "pairs": _log(rng, 8, 2500), "al": 350, "win_max": _log(rng, 5000, 50000)}
    if kind == "ext":
        return {"kind": kind, "n": _log(rng, 100, 65536), "win_max": rng.choice([100, 256]),
                "tracks": rng.random() < 0.3}
    if kind == "gapless":
        return {"kind": kind, "n": _log(rng, 300, 131072), "anchors": rng.choice([3, 8]),
                "genome": _log(rng, 2_000_000, 100_000_000), "genes": _log(rng, 100, 1500)}
    if kind == "hmm":
        return {"kind": kind, "profiles": _log(rng, 1, 64), "slice": _log(rng, 60_000, 2_000_000),
                "region": rng.choice([3001, 12000, 30000]), "m_max": rng.choice([300, 800, 1100])}
    if kind == "recheck":
        return {"kind": kind, "profiles": _log(rng, 1, 96), "n": _log(rng, 40, 4000), "len_max": rng.choice([200, 600]),
                "m_max": rng.choice([300, 800]), "null2": rng.random() < 0.7}
    if kind == "seed":
        return {"kind": kind, "n": _log(rng, 20, 10000), "al": 350, "max_occ": rng.choice([200, 20000])}
    if kind == "chain":
        return {"kind": kind, "n": _log(rng, 50, 10000), "al": rng.choice([200, 350])}
    if kind == "pf_select":
        return {"kind": kind, "proteins": _log(rng, 20, 2048), "al": 350}
    batch = 128 * rng.randint(2, 32)
    return {"kind": kind, "batch": batch, "steps": rng.randint(3, 20), "rows": batch * rng.randint(3, 10)}


# ------------------------------------------------------------------------------ generators

def _lengths(rng, n, median, sigma=0.6, lo=50, hi=2500):
    return np.clip(np.round(np.exp(rng.normal(math.log(median), sigma, n))), lo, hi).astype(np.int64)


def _starts(lens):
    out = np.zeros(len(lens), np.int64)
    if len(lens) > 1:
        out[1:] = np.cumsum(lens[:-1])
    return out


def _genes(rng, al, intron_lambda=4.0, intron_median=150.0, intron_cap=20000, frameshifts=2, divergence=0.25):
    """Spliced, diverged, frameshifted genes of proteins of `al` residues.  Returns the
    proteins (one byte array), every coding base with its gene and its position inside the
    gene, the genes' lengths, and the introns (gene, first and last base) for their GT..AG."""
    n, tot = len(al), int(al.sum())
    prot = W.random_protein(rng, tot)
    cds = np.frombuffer(W.reverse_translate(rng, W.mutate(rng, prot, divergence)).encode(), np.uint8)
    gene = np.repeat(np.arange(n), 3 * al)
    first = 3 * _starts(al)
    k = np.minimum(rng.poisson(intron_lambda, n), np.maximum(al // 8, 0))
    ig = np.repeat(np.arange(n), k)
    cut = (6 + rng.random(len(ig)) * (3 * al[ig] - 12)).astype(np.int64)
    ilen = np.clip(np.round(np.exp(rng.normal(math.log(intron_median), 0.8, len(ig)))), 20, intron_cap).astype(np.int64)
    shift = np.zeros(3 * tot, np.int64)
    np.add.at(shift, first[ig] + cut, ilen)
    if frameshifts:
        fg = np.repeat(np.arange(n), rng.integers(0, frameshifts + 1, n))
        fc = (3 + rng.random(len(fg)) * (3 * al[fg] - 6)).astype(np.int64)
        np.add.at(shift, first[fg] + fc, np.where(rng.random(len(fg)) < 0.5, 1, -1))
    run = np.cumsum(shift)
    run -= (run[first] - shift[first])[gene]
    pos = np.maximum(np.arange(3 * tot) - first[gene] + run, 0)
    glen = np.zeros(n, np.int64)
    np.maximum.at(glen, gene, pos + 1)
    i_end = pos[first[ig] + cut] - 1
    return np.frombuffer(prot.encode(), np.uint8), cds, gene, pos, glen, (ig, np.maximum(i_end - ilen + 1, 0), i_end)


def _windows(rng, al, win_min, win_max, **kw):
    """One genomic window per protein holding its gene: (proteins, windows, window lengths)."""
    prot, cds, gene, pos, glen, (ig, i0, i1) = _genes(rng, al, **kw)
    wl = np.maximum(rng.integers(win_min, win_max + 1, len(al)), glen + 200)
    off = _starts(wl)
    base = off + 100 + (rng.random(len(al)) * (wl - glen - 199)).astype(np.int64)
    nt = NT[rng.integers(0, 4, int(wl.sum()), dtype=np.uint8)]
    nt[base[gene] + pos] = cds
    ok = i1 - i0 >= 7
    for at, ch in ((i0, b"G"), (i0 + 1, b"T"), (i1 - 1, b"A"), (i1, b"G")):
        nt[(base[ig] + at)[ok]] = ch[0]
    return prot, nt, wl


def _revcomp(nt, wl):
    """Every window's reverse complement, windows in the same order."""
    off = _starts(wl)
    w = np.repeat(np.arange(len(wl)), wl)
    return COMP[nt[(2 * off + wl - 1)[w] - np.arange(len(nt))]]


def _tracks(rng, n):
    """Splice-score tracks: 20 % of the positions carry a donor or acceptor score."""
    v = rng.integers(0, 256, n, dtype=np.uint8)
    return np.where(rng.integers(0, 5, n, dtype=np.uint8) == 0, v, 0xff).astype(np.uint8)


def _options(model, flag=NS_F_CIGAR):
    return Options(flag=flag, sp_model=NS_S_MAMMAL if model == "mammal" else NS_S_GENERIC)


def _jobs(dtype, nl, al, nt_off, aa_off):
    j = np.zeros(len(nl), dtype)
    j["nt_off"], j["aa_off"], j["ss_off"], j["nl"], j["al"] = nt_off, aa_off, -1, nl, al
    return j


def _dev(a):
    return torch.from_numpy(np.array(a)).to("cuda")


def _pinned(a):
    return torch.from_numpy(np.array(a)).pin_memory()


def _check(ok, what):
    if not ok:
        raise RuntimeError(what + ": " + L.error())


def _stream():
    return torch.cuda.current_stream().cuda_stream


# ------------------------------------------------------------------------------ profiles

def _profile_tables(rng, n, m_max):
    """Match emissions and transitions of n Plan7 profiles of 50..m_max states."""
    out = []
    for _ in range(n):
        m = int(rng.integers(50, m_max + 1))
        mat = rng.dirichlet(W.P7_BG * 20.0, size=m) + 1e-5
        mat /= mat.sum(axis=1, keepdims=True)
        mm = np.clip(rng.normal(0.95, 0.02, m), 0.80, 0.995)
        mi = (1 - mm) * rng.uniform(0.3, 0.7, m)
        im = np.clip(rng.normal(0.6, 0.1, m), 0.2, 0.95)
        dm = np.clip(rng.normal(0.7, 0.1, m), 0.2, 0.95)
        out.append((mat, np.stack([mm, mi, 1 - mm - mi, im, 1 - im, dm, 1 - dm], axis=1)))
    return out


def _int_tables(mat, tr):
    """The integer profile of the HMM DP: twice the log probabilities, best emission +4."""
    e = np.rint(2.0 * np.log(mat)).astype(np.int64)
    e = e - e.max(axis=1, keepdims=True) + 4
    return e.astype(np.int16), np.rint(2.0 * np.log(tr)).astype(np.int16)


def _float_tables(mat, tr):
    """The recheck's search profile: match log-odds (column 20 degenerate) and transitions
    in the order MM, IM, DM, BM, MI, II, MD, DD, uniform local entry."""
    m = len(mat)
    msc = np.zeros((m, 21))
    msc[:, :20] = np.log(mat / W.P7_BG)
    msc[:, 20] = (msc[:, :20] * W.P7_BG).sum(axis=1)
    t = np.log(tr)
    bm = np.full(m, math.log(2.0 / (m * (m + 1.0))))
    tsc = np.stack([t[:, 0], t[:, 3], t[:, 5], bm, t[:, 1], t[:, 4], t[:, 2], t[:, 6]], axis=1)
    return msc.astype(np.float32), tsc.astype(np.float32)


def _sample(rng, mat, a, b):
    """Residues (HMMER codes) of a domain of states a..b-1."""
    return (rng.random(b - a)[:, None] > np.cumsum(mat[a:b], axis=1)).sum(axis=1).clip(0, 19).astype(np.uint8)


# ------------------------------------------------------------------------------ prepare

def prepare(case, seed):
    rng = np.random.default_rng(seed)
    return globals()["_prepare_" + case["kind"]](case, rng)


def _prepare_splice_locus(c, rng):
    prot, nt, _ = _windows(rng, np.array([c["al"]]), c["window"], c["window"], intron_lambda=3.0)
    if not L.gpu_init(0):
        raise RuntimeError("ns_gpu_init")
    return {"kind": c["kind"], "nt": nt.tobytes(), "aa": prot.tobytes(), "opt": _options(c["model"]),
            "cigar": np.zeros(c["window"] + c["al"] + 8, np.uint32)}


def _prepare_splice_host(c, rng):
    al = _lengths(rng, c["n"], c["al"], lo=20, hi=c["al_max"])
    prot, nt, wl = _windows(rng, al, c["win_min"], c["win_max"], intron_lambda=1.0 if c["al"] < 100 else 4.0)
    jobs = _jobs(JOB, wl, al, _starts(wl), _starts(al))
    ss = _tracks(rng, len(nt)) if c["tracks"] else None
    if c["tracks"]:
        jobs["ss_off"] = jobs["nt_off"]
    cap = 512 * c["n"] + 65536
    return {"kind": c["kind"], "eng": L.Engine(0), "opt": _options(c["model"]), "jobs": jobs, "nt": _pinned(nt),
            "aa": _pinned(prot), "ss": _pinned(ss) if ss is not None else None,
            "res": torch.zeros(len(al) * 24, dtype=torch.uint8).pin_memory(),
            "cig": torch.zeros(cap, dtype=torch.int32).pin_memory()}


@functools.cache
def _batch_engine():
    """The engine of a program that aligns batch after batch: one for the process, with the
    72 GB of trace memory that pl_engine_create gives an otherwise empty card."""
    return L.Engine(0, 72 << 30)


def _prepare_splice_strands(c, rng):
    al = _lengths(rng, c["pairs"], c["al"])
    prot, nt, wl = _windows(rng, al, 1000, c["win_max"])
    n = 2 * len(al)
    jobs = _jobs(JOB, np.repeat(wl, 2), np.repeat(al, 2), 0, np.repeat(_starts(al), 2))
    jobs["nt_off"][0::2], jobs["nt_off"][1::2] = _starts(wl), _starts(wl) + len(nt)
    cap = 512 * n + 65536
    return {"kind": c["kind"], "eng": _batch_engine(), "opt": _options("generic"), "jobs": jobs,
            "nt": _dev(np.concatenate([nt, _revcomp(nt, wl)])), "aa": _dev(prot), "ss": None,
            "res": torch.zeros(n * 24, dtype=torch.uint8, device="cuda"),
            "cig": torch.zeros(cap, dtype=torch.int32, device="cuda"), "cap": cap}


def _prepare_ext(c, rng):
    n = c["n"]
    al = rng.integers(min(64, c["win_max"] // 2), c["win_max"] + 1, n)
    part = np.maximum(8, (al * rng.uniform(0.3, 1.0, n)).astype(np.int64))
    left = np.arange(n) % 2 == 1
    prot, cds, gene, pos, glen, (ig, i0, i1) = _genes(rng, al, intron_lambda=0.5, intron_cap=2000, frameshifts=1)
    # the anchored part of the gene is kept, at the window's anchor end; the rest stays random
    idx = np.arange(len(cds)) - 3 * _starts(al)[gene]
    keep = np.where(left[gene], idx >= 3 * (al - part)[gene], idx < 3 * part[gene])
    wl = np.maximum(3 * al, glen) + rng.integers(60, 601, n)
    off = _starts(wl)
    base = off + np.where(left, wl - glen, 0)
    nt = NT[rng.integers(0, 4, int(wl.sum()), dtype=np.uint8)]
    nt[(base[gene] + pos)[keep]] = cds[keep]
    for at, ch in ((i0, b"G"), (i0 + 1, b"T"), (i1 - 1, b"A"), (i1, b"G")):
        nt[base[ig] + at] = ch[0]
    jobs = _jobs(EXT_JOB, wl, al, off, _starts(al))
    jobs["pssm_off"] = -1
    jobs["flag"] = np.where(left, NS_F_EXT_LEFT, NS_F_EXT_RIGHT)
    ss = None
    if c["tracks"]:
        ss, jobs["ss_off"] = _dev(_tracks(rng, len(nt))), off
    return {"kind": c["kind"], "eng": L.Engine(0), "opt": _options("generic", 0), "jobs": jobs, "nt": _dev(nt),
            "aa": _dev(prot), "ss": ss, "res": torch.zeros(n * 16, dtype=torch.uint8, device="cuda")}


def _prepare_gapless(c, rng):
    al, n_contig = 500, 64
    nt4, aa20, codon = make_tables()
    glen = c["genome"] // n_contig * n_contig
    clen = glen // n_contig
    genome = rng.choice(4, size=glen, p=[0.275, 0.225, 0.225, 0.275]).astype(np.uint8)
    n_g = max(1, min(c["genes"], glen // 12000))
    prot, cds, gene, pos, span, _ = _genes(rng, np.full(n_g, al), intron_lambda=3.0, intron_cap=2000, frameshifts=0)
    slot = glen // n_g
    start = np.arange(n_g) * slot + (rng.random(n_g) * np.maximum(slot - span, 1)).astype(np.int64)
    ctg = start // clen
    start = np.maximum(np.minimum(start, (ctg + 1) * clen - span - 1), ctg * clen)
    rev = rng.random(n_g) < 0.5
    codes = nt4[cds]
    at = start[gene] + np.where(rev[gene], span[gene] - 1 - pos, pos)
    genome[at] = np.where(rev[gene], 3 - codes, codes)
    # last base of every codon in the oriented coordinates of its contig
    ends = pos.reshape(-1, 3)[:, 2].reshape(n_g, al) + \
        np.where(rev, (ctg + 1) * clen - start - span, start - ctg * clen)[:, None]
    n, k = c["n"], c["anchors"]
    g = rng.integers(0, n_g, n)
    true = rng.random(n) < 0.3
    cc = np.where(true, ctg[g], rng.integers(0, n_contig, n))
    cr = np.where(true, rev[g], rng.random(n) < 0.5)
    qe = np.sort(rng.integers(5, al, (n, k)), axis=1)
    tp = np.where(true[:, None], ends[g[:, None], qe] - rng.integers(0, 7, n)[:, None], rng.integers(0, clen, (n, k)))
    cand = np.zeros(n, W.GAPLESS_CAND_DTYPE)
    cand["target_offset"], cand["target_length"], cand["query_offset"] = cc * clen, clen, g * al
    cand["query_length"], cand["anchor_offset"], cand["anchor_count"] = al, np.arange(n) * k, k
    cand["reverse"] = cr
    anc = np.zeros(n * k, W.GAPLESS_ANCHOR_DTYPE)
    anc["target_block"] = ((np.clip(tp, 0, clen - 1) >> 8) << 8).reshape(-1)
    anc["query_end"] = qe.reshape(-1)
    q = aa20[prot]
    return {"kind": c["kind"], "eng": L.Engine(0), "mat": Options().mat, "codon": codon, "bases": glen,
            "packed": _dev(W.pack_nt4(genome)), "queries": _dev(q), "cand": _dev(cand.view(np.uint8)),
            "anc": _dev(anc.view(np.uint8)), "n": n, "na": n * k, "nq": len(q),
            "score": torch.zeros(n, dtype=torch.int32, device="cuda")}


def _hmm_step(region):
    """Windows overlap by 2.4 kb (a domain of 800 codons lies inside one), small ones by half."""
    return max(region - 2400, region // 2)


def _prepare_hmm(c, rng):
    tabs = _profile_tables(rng, c["profiles"], c["m_max"])
    g = rng.choice(4, size=c["slice"], p=[0.275, 0.225, 0.225, 0.275]).astype(np.uint8)
    for _ in range(max(1, c["slice"] // 30000)):
        mat = tabs[int(rng.integers(0, len(tabs)))][0]
        dom = _sample(rng, mat, 0, len(mat))
        cds = H.nt4(W.reverse_translate(rng, "".join(H.ALPHABET[int(x)] for x in dom)).encode())
        if rng.random() < 0.5:
            cds = 3 - cds[::-1]
        if len(cds) < len(g):
            at = int(rng.integers(0, len(g) - len(cds)))
            g[at:at + len(cds)] = cds
    parts = []
    for strand in (g, 3 - g[::-1]):
        for st in range(0, max(1, len(strand) - 2400), _hmm_step(c["region"])):
            w = strand[st:st + c["region"]]
            parts += [w[f:] for f in range(3)]
    lens = np.array([len(x) for x in parts], np.int32)
    ca = H.codon_alpha()
    profs = [L.HmmProfile(*_int_tables(*t), ca, 0) for t in tabs]
    return {"kind": c["kind"], "eng": L.Engine(0), "profs": profs, "n": len(lens),
            "handles": (C.c_void_p * len(profs))(*[p.h for p in profs]), "nt": _dev(np.concatenate(parts)),
            "off": _starts(lens).astype(np.int32), "len": lens,
            "score": torch.zeros(len(profs) * len(lens), dtype=torch.int32, device="cuda")}


def _recheck_inputs(c, rng):
    tabs = _profile_tables(rng, c["profiles"], c["m_max"])
    pid = np.sort(rng.integers(0, len(tabs), c["n"])).astype(np.int32)
    lens = rng.integers(30, c["len_max"] + 1, c["n"]).astype(np.int32)
    off = _starts(lens)
    dsq = rng.choice(20, size=int(lens.sum()), p=W.P7_BG).astype(np.uint8)
    for q in range(0, c["n"], 2):  # a reported peptide carries (part of) its domain
        mat = tabs[pid[q]][0]
        k = int(min(len(mat), lens[q]))
        a = int(rng.integers(0, len(mat) - k + 1))
        o = off[q] + int(rng.integers(0, lens[q] - k + 1))
        dsq[o:o + k] = _sample(rng, mat, a, a + k)
    dsq[rng.integers(0, len(dsq), max(1, len(dsq) // 1000))] = 20
    return [_float_tables(*t) for t in tabs], pid, lens, off, dsq


def _prepare_recheck(c, rng):
    tabs, pid, lens, off, dsq = _recheck_inputs(c, rng)
    profs = [L.RcProfile(m, t, 0) for m, t in tabs]
    return {"kind": c["kind"], "eng": L.Engine(0), "profs": profs, "null2": int(c["null2"]), "pid": pid, "len": lens,
            "handles": (C.c_void_p * len(profs))(*[p.h for p in profs]), "off": off, "dsq": dsq,
            "bits": np.zeros(c["n"], np.float32), "bias": np.zeros(c["n"], np.float32)}


class _Index(L.SeedIndex):
    def __del__(self):
        self.close()


def _prepare_seed(c, rng):
    n_bucket = 1 << 23
    cnt = rng.poisson(12.0, size=n_bucket).astype(np.int64)
    cnt[rng.choice(n_bucket, size=256, replace=False)] = rng.integers(10000, 30000, size=256)
    # the mapper's index keeps each bucket's blocks ascending
    kb = rng.integers(0, (100_000_000 >> 8) * 2, size=int(cnt.sum()), dtype=np.uint32)
    key = torch.from_numpy(np.repeat(np.arange(n_bucket, dtype=np.int64) << 32, cnt) | kb).to("cuda")
    kb = (torch.sort(key).values & 0xffffffff).cpu().numpy().astype(np.uint32)
    del key
    al = _lengths(rng, c["n"], c["al"], 0.7)
    seq = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", np.uint8)[rng.integers(0, 20, int(al.sum()))]
    return {"kind": c["kind"], "eng": L.Engine(0), "idx": _Index(_starts(cnt), kb, 6, 1, 0), "seq": seq,
            "off": _starts(al), "len": al.astype(np.int32), "opt": L.SeedOpt(c["max_occ"], 0, 0, None), "n": c["n"],
            "a_off": np.zeros(c["n"] + 1, np.int64),
            "anchors": torch.zeros(8000 * c["n"] + 200_000, dtype=torch.int64, device="cuda")}


def _prepare_chain(c, rng):
    genome, bbit = 100_000_000, 8
    al = _lengths(rng, c["n"], c["al"])
    parts = []
    for rate, some in ((0.15, 1.0), (0.05, 0.5)):  # the gene and, half the time, a weaker paralog
        _, _, gene, pos, glen, _ = _genes(rng, al, frameshifts=0)
        start = (rng.random(len(al)) * (genome - glen)).astype(np.int64)
        g, p = gene[::3], pos[::3]
        res = np.arange(len(g)) - _starts(al)[g]
        hit = (rng.random(len(g)) < rate) & (rng.random(len(al)) < some)[g]
        parts.append((g[hit], (start[g] + p)[hit] >> bbit, res[hit]))
    k = rng.poisson(40.0, len(al))
    g = np.repeat(np.arange(len(al)), k)
    parts.append((g, rng.integers(0, genome, len(g)) >> bbit, (rng.random(len(g)) * al[g]).astype(np.int64)))
    g, b, r = (np.concatenate(x) for x in zip(*parts))
    a = (b.astype(np.uint64) << np.uint64(32)) | r.astype(np.uint64)
    order = np.lexsort((a, g))
    g, a = g[order], a[order]
    new = np.ones(len(g), bool)
    new[1:] = (g[1:] != g[:-1]) | (a[1:] != a[:-1])
    g, a = g[new], np.ascontiguousarray(a[new])
    n = np.bincount(g, minlength=len(al)).astype(np.int32)
    cap = max(200 * c["n"] + 20000, len(a))
    return {"kind": c["kind"], "eng": L.Engine(0), "opt": chain_opt_struct(chain_opt("main")), "n": n,
            "off": _starts(n), "a": a, "u": np.zeros(cap, np.uint64), "a_out": np.zeros(cap, np.uint64),
            "n_u": np.zeros(len(n), np.int32)}


PF_MODEL = os.path.join(os.path.dirname(os.path.abspath(P.__file__)), "data", "prefilter.npz")


def _prepare_pf_select(c, rng):
    al = _lengths(rng, c["proteins"], c["al"])
    prot, nt, wl = _windows(rng, al, 1000, 50000)
    n, per = len(al), 8
    pid = np.repeat(np.arange(n), per)
    own = np.tile(np.arange(per) < 3, n)  # own window on both strands, a part of it, windows of other proteins
    win = np.where(own, pid, rng.integers(0, n, n * per))
    minus = np.where(own, np.tile(np.arange(per) == 1, n), rng.random(n * per) < 0.5)
    part = np.tile(np.arange(per) == 2, n)
    nl = np.where(part, np.maximum((wl[win] * rng.uniform(0.3, 0.7, n * per)).astype(np.int64), 3), wl[win])
    jobs = _jobs(JOB, nl, al[pid], _starts(wl)[win] + np.where(minus, len(nt), 0), _starts(al)[pid])
    model, meta = P.load_model(PF_MODEL, 0)
    m = n * per
    return {"kind": c["kind"], "eng": L.Engine(0), "opt": _options("generic"), "model": model, "jobs": jobs,
            "nt": _dev(np.concatenate([nt, _revcomp(nt, wl)])), "aa": _dev(prot), "tau": float(meta["tau"]),
            "margin": int(meta["margin"]), "tau_fb": float(meta["tau_fb"]), "keep": np.zeros(m, np.uint8),
            "fb": np.zeros(m, np.uint8), "out": np.zeros(m, JOB), "prob": np.zeros(m, np.float32)}


def _train_inputs(c, rng):
    rows = c["rows"]
    w = rng.normal(0, 1, P.FDIM)
    f = np.abs(rng.normal(0, 0.12, (rows, P.FDIM))) * (rng.random((rows, P.FDIM)) < 0.6)
    z = f @ w
    y = (z > np.quantile(z, 0.875)).astype(np.float32)  # one candidate in eight passes
    s = np.sort(rng.random((rows, 2)), axis=1) * y[:, None]
    t = np.stack([y, s[:, 0], s[:, 1], y], axis=1).astype(np.float32)
    perm = rng.permutation(rows)[: rows // c["batch"] * c["batch"]].astype(np.int32)
    par = []
    for out, inn, a in ((256, P.FDIM, 1.0), (256, 256, 1.0), (256, 256, 1.0), (16, 256, 0.25)):
        par += [(rng.uniform(-1, 1, out * inn) * a * math.sqrt(6.0 / inn)), np.zeros(out)]
    return torch.from_numpy(f.astype(np.float32)).to(torch.bfloat16), t, perm, np.concatenate(par).astype(np.float32)


TRAIN = {"lr": 1e-3, "pos_w": 4.0, "box_w": 2.0}


def _prepare_pf_train(c, rng):
    f, t, perm, par = _train_inputs(c, rng)
    return {"kind": c["kind"], "model": P.PrefilterModel(0, 256, 1), "feats": f.cuda(), "tgt": _dev(t),
            "perm": _dev(perm), "params": par, "batch": c["batch"], "steps": c["steps"]}


# ------------------------------------------------------------------------------ run

def run(s):
    return globals()["_run_" + s["kind"]](s)


def _run_splice_locus(s):
    ok, score, ntl, aal, cig = L.gpu_global(s["nt"], s["aa"], s["opt"])
    _check(ok, "ns_gpu_global")
    s["cigar"][:len(cig)] = cig
    return {"score": score, "nt_len": ntl, "aa_len": aal, "n_cigar": len(cig), "cigar": s["cigar"]}


def _run_splice_host(s):
    e, ss = s["eng"], s["ss"]
    _check(e.lib.pl_splice_batch_host(e.h, s["opt"].ptr, P.job_ptr(s["jobs"]), len(s["jobs"]), s["nt"].data_ptr(),
                                      s["nt"].numel(), s["aa"].data_ptr(), s["aa"].numel(),
                                      None if ss is None else ss.data_ptr(), 0 if ss is None else ss.numel(),
                                      C.cast(s["res"].data_ptr(), C.POINTER(L.SpliceResult)), s["cig"].data_ptr(),
                                      s["cig"].numel()), "pl_splice_batch_host")
    return {"results": s["res"], "cigar": s["cig"]}


def _run_splice_strands(s):
    e, total = s["eng"], C.c_int64()
    _check(e.lib.pl_splice_batch_device(e.h, s["opt"].ptr, P.job_ptr(s["jobs"]), len(s["jobs"]), s["nt"].data_ptr(),
                                        s["aa"].data_ptr(), None, s["res"].data_ptr(), s["cig"].data_ptr(), s["cap"],
                                        C.byref(total), _stream()), "pl_splice_batch_device")
    return {"results": s["res"], "cigar": s["cig"]}


def _run_ext(s):
    e = s["eng"]
    _check(e.lib.pl_ext_batch_device(e.h, s["opt"].ptr, C.cast(s["jobs"].ctypes.data, C.POINTER(L.ExtJob)),
                                     len(s["jobs"]), s["nt"].data_ptr(), s["aa"].data_ptr(),
                                     None if s["ss"] is None else s["ss"].data_ptr(), None, s["res"].data_ptr(),
                                     _stream()), "pl_ext_batch_device")
    return s["res"]


def _run_gapless(s):
    e = s["eng"]
    _check(e.lib.pl_gapless_score_device(e.h, s["packed"].data_ptr(), s["bases"], s["queries"].data_ptr(), s["nq"],
                                         s["cand"].data_ptr(), s["n"], s["anc"].data_ptr(), s["na"], 256, 6, 40,
                                         s["mat"].ctypes.data, 22, s["codon"].ctypes.data, s["score"].data_ptr(),
                                         _stream()), "pl_gapless_score_device")
    return s["score"]


def _run_hmm(s):
    e = s["eng"]
    _check(e.lib.pl_hmm_score_many_device(e.h, s["handles"], len(s["profs"]), s["n"], s["nt"].data_ptr(),
                                          s["off"].ctypes.data, s["len"].ctypes.data, s["score"].data_ptr(),
                                          _stream()), "pl_hmm_score_many_device")
    return s["score"]


def _run_recheck(s):
    e = s["eng"]
    _check(e.lib.pl_rc_score_host(e.h, s["handles"], len(s["profs"]), len(s["pid"]), s["pid"].ctypes.data,
                                  s["dsq"].ctypes.data, s["dsq"].size, s["off"].ctypes.data, s["len"].ctypes.data,
                                  s["null2"], s["bits"].ctypes.data, s["bias"].ctypes.data), "pl_rc_score_host")
    return {"bits": s["bits"], "bias": s["bias"]}


class _Words:
    """n 64-bit words of device memory that the engine owns, for torch.as_tensor (which
    holds this object, and with it the engine)."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i8", "data": (ptr, False), "version": 3}


def _run_seed(s):
    e, ptr = s["eng"], C.c_void_p()
    tot = e.lib.pl_seed_anchors_opt_device(e.h, s["idx"].h, s["n"], s["seq"].ctypes.data, s["seq"].size,
                                           s["off"].ctypes.data, s["len"].ctypes.data, C.byref(s["opt"]),
                                           s["a_off"].ctypes.data, C.byref(ptr))
    _check(tot >= 0, "pl_seed_anchors_opt_device")
    if tot:  # the engine's next call reuses its memory: a program that keeps the anchors copies them
        s["anchors"][:tot] = torch.as_tensor(_Words(e, ptr.value, tot), device="cuda")
    return {"offsets": s["a_off"], "anchors": s["anchors"]}


def _run_chain(s):
    e = s["eng"]
    _check(e.lib.pl_chain_host(e.h, C.byref(s["opt"]), len(s["n"]), s["off"].ctypes.data, s["n"].ctypes.data,
                               s["a"].ctypes.data, len(s["a"]), s["u"].ctypes.data, s["n_u"].ctypes.data,
                               s["a_out"].ctypes.data), "pl_chain_host")
    return {"n_u": s["n_u"], "u": s["u"], "anchors": s["a_out"]}


def _run_pf_select(s):
    e, j = s["eng"], s["jobs"]
    _check(e.lib.pl_pf_select_device(s["model"].h, e.h, s["opt"].ptr, j.ctypes.data, len(j), s["nt"].data_ptr(),
                                     s["aa"].data_ptr(), s["tau"], s["margin"], s["tau_fb"], s["keep"].ctypes.data,
                                     s["fb"].ctypes.data, s["out"].ctypes.data, s["prob"].ctypes.data, _stream()),
           "pl_pf_select_device")
    return {"keep": s["keep"], "fallback": s["fb"], "jobs": s["out"].view(np.uint8), "prob": s["prob"]}


def _run_pf_train(s):
    m = s["model"]
    m.set_params(s["params"])
    loss = m.train(s["feats"], s["tgt"], s["perm"], s["batch"], s["steps"], TRAIN["lr"], TRAIN["pos_w"], TRAIN["box_w"])
    return {"loss": loss, "params": m.params()}


# ------------------------------------------------------------------------------ work

OPS_SPLICE, OPS_EXT, OPS_HMM, OPS_GAPLESS, OPS_RECHECK = 65, 31, 17, 12, 60


def work(case):
    c, k = case, case["kind"]
    mean_al = lambda med, sig=0.6: med * math.exp(sig * sig / 2)
    if k == "splice_locus":
        return {"bytes": c["window"] + c["al"] + 200, "flops": OPS_SPLICE * c["window"] * c["al"]}
    if k == "splice_host":
        al, w = min(mean_al(c["al"]), c["al_max"]), (c["win_min"] + c["win_max"]) / 2
        return {"bytes": int(c["n"] * (w * (2 if c["tracks"] else 1) + al + 100)), "flops": int(OPS_SPLICE * c["n"] * w * al)}
    if k == "splice_strands":
        al, w = mean_al(c["al"]), (1000 + c["win_max"]) / 2
        return {"bytes": int(c["pairs"] * (2 * w + al + 300)), "flops": int(OPS_SPLICE * 2 * c["pairs"] * w * al)}
    if k == "ext":
        al = (min(64, c["win_max"] // 2) + c["win_max"]) / 2
        w = 3 * al + 400
        return {"bytes": int(c["n"] * (w * (2 if c["tracks"] else 1) + al + 64)), "flops": int(OPS_EXT * c["n"] * w * al * 0.7)}
    if k == "gapless":
        return {"bytes": int(c["n"] * (44 + c["anchors"] * (16 + 3 * 256 // 2))), "flops": OPS_GAPLESS * c["n"] * c["anchors"] * 256}
    if k == "hmm":
        m = (50 + c["m_max"]) / 2
        codons = 2 * c["slice"] * c["region"] / _hmm_step(c["region"])
        return {"bytes": int(6 * c["slice"] + c["profiles"] * m * 54), "flops": int(OPS_HMM * c["profiles"] * codons * m)}
    if k == "recheck":
        cells = c["n"] * (30 + c["len_max"]) / 2 * (50 + c["m_max"]) / 2
        return {"bytes": int(c["n"] * (c["len_max"] / 2 + 32) + c["profiles"] * 400 * 116),
                "flops": int(OPS_RECHECK * cells * (3 if c["null2"] else 1))}
    if k == "seed":
        res = c["n"] * mean_al(c["al"], 0.7)
        per = 6.0  # anchors a residue: every other k-mer kept, 12 blocks a bucket
        return {"bytes": int(res * (1 + 8 + per * 12)), "flops": int(res * 40)}
    if k == "chain":
        a = c["n"] * 110.0
        return {"bytes": int(a * 8 * 2), "flops": int(a * 13 * 47)}
    if k == "pf_select":
        n = 8 * c["proteins"]
        return {"bytes": int(c["proteins"] * 52000 + n * 60), "flops": int(n * 2 * (576 * 256 + 2 * 256 * 256 + 256 * 16))}
    flops = 3 * c["steps"] * c["batch"] * 2 * (576 * 256 + 2 * 256 * 256 + 256 * 16)
    return {"bytes": c["steps"] * (c["batch"] * (576 * 2 + 16) + 284000 * 4 * 6), "flops": flops}


# ------------------------------------------------------------------------------ exact values

def exact(case, seed):
    """64-bit values of the two paths with computed numbers: the recheck's bits and bias, and
    training's losses and parameters.  All other outputs are integers (the selector's
    probabilities come from features that only the framework computes: no value)."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "recheck":
        return _exact_recheck(case, rng)
    if case["kind"] == "pf_train":
        return _exact_train(case, rng)
    return None


def _exact_recheck(c, rng):
    tabs, pid, lens, off, dsq = _recheck_inputs(c, rng)
    bits, bias = np.zeros(c["n"]), np.zeros(c["n"])
    for k in range(len(tabs)):
        q = np.nonzero(pid == k)[0]
        if len(q):
            bits[q], bias[q] = _forward64(*tabs[k], [dsq[off[x]:off[x] + lens[x]] for x in q], c["null2"])
    return {"bits": bits, "bias": bias}


def _forward64(msc, tsc, peps, null2):
    """Multihit-local Forward (and Backward with null2) of one profile's peptides, in scaled
    64-bit probabilities; the delete chain of a row is one matrix product."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = dict(dtype=torch.float64, device=dev)
    M, n, Lm = len(msc), len(peps), max(len(p) for p in peps)
    t = torch.tensor(np.asarray(tsc, np.float64), **f64)
    e = torch.exp(torch.tensor(np.asarray(msc, np.float64), **f64))
    tp = torch.exp(t)
    MM, IM, DM, BM, MI, II, MD, DD = (tp[:, j] for j in range(8))
    x = torch.full((n, Lm), 20, dtype=torch.long, device=dev)
    for j, p in enumerate(peps):
        x[j, :len(p)] = torch.tensor(p.astype(np.int64), device=dev)
    ln = torch.tensor([len(p) for p in peps], **f64)
    lmask = torch.tensor([len(p) for p in peps], device=dev)
    move, loop = 3.0 / (ln + 3.0), 1.0 - 3.0 / (ln + 3.0)
    # D(k) = sum over k' < k of M(k') MD(k') prod DD(k'+1 .. k-1), columns 0-based
    cs = torch.cumsum(t[:, 7], 0)
    T = torch.exp(cs[None, :] - cs[:, None] + (t[:, 6])[:, None])
    T = torch.triu(torch.cat([torch.zeros(M, 1, **f64), T[:, :-1]], 1), 1)
    Z = torch.zeros(n, 1, **f64)
    Mv, Iv, Dv = (torch.zeros(n, M, **f64) for _ in range(3))
    N, B, J, Cc = torch.ones(n, **f64), move.clone(), torch.zeros(n, **f64), torch.zeros(n, **f64)
    logs, tot = torch.zeros(n, **f64), torch.zeros(n, **f64)
    FM, FI, FS, LS = [Mv], [Iv], [(N, J, Cc)], [logs]
    for i in range(Lm):
        prev = lambda v: torch.cat([Z, v[:, :-1]], 1)
        m2 = (prev(Mv) * MM + prev(Iv) * IM + prev(Dv) * DM + B[:, None] * BM) * e[:, x[:, i]].T
        i2 = Mv * MI + Iv * II
        i2[:, -1] = 0.0
        d2 = m2 @ T
        E = (m2 + d2).sum(1)
        J, Cc, N = J * loop + 0.5 * E, Cc * loop + 0.5 * E, N * loop
        B = (N + J) * move
        sc = (N + J + Cc + E)
        Mv, Iv, Dv = m2 / sc[:, None], i2 / sc[:, None], d2 / sc[:, None]
        N, B, J, Cc = N / sc, B / sc, J / sc, Cc / sc
        logs = logs + torch.log(sc)
        tot = torch.where(lmask == i + 1, torch.log(Cc) + logs + torch.log(move), tot)
        if null2:
            FM.append(Mv), FI.append(Iv), FS.append((N, J, Cc)), LS.append(logs)
    null1 = ln * torch.log(ln / (ln + 1.0)) + torch.log(1.0 / (ln + 1.0))
    b = torch.zeros(n, **f64)
    if null2:
        um, ui = torch.zeros(n, M, **f64), torch.zeros(n, M, **f64)
        uS = torch.zeros(n, **f64)
        cd = torch.cumsum(t[:, 7], 0)
        # D(k) = sum over k' >= k of u(k') prod DD(k .. k'-1): strictly a row-wise product
        TB = torch.triu(torch.exp(torch.cat([Z[0, :1], cd[:-1]])[None, :] - torch.cat([Z[0, :1], cd[:-1]])[:, None]))
        nxt = lambda v: torch.cat([v[:, 1:], Z], 1)
        nx1 = lambda v: torch.cat([v[1:], v[:1]])
        bM, bI = torch.zeros(n, M, **f64), torch.zeros(n, M, **f64)
        bN, bJ, bC, bl = (torch.zeros(n, **f64) for _ in range(4))
        for i in range(Lm, 0, -1):
            last, live = lmask == i, lmask >= i
            col = x[:, min(i, Lm - 1)]
            me = bM * e[:, col].T
            bB = (me * BM).sum(1)
            J2, C2, N2 = bJ * loop + bB * move, bC * loop, bN * loop + bB * move
            J2 = torch.where(last, torch.zeros_like(J2), J2)
            C2, N2 = torch.where(last, move, C2), torch.where(last, torch.zeros_like(N2), N2)
            bE = 0.5 * (J2 + C2)
            mn = nxt(me)
            u = mn * nx1(DM) + bE[:, None]
            u[:, -1] = bE
            u = torch.where(last[:, None], bE[:, None].expand_as(u), u)
            D = u @ TB.T
            m2 = mn * nx1(MM) + bI * MI + bE[:, None] + nxt(D) * MD
            i2 = mn * nx1(IM) + bI * II
            m2 = torch.where(last[:, None], bE[:, None] + nxt(D) * MD, m2)
            i2 = torch.where(last[:, None], torch.zeros_like(i2), i2)
            m2[:, -1], i2[:, -1] = bE, 0.0
            sc = torch.where(live, J2 + C2 + N2, torch.ones_like(J2))
            bl = torch.where(last, torch.zeros_like(bl), bl) + torch.where(live, torch.log(sc), torch.zeros_like(sc))
            bM, bI, bN, bJ, bC = (v / (sc[:, None] if v.dim() == 2 else sc) for v in (m2, i2, N2, J2, C2))
            w = torch.where(live, torch.exp(LS[i] + bl - tot), torch.zeros_like(bl))
            um += FM[i] * bM * w[:, None]
            ui += FI[i] * bI * w[:, None]
            wp = torch.where(live, torch.exp(LS[i - 1] + bl - tot), torch.zeros_like(bl)) * loop
            pN, pJ, pC = FS[i - 1]
            uS += wp * (pN * bN + pJ * bJ + pC * bC)
        v = ((uS + ui[:, :-1].sum(1))[:, None] + um @ e[:, :20]) / ln[:, None]
        lv = torch.log(torch.cat([v, v.mean(1, keepdim=True)], 1))
        live = torch.arange(Lm, device=dev)[None, :] < lmask[:, None]
        n2 = (torch.gather(lv, 1, x) * live).sum(1)
        b = torch.nn.functional.softplus(math.log(1.0 / 256.0) + n2, threshold=700.0)
    return ((tot - null1 - b) / math.log(2.0)).cpu().numpy(), (b / math.log(2.0)).cpu().numpy()


def _exact_train(c, rng):
    f, t, perm, par = _train_inputs(c, rng)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f, t = f.to(torch.float64).to(dev), torch.from_numpy(t).double().to(dev)
    perm = torch.from_numpy(perm.astype(np.int64)).to(dev)
    ps, at = [], 0
    for out, inn in ((256, P.FDIM), (256, 256), (256, 256), (16, 256)):
        for shape in ((out, inn), (out,)):
            k = int(np.prod(shape))
            ps.append(torch.from_numpy(par[at:at + k].astype(np.float64)).reshape(shape).to(dev).requires_grad_(True))
            at += k
    mom, var = [torch.zeros_like(p) for p in ps], [torch.zeros_like(p) for p in ps]
    losses, B = [], c["batch"]
    for s in range(c["steps"]):
        j = s % (len(perm) // B)
        rows = perm[j * B:(j + 1) * B]
        h, y = f[rows], t[rows]
        for k in range(4):
            h = h @ ps[2 * k].T + ps[2 * k + 1]
            h = torch.relu(h) if k < 3 else h
        cw = torch.where(y[:, 0] > 0.5, TRAIN["pos_w"], 1.0)
        bce = torch.nn.functional.binary_cross_entropy_with_logits(h[:, 0], y[:, 0], reduction="none")
        d = (h[:, 1:3] - y[:, 1:3]).abs()
        box = torch.where(d < 0.05, d * d / 0.1, d - 0.025).sum(1)
        loss = (cw * bce + TRAIN["box_w"] * y[:, 3] * box).mean()
        g = torch.autograd.grad(loss, ps)
        losses.append(float(loss.detach()))
        with torch.no_grad():
            for k, p in enumerate(ps):
                mom[k] = 0.9 * mom[k] + 0.1 * g[k]
                var[k] = 0.999 * var[k] + 0.001 * g[k] * g[k]
                step = (mom[k] / (1 - 0.9 ** (s + 1))) / (torch.sqrt(var[k] / (1 - 0.999 ** (s + 1))) + 1e-8)
                p -= TRAIN["lr"] * (step + (1e-5 * p if p.dim() == 2 else 0.0))
    return {"loss": np.array(losses), "params": torch.cat([p.detach().reshape(-1) for p in ps]).cpu().numpy()}
