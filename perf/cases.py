"""The calls a user of the aligner makes, as measurable cases: whole alignments (one pair, one reference against many
queries, resident batches, whole 200 kb pairs, served requests), the x-seed paths (seeded, weighted) and the
kernel-level calls (x-drop extension, two-piece semi-global DP, sliding window), each through its public entry point.

Inputs are synthetic sequences of the shapes the benchmark uses (log-normal lengths, conserved segments planted at the
same relative place, indels of 1-5 bp, masked runs deleted before aligning), plus what real sequences also hold: runs
of N (assembly gaps) and short tandem repeats that the masking missed.
"""
import ctypes
import math

import numpy as np
import torch

import dcns_gb300 as D

CODES = np.array([0, 1, 3, 4], np.int8)  # A C G T
CATS = [(2, -3, -4, -2, -45, 0, 100), (3, -4, -6, -2, -60, -1, 50), (1, -2, -3, -1, -30, 0, 200)]


def listed():
    return [
        # the smallest call: one gene's upstream regions, one pair, where launches and waits count
        {"name": "pair_1kb", "kind": "pair", "n1": 1013, "n2": 877, "mode": 1},
        # the single-pair workload: 5 kb regions, both gap models' drivers call it once per gene
        {"name": "pair_5kb", "kind": "pair", "n1": 5000, "n2": 5000, "mode": 1},
        # multCns: one species' region against the regions of many others, from host buffers
        {"name": "one_to_many_64", "kind": "many", "ref": 20011, "queries": 64},
        # the headline batch, resident on the device (cut1Gap)
        {"name": "batch_10000", "kind": "batch", "pairs": 10000, "mode": 1},
        # cut2Gaps over a batch: the x-seeds and the two-piece DPs
        {"name": "batch_2gap_500", "kind": "batch", "pairs": 500, "mode": 2},
        # whole long regions: 200 kb against 200 kb with duplicated blocks
        {"name": "long_200kb", "kind": "long", "pairs": 2, "length": 200000},
        # served requests, a tenth of them 50-100 kb, all in the queue at once
        {"name": "serve_128", "kind": "serve", "requests": 128},
        # seed extension by itself, with CIGARs (the C call on host buffers)
        {"name": "xextend_50000", "kind": "xextend", "tasks": 50000, "cigar": True},
        # the two-piece DP by itself, with CIGARs
        {"name": "semiglobal_400", "kind": "semiglobal", "tasks": 400, "cigar": True},
        # cut2Gaps2 on a whole region with seeds from an earlier alignment, no length cap
        {"name": "seeded_200kb", "kind": "seeded", "length": 200000, "seeds": 16},
        # weighted2Gaps: per-base categories from an annotation
        {"name": "weighted_100", "kind": "weighted", "pairs": 100, "pieces": 2},
        # slidingWindowAlignment: every window of one sequence against seven others
        {"name": "sliding_10kb", "kind": "sliding", "length": 10007, "seqs": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "many", "batch", "batch", "long", "serve", "xextend", "semiglobal", "seeded",
                       "weighted", "sliding"])
    if kind == "pair":
        return {"kind": kind, "n1": _log(rng, 300, 20000), "n2": _log(rng, 300, 20000), "mode": rng.choice([1, 2])}
    if kind == "many":
        return {"kind": kind, "ref": _log(rng, 1000, 20011), "queries": _log(rng, 4, 64)}
    if kind == "batch":
        mode = rng.choice([1, 1, 2])
        return {"kind": kind, "pairs": _log(rng, 50, 10000 if mode == 1 else 500), "mode": mode}
    if kind == "long":
        return {"kind": kind, "pairs": rng.choice([1, 2]), "length": _log(rng, 30000, 200000)}
    if kind == "serve":
        return {"kind": kind, "requests": _log(rng, 8, 128)}
    if kind == "xextend":
        return {"kind": kind, "tasks": _log(rng, 100, 50000), "cigar": rng.random() < 0.7}
    if kind == "semiglobal":
        return {"kind": kind, "tasks": _log(rng, 10, 400), "cigar": rng.random() < 0.7}
    if kind == "seeded":
        return {"kind": kind, "length": _log(rng, 10000, 200000), "seeds": _log(rng, 2, 16)}
    if kind == "weighted":
        return {"kind": kind, "pairs": _log(rng, 4, 100), "pieces": rng.choice([1, 2])}
    return {"kind": kind, "length": _log(rng, 200, 10007), "seqs": rng.randint(2, 8)}


# ---------------------------------------------------------------------------------------------------- sequences
def _offsets(lens):
    return np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)


def _ranges(starts, lens):
    """The concatenation of arange(start, start + len)."""
    lens = np.asarray(lens, np.int64)
    off = _offsets(lens)
    return np.arange(off[-1]) - np.repeat(off[:-1] - np.asarray(starts, np.int64), lens)


def _bases(rng, n, gc=0.5):
    if gc == 0.5:
        return rng.integers(0, 4, n, dtype=np.uint8)
    u = rng.random(n, dtype=np.float32)
    return np.searchsorted(np.array([(1 - gc) / 2, 0.5, (1 + gc) / 2], np.float32), u).astype(np.uint8)


def _mutate(rng, seq, seg, nseg, identity, indel):
    """Substitutions down to identity[seg] per base, then insertions and deletions of 1-5 bases at rate indel[seg]:
    the mutated bases and the length of each segment."""
    n = len(seq)
    out = seq.copy()
    sub = np.nonzero(rng.random(n, dtype=np.float32) > identity[seg])[0]
    out[sub] = (out[sub] + rng.integers(1, 4, len(sub), dtype=np.uint8)) % 4
    ev = np.nonzero(rng.random(n, dtype=np.float32) < indel[seg])[0]
    k = rng.integers(1, 6, len(ev))
    gone = rng.random(len(ev)) < 0.5
    end = _offsets(np.bincount(seg, minlength=nseg))[1:]
    diff = np.zeros(n + 1, np.int32)
    np.add.at(diff, ev[gone], 1)
    np.add.at(diff, np.minimum(ev[gone] + k[gone], end[seg[ev[gone]]]), -1)
    rep = (np.cumsum(diff[:n]) == 0).astype(np.int64)
    ins, ki = ev[~gone], k[~gone]
    rep[ins] += ki
    at = np.cumsum(rep) - rep
    out = np.repeat(out, rep)
    put = _ranges(at[ins], np.minimum(ki, rep[ins]))
    out[put] = rng.integers(0, 4, len(put), dtype=np.uint8)
    return out, np.bincount(seg, weights=rep, minlength=nseg).astype(np.int64)


def _plant(rng, a, aoff, b, boff, per_pair, lo, hi, id_lo, id_hi, indel):
    """Copies per_pair[k] mutated segments of pair k's first sequence to the same relative place of its second:
    returns their (pair, start1, start2, length in the first, length in the second)."""
    pair = np.repeat(np.arange(len(per_pair)), per_pair)
    n1, n2 = np.diff(aoff)[pair], np.diff(boff)[pair]
    L = rng.integers(lo, hi + 1, len(pair))
    ok = (L < n1) & (L < n2)
    pair, n1, n2, L = pair[ok], n1[ok], n2[ok], L[ok]
    s1 = (rng.random(len(pair)) * (n1 - L)).astype(np.int64)
    s2 = np.minimum((s1 / n1 * n2).astype(np.int64), n2 - L)
    seg = np.repeat(np.arange(len(pair)), L)
    got, m = _mutate(rng, a[_ranges(aoff[pair] + s1, L)], seg, len(pair),
                     rng.uniform(id_lo, id_hi, len(pair)).astype(np.float32), np.full(len(pair), indel, np.float32))
    src = _offsets(m)[:-1]
    fit = np.minimum(m, n2 - s2)
    b[_ranges(boff[pair] + s2, fit)] = got[_ranges(src, fit)]
    return pair, s1, s2, L, fit


def _finish(rng, x, off, mask, gaps, repeats):
    """Codes of the sequences with tandem repeats and runs of N put in and about `mask` of each deleted in runs of
    20-500 bases; their offsets."""
    n = np.diff(off)
    if repeats:
        k = rng.poisson(n * (repeats / 110.0))
        own = np.repeat(np.arange(len(n)), k)
        L = np.minimum(rng.integers(20, 201, len(own)), n[own])
        at = off[own] + (rng.random(len(own)) * (n[own] - L + 1)).astype(np.int64)
        for s, m in zip(at, L):
            x[s:s + m] = np.resize(x[s:s + int(rng.integers(1, 7))], m)
    codes = CODES[x]
    if gaps:
        own = np.nonzero(rng.random(len(n)) < gaps)[0]
        L = np.minimum(rng.integers(50, 101, len(own)), n[own])
        at = off[own] + (rng.random(len(own)) * (n[own] - L + 1)).astype(np.int64)
        codes[_ranges(at, L)] = 2
    if not mask:
        return codes, off
    k = np.ceil(n * (mask / 260.0)).astype(np.int64)
    own = np.repeat(np.arange(len(n)), k)
    L = np.minimum(rng.integers(20, 501, len(own)), n[own] // 3)
    at = off[own] + (rng.random(len(own)) * (n[own] - L)).astype(np.int64)
    diff = np.zeros(len(x) + 1, np.int32)
    np.add.at(diff, at, 1)
    np.add.at(diff, at + L, -1)
    keep = np.cumsum(diff[:-1]) == 0
    left = np.add.reduceat(keep, off[:-1]) if len(x) else n
    return codes[keep], _offsets(left)


def _views(codes, off):
    return [codes[off[k]:off[k + 1]] for k in range(len(off) - 1)]


def _lognormal(rng, n, median, sigma, lo, hi):
    return np.clip(np.round(rng.lognormal(math.log(median), sigma, n)), lo, hi).astype(np.int64)


def _pairs(rng, n1, n2, per_pair, lo=30, hi=300, id_lo=0.70, id_hi=0.95, mask=0.15, gaps=0.02, repeats=0.001, gc=0.5):
    aoff, boff = _offsets(n1), _offsets(n2)
    a, b = _bases(rng, aoff[-1], gc), _bases(rng, boff[-1], gc)
    seg = _plant(rng, a, aoff, b, boff, np.asarray(per_pair), lo, hi, id_lo, id_hi, 0.01)
    ca, ao = _finish(rng, a, aoff, mask, gaps, repeats)
    cb, bo = _finish(rng, b, boff, mask, gaps, repeats)
    return list(zip(_views(ca, ao), _views(cb, bo))), seg


def _flanks(rng, n, lo, hi, id_lo, id_hi, indel, tail):
    """n (seq1, seq2) tasks that start in a 38-base core with 0-7 substitutions, go on through lo..hi bases mutated to
    an identity of id_lo..id_hi, and end in `tail` times as many unrelated bases."""
    L = rng.integers(lo, hi + 1, n)
    seg = np.repeat(np.arange(n), L)
    f = _bases(rng, len(seg))
    g, m = _mutate(rng, f, seg, n, rng.uniform(id_lo, id_hi, n).astype(np.float32),
                   rng.uniform(0.0, indel, n).astype(np.float32))
    core = _bases(rng, n * 38)
    core2 = core.copy()
    hit = rng.random((n, 38)).argsort(1) < rng.integers(0, 8, n)[:, None]
    at = np.nonzero(hit.reshape(-1))[0]
    core2[at] = (core2[at] + rng.integers(1, 4, len(at), dtype=np.uint8)) % 4

    def join(c, x, lens, t):
        end = _bases(rng, int(t.sum()))
        off = _offsets(38 + lens + t)
        y = np.empty(off[-1], np.uint8)
        y[_ranges(off[:-1], np.full(n, 38))] = c
        y[_ranges(off[:-1] + 38, lens)] = x
        y[_ranges(off[:-1] + 38 + lens, t)] = end
        return _views(CODES[y], off)

    t1, t2 = (rng.random((2, n)) * tail * L).astype(np.int64)
    return list(zip(join(core, f, L, t1), join(core2, g, m, t2)))


# ---------------------------------------------------------------------------------------------------- prepare
_ENGINES = {}


def _engine(which="align"):
    """A program keeps one engine for all it aligns, and one more where it serves requests."""
    if which not in _ENGINES:
        e = D.Engine(0)
        if which == "serve":
            e.serve_start()
        _ENGINES[which] = e
    return _ENGINES[which]


class _Resident:
    """A batch that lives on the device until the program drops it."""

    def __init__(self, engine, pairs):
        self.engine, self.handle = engine, engine.upload(pairs)

    def __del__(self):
        self.engine.free_batch(self.handle)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = {"kind": kind, "case": case, "engine": _engine("serve" if kind == "serve" else "align")}
    if kind == "pair":
        s["pairs"], _ = _pairs(rng, [case["n1"]], [case["n2"]],
                               [max(1, min(case["n1"], case["n2"]) // 250)], 30, 200, mask=0.20, gaps=0.0, repeats=0.0)
    elif kind == "many":
        q = _lognormal(rng, case["queries"], case["ref"] / 3.0, 0.8, 500, 20000)
        many, _ = _pairs(rng, [case["ref"]] * len(q), q, np.zeros(len(q), np.int64))
        ref, queries = many[0][0], [b.copy() for _, b in many]
        for b in queries:  # segments of the one reference in each query, at the same relative place
            for _ in range(int(min(40, max(1, len(b) // 400)))):
                L = int(rng.integers(30, 301))
                if L < len(b) and L < len(ref):
                    at = int(rng.integers(0, len(ref) - L))
                    seg = ref[at:at + L].copy()
                    hit = rng.random(L) > rng.uniform(0.70, 0.95)
                    seg[hit] = CODES[rng.integers(0, 4, int(hit.sum()))]
                    to = min(int(at / len(ref) * len(b)), len(b) - L)
                    b[to:to + L] = seg
        s["ref"], s["queries"] = ref, queries
    elif kind == "batch":
        n = case["pairs"]
        n1, n2 = _lognormal(rng, n, 3000, 0.8, 500, 20000), _lognormal(rng, n, 3000, 0.8, 500, 20000)
        pairs, _ = _pairs(rng, n1, n2, np.minimum(rng.poisson(8, n), 30))
        if case["mode"] == 1:
            s["batch"] = _Resident(s["engine"], pairs)
        else:
            s["pairs"] = pairs
    elif kind == "long":
        n, L = case["pairs"], case["length"]
        pairs, _ = _pairs(rng, [L] * n, [L] * n, [L // 400] * n, 20, 400, 0.80, 0.80, mask=0.0, gaps=0.5,
                          repeats=0.0002, gc=0.45)
        s["pairs"] = []
        for a, b in pairs:  # transposon-like blocks of the reference inserted into the query
            for _ in range(5):
                m = min(int(rng.integers(2000, 10001)), L // 4)
                at, to = int(rng.integers(0, L - m)), int(rng.integers(0, len(b)))
                blk = a[at:at + m].copy()
                hit = rng.random(m) > 0.9
                blk[hit] = CODES[rng.integers(0, 4, int(hit.sum()))]
                b = np.concatenate([b[:to], blk, b[to:]])
            s["pairs"].append((a, b))
    elif kind == "serve":
        n = case["requests"]
        n1, n2 = _lognormal(rng, n, 4000, 1.0, 200, 100000), _lognormal(rng, n, 4000, 1.0, 200, 100000)
        big = rng.permutation(n) < max(1, n // 10)
        n1[big], n2[big] = rng.integers(50001, 100001, (2, int(big.sum())))
        s["pairs"], _ = _pairs(rng, n1, n2, np.minimum(rng.poisson(8.0 * np.minimum(n1, n2) / 3000.0), 300))
    elif kind == "xextend":
        n = case["tasks"]
        s["table"], s["keep"] = s["engine"].prepare(_flanks(rng, n, 50, 2000, 0.50, 0.98, 0.03, 0.0))
    elif kind == "semiglobal":
        s["tasks"] = _flanks(rng, case["tasks"], 100, 3000, 0.70, 0.98, 0.02, 1.5)
    elif kind == "seeded":
        L = case["length"]
        pairs, (_, s1, s2, m1, m2) = _pairs(rng, [L], [L + L // 6], [L // 400], 38, 400, 0.80, 0.90, mask=0.0,
                                            gaps=0.0, repeats=0.0, gc=0.45)
        pick = rng.permutation(len(s1))[:case["seeds"]]
        s["pairs"] = pairs
        s["seeds"] = [[(int(s1[k]), int(s1[k] + 37), int(s2[k]), int(s2[k] + 37)) for k in sorted(pick)]]
    elif kind == "weighted":
        n = case["pairs"]
        n1, n2 = _lognormal(rng, n, 2500, 0.5, 500, 6000), _lognormal(rng, n, 2500, 0.5, 500, 6000)
        s["pairs"], _ = _pairs(rng, n1, n2, np.minimum(rng.poisson(10, n), 30), 60, 300, 0.85, 0.97, mask=0.0)
        s["weights"] = []
        for a, _ in s["pairs"]:  # categories in runs, as annotated features lie
            runs = rng.integers(50, 600, len(a) // 50 + 1)
            s["weights"].append(np.repeat(rng.integers(0, len(CATS), len(runs)), runs)[:len(a)].astype(np.int16))
    else:
        L = case["length"]
        lens = [L] + [max(1, L - int(v)) for v in rng.integers(0, L // 2 + 1, case["seqs"] - 1)]
        first = _bases(rng, L)
        seqs = [CODES[first]]
        for n in lens[1:]:
            got, _ = _mutate(rng, first[:n], np.zeros(n, np.int64), 1, rng.uniform(0.6, 0.95, 1).astype(np.float32),
                             np.full(1, 0.01, np.float32))
            seqs.append(CODES[got])
        s["seqs"] = seqs
    return s


# ---------------------------------------------------------------------------------------------------- run
def _most(case):
    """Fragments and CIGAR words that the results of such a case stay well under: results come in tables of that many
    rows, zero past the end, whatever the inputs hold."""
    kind = case["kind"]
    if kind == "pair":
        return 400, 40000
    if kind == "many":
        return 200 * case["queries"], 10000 * case["queries"]
    if kind == "batch":
        return 60 * case["pairs"], (300 if case["mode"] == 1 else 7000) * case["pairs"] + 40000
    if kind == "long":
        return case["pairs"] * (case["length"] // 50 + 100), case["pairs"] * (case["length"] + 2000)
    if kind == "serve":
        return 300 * case["requests"] + 2000, 6000 * case["requests"] + 40000
    if kind == "xextend":
        return 0, 70 * case["tasks"] + 30000
    if kind == "semiglobal":
        return 0, 6000 * case["tasks"]
    if kind == "seeded":
        return case["seeds"], case["seeds"] * case["length"]
    return 60 * case["pairs"] + 100, 39000 * case["pairs"]


def _in(x, n):
    """x in the first rows of a zero table of n rows."""
    t = np.zeros((n,) + x.shape[1:], x.dtype)
    t[:len(x)] = x
    return t


def _arrays(r, most):
    return {"pair_offset": r.pair_offset, "frag": _in(r.frag, most[0]), "cigar": _in(r.cigar.view(np.int32), most[1]),
            "pvalue": _in(r.pvalue, most[0]), "evalue": _in(r.evalue, most[0])}


def _rows(lists, most):
    """The fragments of several lists in one table, their CIGARs and their p- and e-values."""
    fr = [f for one in lists for f in one]
    table = np.array([[f.start1, f.end1, f.start2, f.end2, f.score, len(f.cigar)] for f in fr], np.int64)
    return {"count": np.array([len(one) for one in lists], np.int64), "frag": _in(table.reshape(-1, 6), most[0]),
            "cigar": _in(np.array([c for f in fr for c in f.cigar], np.int64), most[1]),
            "pvalue": _in(np.array([f.pvalue for f in fr], np.float64), most[0]),
            "evalue": _in(np.array([f.evalue for f in fr], np.float64), most[0])}


def run(state):
    s, kind, eng = state, state["kind"], state["engine"]
    if kind == "sliding":
        return eng.slidingWindowAlignment(s["seqs"])
    most = _most(s["case"])
    if kind == "pair":
        a, b = s["pairs"][0]
        return _rows([eng.findSimilarFragmentsForPairedSequence(a, b, two_gap=s["case"]["mode"] == 2)], most)
    if kind == "many":
        return _arrays(eng.align_one_to_many(s["ref"], s["queries"]), most)
    if kind == "batch":
        if s["case"]["mode"] == 1:
            return _arrays(eng.align_resident(s["batch"].handle), most)
        return _arrays(eng.align_pairs(s["pairs"], D.MODE_TWO_GAP), most)
    if kind == "long":
        return _arrays(eng.align_pairs(s["pairs"]), most)
    if kind == "serve":
        tickets = [eng.submit(a, b) for a, b in s["pairs"]]
        return _rows([eng.wait(t) for t in tickets], most)
    if kind == "xextend":
        n = len(s["keep"])
        out, off, cigar = np.zeros((n, 6), np.int32), np.zeros(n + 1, np.int64), np.zeros(most[1], np.uint32)
        p = D.params()
        rc = eng.lib.dcns_xextend_batch(eng.h, s["table"], n, ctypes.byref(p), int(s["case"]["cigar"]),
                                        out.ctypes.data_as(D._I32P), cigar.ctypes.data_as(D._U32P), len(cigar),
                                        off.ctypes.data_as(D._I64P))
        if rc != 0:
            raise D.DcnsError(rc, eng.lib.dcns_last_error(eng.h).decode())
        return {"out": out, "offset": off, "cigar": cigar.view(np.int32)}
    if kind == "semiglobal":
        out, cigars = eng.SemiGlobal(s["tasks"], cigar=s["case"]["cigar"])
        return {"out": out, "cigar": _in(np.array([c for one in cigars for c in one], np.int64), most[1])}
    if kind == "seeded":
        return _arrays(eng.align_seeded(s["pairs"], s["seeds"]), most)
    return _arrays(eng.align_weighted(s["pairs"], s["weights"], CATS, s["case"]["pieces"]), most)


# ---------------------------------------------------------------------------------------------------- work, exact
def work(case):
    """Bytes: the sequences in (one byte a base) and the results out.  Operations: a whole alignment has to compare
    every base of one sequence with every base of the other once (about six integer operations a cell); an x-drop pass
    fills a band of at least 21 cells a row, a two-piece DP every column of the rows it goes through."""
    kind = case["kind"]
    if kind == "pair":
        n1, n2 = case["n1"] * 0.82, case["n2"] * 0.82
        return {"bytes": n1 + n2 + 100 * n2 / 250, "flops": 6.0 * n1 * n2}
    if kind == "many":
        n2 = 0.85 * case["queries"] * case["ref"] / 2.3
        return {"bytes": 0.85 * case["ref"] + 1.1 * n2, "flops": 6.0 * 0.85 * case["ref"] * n2}
    if kind == "batch":
        n = 0.85 * 4000.0
        return {"bytes": case["pairs"] * (2 * n + 600), "flops": 6.0 * case["pairs"] * n * n * (1 if case["mode"] == 1 else 2)}
    if kind == "long":
        n1, n2 = float(case["length"]), case["length"] + 5 * min(6000, case["length"] / 5)
        return {"bytes": case["pairs"] * (n1 + n2 + n1 / 4), "flops": 6.0 * case["pairs"] * n1 * n2}
    if kind == "serve":
        n = case["requests"]
        return {"bytes": 2 * 0.85 * n * (0.9 * 6500 + 0.1 * 75000),
                "flops": 6.0 * 0.72 * n * (0.9 * 6500.0 ** 2 + 0.1 * 75000.0 ** 2)}
    if kind == "xextend":
        return {"bytes": case["tasks"] * (2 * 1063 + 24 + (400 if case["cigar"] else 0)),
                "flops": 6.0 * case["tasks"] * 21 * 400}
    if kind == "semiglobal":
        return {"bytes": case["tasks"] * (2 * 2750 + 16), "flops": 10.0 * case["tasks"] * 1550 * 2750}
    if kind == "seeded":
        n1, n2 = float(case["length"]), case["length"] * 7 / 6
        return {"bytes": n1 + n2, "flops": 10.0 * n1 * min(n2, 20000.0)}
    if kind == "weighted":
        n = 2800.0
        return {"bytes": case["pairs"] * (2 * n + 2 * n + 600), "flops": 6.0 * case["pairs"] * n * n * 2}
    n, k = float(case["length"]), case["seqs"] - 1
    return {"bytes": n + 0.75 * n * k + 12.0 * k * n / 8, "flops": 6.0 * 38 * (n / 8) * 0.75 * n * k}


def exact(case, seed):
    """The sliding window's scores in 64-bit integers and floats.  The alignments' p- and e-values follow from whole
    pipelines of sequential DPs and sets, which plain arrays do not get through in the time there is."""
    if case["kind"] != "sliding":
        return None
    seqs = prepare(case, seed)["seqs"]
    window, step, match, mismatch, opening, ext = 38, 8, 2, -3, -4, -2
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    L0, others = len(seqs[0]), seqs[1:]
    start = torch.arange(0, L0, step, device=dev)
    col = start[:, None] + torch.arange(window, device=dev)
    live = col < L0
    read = torch.as_tensor(seqs[0].astype(np.int64), device=dev)[col.clamp(max=L0 - 1)]
    lens = torch.tensor([len(x) for x in others], device=dev)
    rows = int(lens.max())
    ref = torch.full((len(others), rows), 2, dtype=torch.int64, device=dev)
    for k, x in enumerate(others):
        ref[k, :len(x)] = torch.as_tensor(x.astype(np.int64), device=dev)
    shape = (len(others),) + tuple(read.shape)
    H, E = (torch.zeros(shape, dtype=torch.int64, device=dev) for _ in range(2))
    best = torch.zeros(shape[:2], dtype=torch.int64, device=dev)
    far = torch.full(shape[:2] + (1,), -(1 << 40), dtype=torch.int64, device=dev)
    slope = ext * torch.arange(window, device=dev)
    for i in range(rows):
        c = ref[:, i, None, None]
        sc = torch.where(c == read, match, mismatch) * ((c != 2) & (read != 2))
        pre = torch.maximum((torch.nn.functional.pad(H[..., :-1], (1, 0)) + sc).clamp(min=0), E)
        E = torch.maximum(E + ext, pre + opening)
        gap = torch.cummax(torch.cat([far, (pre + opening - slope - ext)[..., :-1]], -1), -1).values + slope
        H = torch.where(live, torch.maximum(pre, gap), 0)
        best = torch.where((i < lens)[:, None], torch.maximum(best, H.amax(-1)), best)
    most = torch.minimum(torch.clamp(L0 - start, max=window)[None], lens[:, None]) * match
    return (best.double() / most.double()).cpu().numpy(), best.cpu().numpy()
