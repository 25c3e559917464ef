"""Two-piece DPs at the edges of the flow kernel's units and of the retrace's tiles, against the oracle: sequence
lengths around multiples of 128 (stripes, checkpoint columns) and of 16 and 32 (half chunks, chunks), bands whose edges
cross tiles, gaps of the second piece that run over many tiles in either direction, runs of N, DPs that leave SMs idle
(eight tiles at a time) and more DPs than SMs (four), and the weighted drivers with categories that change at every
base."""
import numpy as np
import pytest

from dcns_gb300 import workloads as W

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 126, 127, 128, 129, 130, 255, 256, 257, 384, 385]


def similar(rng, n1, n2, n_run=0):
    a, b = W.planted_pair(rng, max(n1, 1), max(n2, 1), max(1, min(n1, n2) // 100), 20, 90, 0.8, 0.97, 0.02, 0.0)
    a, b = W.prepare(a)[:n1], W.prepare(b)[:n2]
    for x in (a, b):
        for _ in range(n_run):
            at = int(rng.integers(0, max(1, len(x) - 10)))
            x[at:at + int(rng.integers(1, 10))] = 2
    return a, b


def check(eng, oracle, tasks, **kw):
    for cig in (False, True):
        out, cigars = eng.SemiGlobal(tasks, cigar=cig, **kw)
        for k, (a, b) in enumerate(tasks):
            exp = oracle.semiglobal(a, b, cigar=cig, **kw)
            assert tuple(int(v) for v in out[k, :3]) == (exp["score"], exp["end1"], exp["end2"]), (k, len(a), len(b))
            assert cigars[k] == exp["cigar"], (k, len(a), len(b), cig)


@pytest.mark.parametrize("kw", [dict(), dict(ext2=-1, open2=-30), dict(bandwidth=16), dict(bandwidth=128, zdrop=500),
                                dict(bandwidth=129, zdrop=500), dict(bandwidth=300, zdrop=20)])
@pytest.mark.parametrize("many", [False, True])
def test_edges(lib, oracle, kw, many):
    rng = np.random.default_rng(11)
    tasks = [similar(rng, int(n1), int(n2), k % 3) for k, (n1, n2) in
             enumerate((a, b) for a in EDGES for b in EDGES if many or (a + b) % 5 == 0)]
    assert many == (len(tasks) > 152)
    check(lib, oracle, tasks, **kw)


@pytest.mark.parametrize("gap", [127, 128, 129, 700, 1500])
def test_long_gaps(lib, oracle, gap):
    """Both halves of a match around one gap of the second piece, in seq1 and in seq2, at several tile offsets."""
    rng = np.random.default_rng(12)
    tasks = []
    for off in (0, 5, 64, 127):
        core = W.prepare(bytes(W.random_seq(rng, 420 + off)).decode())
        ins = W.prepare(bytes(W.random_seq(rng, gap)).decode())
        long = np.concatenate([core[:200 + off], ins, core[200 + off:]])
        tasks += [(core, long), (long, core)]
    check(lib, oracle, tasks)
    check(lib, oracle, tasks, ext2=-1, open2=-20, zdrop=5000)


def test_weighted_edges(lib, oracle):
    rng = np.random.default_rng(13)
    cats = [(2, -3, -4, -2, -45, 0, 100), (3, -4, -6, -2, -60, -1, 50), (1, -2, -3, -1, -30, 0, 200)]
    sizes = [(127, 300), (128, 129), (129, 128), (300, 127), (256, 257), (500, 384), (641, 600)] * 6
    cases = []
    for n1, n2 in sizes:
        a, b = W.planted_pair(rng, n1, n2, 3, 40, 100, 0.9, 0.98, 0.01, 0.0)
        a, b = W.prepare(a), W.prepare(b)
        a[rng.integers(0, n1, 2)] = 2
        cases.append((a, b, rng.integers(0, 3, n1).astype(np.int16)))
    found = 0
    for pieces in (1, 2):
        for bandwidth in (20000, 40):
            got = lib.align_weighted([(a, b) for a, b, _ in cases], [w for _, _, w in cases], cats, pieces,
                                     bandwidth=bandwidth)
            for k, (a, b, w) in enumerate(cases):
                exp = oracle.find_weighted(a, b, w, cats, pieces, bandwidth=bandwidth)
                assert [f.key() for f in got[k]] == [f.key() for f in exp], (k, pieces, bandwidth)
                found += len(exp)
    assert found > 100


def related(rng, n1, n2, shift):
    """A pair that aligns from its first base on; after 150 bases one of the two holds `shift` bases more, so that the
    path runs that far off the diagonal."""
    a = W.random_seq(rng, max(n1, n2) + abs(shift) + 1)
    b = bytes(a[:150]) + W.mutate(rng, bytes(a[150:]), 0.93, 0.004)
    ins = bytes(W.random_seq(rng, abs(shift)))
    a, b = (bytes(a), b[:150] + ins + b[150:]) if shift > 0 else (bytes(a[:150]) + ins + bytes(a[150:]), b)
    return W.prepare(a[:n1].decode()), W.prepare(b[:n2].decode())


@pytest.mark.parametrize("w", [20, 65, 79, 80, 96, 127, 143, 144, 160, 200, 333, 700])
def test_sliding_bands(lib, oracle, w):
    """Bands that slide over several stripes, with the path in their middle and along either edge: chunks that hold the
    left end, the right end or both, stripes with the stale column, sequences that end inside the band."""
    rng = np.random.default_rng(w)
    tasks = [related(rng, n1, n2, s) for n1, n2 in ((900, 900), (1100, 700), (641, 1000), (1025, 1024), (897, 640 + w))
             for s in (0, w - 3, 3 - w)]
    for kw in (dict(), dict(ext2=-1, open2=-30)):
        check(lib, oracle, tasks, bandwidth=w, zdrop=4000, **kw)


@pytest.mark.parametrize("w", [65, 160, 333])
def test_weighted_sliding_bands(lib, oracle, w):
    rng = np.random.default_rng(w)
    cats = [(2, -3, -4, -2, -45, 0, 4000), (3, -4, -6, -2, -60, -1, 4000), (1, -2, -3, -1, -30, 0, 4000)]
    found = 0
    for pieces in (1, 2):
        cases = [related(rng, n1, n2, s) for n1, n2 in ((900, 900), (1100, 700), (641, 1000)) for s in (0, w - 3, 3 - w)]
        cat = [rng.integers(0, 3, len(a)).astype(np.int16) for a, _ in cases]
        got = lib.align_weighted(cases, cat, cats, pieces, bandwidth=w)
        for k, ((a, b), c) in enumerate(zip(cases, cat)):
            exp = oracle.find_weighted(a, b, c, cats, pieces, bandwidth=w)
            assert [f.key() for f in got[k]] == [f.key() for f in exp], (k, pieces)
            found += len(exp)
    assert found >= 12
