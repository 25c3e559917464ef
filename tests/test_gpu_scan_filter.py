"""The seed-scan filter leaves out only windows that stay below min_score: with it (the default) every call gives the
fragments of a context that scans every window against its whole reference (DCNS_SCAN_FILTER=0, the form the other
tests pin to the reference's outputs), and the oracle's.  Sizes lie at the edges of the filter's tiles: strips of 16
columns, systems of 32 strips of which 3 are repeated (464 new columns; two to a warp), blocks of 16 rows, row chunks;
empty and tiny sequences; runs of N on both sides; scorings inside and outside the filter's rule; references marked
nearly everywhere, where the tile list overflows and the whole scan runs after all."""
import numpy as np
import pytest

from dcns_gb300 import workloads as W
from test_gpu_knobs import engine_with, flat

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engines(lib):
    return engine_with({"DCNS_SCAN_FILTER": "1"}), engine_with({"DCNS_SCAN_FILTER": "0"})


def planted(rng, n1, n2, n_run=0):
    a, b = W.planted_pair(rng, n1, n2, max(1, min(n1, n2) // 150), 30, 200, 0.8, 0.97, 0.02, 0.0)
    a, b = W.prepare(a), W.prepare(b)
    for x in (a, b):
        for _ in range(n_run):
            at = int(rng.integers(0, max(1, len(x) - 20)))
            x[at:at + int(rng.integers(1, 20))] = 2
    return a, b


def same(engines, oracle, pairs, two_gap=False, **kw):
    mode = 2 if two_gap else 1
    on, off = (e.align_pairs(pairs, mode, **kw) for e in engines)
    assert flat(on) == flat(off)
    for k, (a, b) in enumerate(pairs):
        if oracle is not None and len(b) >= 8:
            exp, _ = oracle.find(a, b, two_gap=two_gap, **kw)
            assert [f.key() for f in on[k]] == [f.key() for f in exp], k
    return sum(len(x) for x in on)


@pytest.mark.parametrize("n2", [1, 37, 38, 39, 46, 511, 512, 513, 928, 975, 976, 977, 1439, 1440, 1441])
def test_column_edges(engines, oracle, n2):
    rng = np.random.default_rng(100 + n2)
    found = same(engines, oracle, [planted(rng, int(n1), n2, 2) for n1 in (700, 641, 15, 16, 1)])
    assert found > 0 or n2 < 100


@pytest.mark.parametrize("n1", [1, 19, 20, 38, 59, 60, 61, 119, 120, 121, 159, 160, 161, 319, 320, 321, 495, 512, 1000])
def test_row_edges(engines, oracle, n1):
    """Row chunks of few pairs are as short as the warm-up; one pair alone, and among others."""
    rng = np.random.default_rng(200 + n1)
    pairs = [planted(rng, n1, int(n2), 1) for n2 in (600, 333)]
    same(engines, oracle, pairs[:1])
    same(engines, oracle, pairs + [planted(rng, 2000, 900), (np.zeros(0, np.int8), pairs[0][1])])


def test_matches_at_every_place_of_a_tile(engines, oracle):
    """A 20-base match (the least that reaches min_score 40) at each offset from a strip's and a block's start, the
    sequence's first and last bases among them."""
    rng = np.random.default_rng(3)
    pairs = []
    for k in range(36):
        a, b = W.random_pair(rng, 520, 560, 2)
        a, b = (a * 0).astype(np.int8), (b * 0 + 3).astype(np.int8)  # A against G: nothing matches
        m = rng.choice(np.array([1, 4], np.int8), 20)
        p, q = [(0, 0), (500, 540), (496 + k % 4, k), (k, 496 + k), (240 + k, 230 + 2 * k)][k % 5]
        a[p:p + 20] = m
        b[q:q + 20] = m
        pairs.append((a, b))
    same(engines, oracle, pairs, pvalue=1.1)


@pytest.mark.parametrize("kw", [dict(min_score=30), dict(min_score=48, step=5), dict(window=24, min_score=40),
                                dict(match=5, mismatch=-6, open1=-12, ext1=-3, min_score=100, xdrop=50),
                                dict(open1=-6, ext1=-1, min_score=40), dict(open1=-2, ext1=-4, min_score=44),
                                dict(min_score=20), dict(mismatch=-1), dict(step=40)])
def test_scorings(engines, oracle, kw):
    rng = np.random.default_rng(5)
    same(engines, oracle, [planted(rng, 900, 1100, 1), planted(rng, 300, 500, 3)], pvalue=1e300, **kw)


def test_two_gap(engines, oracle):
    rng = np.random.default_rng(6)
    same(engines, oracle, [planted(rng, 1200, 990, 1) for _ in range(4)], two_gap=True)


def test_marked_nearly_everywhere(engines):
    """17-base repeats on both sides: every place is marked (34 + decay >= 32), few windows reach 40; the tile list
    overflows and the whole scan runs."""
    rng = np.random.default_rng(7)
    word = rng.choice(np.array([0, 1, 3, 4], np.int8), 17)

    def repeats(n):
        x = W.random_pair(rng, n, 1)[0] % 4
        x = np.array([0, 1, 3, 4], np.int8)[x]
        for at in range(0, n - 17, 32):
            x[at:at + 17] = word
        return x

    same(engines, None, [(repeats(9000), repeats(9500))])


def test_identical_long_sequences(engines):
    """A score that grows over the whole reference: the row chunks keep it within 16 bits."""
    rng = np.random.default_rng(8)
    a = W.prepare(bytes(W.random_seq(rng, 40000)).decode())
    assert same(engines, None, [(a, a.copy())]) > 0


def test_batch_in_bins(engines):
    rng = np.random.default_rng(9)
    pairs = [planted(rng, int(rng.integers(60, 400)), int(rng.integers(60, 400))) for _ in range(4200)]
    assert same(engines, None, pairs) > 1000


def test_plans_by_warps_and_by_threads_agree(lib):
    """A call of more than 256 window pairs per multiprocessor plans its exact tiles a thread to each, the same pairs
    one by one a warp to each: the same fragments.  References from one word of marks to many chunks."""
    rng = np.random.default_rng(31)
    pairs = []
    for k in range(140):
        n1 = int(rng.integers(60, 12000)) if k % 3 else int(rng.integers(490, 540))
        a, b = W.planted_pair(rng, n1, int(rng.integers(4400, 5200)), int(rng.integers(0, 8)), 40, 200, 0.8, 0.97, 0.01, 0.0)
        pairs.append((W.prepare(a), W.prepare(b)))
    assert sum(len(b) // 16 for _, b in pairs) > 256 * 152
    found = 0
    for mode in (1, 2):
        whole = lib.align_pairs(pairs, mode)
        found += sum(len(w) for w in whole)
        for k, p in enumerate(pairs):
            alone = lib.align_pairs([p], mode)[0]
            assert [f.key() for f in whole[k]] == [f.key() for f in alone], (k, mode)
    assert found > 200
