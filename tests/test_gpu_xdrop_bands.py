"""x-drop passes on lane groups at the places where their layout can go wrong, against the oracle: lengths around the
16-row blocks and the lanes' head start, every band layout (exact, with spare cells, and the warp form above 325) with
its neighbours, the last column within and beyond the band, runs of N, gap models without an opening cost, scores past
the packed word's range, passes longer than their traceback slot (retried with a whole-pass slot), empty sequences."""
import numpy as np
import pytest

from dcns_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def similar(rng, n1, n2, identity=0.9, indel=0.03, n_run=0):
    a = W.random_seq(rng, max(n1, n2, 1))
    b = bytearray(W.mutate(rng, bytes(a), identity, indel)) + W.random_seq(rng, n2)
    a, b = W.prepare(bytes(a[:n1]).decode()), W.prepare(bytes(b[:n2]).decode())
    for x in (a, b):
        for _ in range(n_run):
            at = int(rng.integers(0, max(1, len(x) - 4)))
            x[at:at + int(rng.integers(1, 4))] = 2
    return a, b


def check(eng, oracle, tasks, **kw):
    """kw as the engine takes it; the oracle's names for the first gap piece differ."""
    okw = {{"open1": "open", "ext1": "ext"}.get(k, k): v for k, v in kw.items()}
    for cig in (False, True):
        out, cigars = eng.SemiGlobal_xextend(tasks, cigar=cig, **kw)
        for k, (a, b) in enumerate(tasks):
            exp = oracle.xextend(a, b, cigar=cig, **okw)
            assert tuple(int(v) for v in out[k, :3]) == (exp["score"], exp["end1"], exp["end2"]), (k, len(a), len(b))
            if cig:
                assert cigars[k] == exp["cigar"], (k, len(a), len(b))
                assert tuple(int(v) for v in out[k, 3:5]) == (exp["iii"], exp["jjj"]), k


@pytest.mark.parametrize("w", [1, 2, 5, 9, 10, 11, 20, 21, 40, 41, 42, 80, 81, 160, 164, 165, 320, 325, 326, 400])
def test_band_layouts(lib, oracle, w):
    rng = np.random.default_rng(w)
    tasks = [similar(rng, int(n1), int(n2), 0.85 + 0.14 * rng.random(), 0.06 * rng.random(), k % 3)
             for k, (n1, n2) in enumerate([(300, 300), (300, 120), (90, 700), (700, 60), (w, w), (w + 1, 2 * w + 3),
                                           (2 * w, w + 2), (33, 33)])]
    check(lib, oracle, tasks, w=w, xdrop=30)


@pytest.mark.parametrize("n", [1, 2, 6, 7, 8, 9, 10, 11, 15, 16, 17, 31, 32, 33, 47, 48, 49])
def test_block_edges(lib, oracle, n):
    rng = np.random.default_rng(100 + n)
    check(lib, oracle, [similar(rng, n1, n2, 0.97, 0.01) for n1 in (n, 64) for n2 in (n, n + 1, 64)])


@pytest.mark.parametrize("kw", [dict(xdrop=0), dict(xdrop=200), dict(open1=0, ext1=0), dict(open1=0, ext1=-1),
                                dict(open1=-2, ext1=-5), dict(match=5, mismatch=-4, open1=-10, ext1=-1, xdrop=60),
                                dict(mismatch=1)])
def test_scorings(lib, oracle, kw):
    rng = np.random.default_rng(7)
    check(lib, oracle, [similar(rng, 400, 380, 0.8 + 0.02 * k, 0.03, k % 2) for k in range(8)], **kw)


def test_scores_past_the_packed_word(lib, oracle):
    rng = np.random.default_rng(8)
    tasks = [similar(rng, 8500, 8450, 0.995, 0.001), similar(rng, 300, 9000, 0.9, 0.02)]
    check(lib, oracle, tasks, match=127, mismatch=-127, open1=-120, ext1=-60, xdrop=2000)


def test_mismatches_past_the_packed_word(lib, oracle):
    """A mismatch that scores more than a match: the mismatches, not the matches, reach 2^20."""
    rng = np.random.default_rng(12)
    check(lib, oracle, [similar(rng, 12000, 11990, 0.3, 0.0), similar(rng, 200, 180, 0.3, 0.0)],
          match=1, mismatch=127, open1=-10, ext1=-5)


def test_long_passes_and_empty_ones(lib, oracle):
    """Passes of 5,000 rows outgrow slots of 2,048; empty and one-base sequences among them."""
    rng = np.random.default_rng(9)
    e = np.zeros(0, np.int8)
    tasks = [similar(rng, 5000, 5100, 0.97, 0.005) for _ in range(3)]
    tasks += [(e, e), (tasks[0][0], e), (e, tasks[0][1]), (tasks[0][0][:1], tasks[0][0][:1])]
    tasks += [similar(rng, 200, 200) for _ in range(40)]
    check(lib, oracle, tasks)


def test_seeds_of_one_alignment_share_its_reverse_pass(lib, oracle):
    """Pairs whose alignments hold many seeds (one reverse pass serves all that extend to the same end) next to pairs
    with a seed each: the fragments are the oracle's."""
    rng = np.random.default_rng(10)
    pairs = [similar(rng, 1500, 1500, 0.93, 0.004) for _ in range(3)]
    for _ in range(6):
        a, b = W.planted_pair(rng, 900, 800, 5, 40, 160, 0.85, 0.98, 0.02, 0.0)
        pairs.append((W.prepare(a), W.prepare(b)))
    for two_gap in (False, True):
        got = lib.align_pairs(pairs, 2 if two_gap else 1)
        for k, (a, b) in enumerate(pairs):
            exp, _ = oracle.find(a, b, two_gap=two_gap)
            assert [f.key() for f in got[k]] == [f.key() for f in exp], (k, two_gap)


def test_lists_by_length_and_in_order_agree(lib, oracle):
    """A call past 16 passes per multiprocessor hands its passes out longest first, the same tasks in smaller calls go
    in order: the same results.  Lengths from 0 to the longest, which stands alone in its class."""
    rng = np.random.default_rng(13)
    n = 16 * 152 + 70
    tasks = [similar(rng, int(rng.integers(0, 130)), int(rng.integers(0, 130)), 0.9, 0.02) for _ in range(n)]
    tasks[5] = similar(rng, 640, 640, 0.97, 0.01)
    for cig in (False, True):
        out, cigars = lib.SemiGlobal_xextend(tasks, cigar=cig, w=3)
        for k in range(0, n, 1000):
            part, pc = lib.SemiGlobal_xextend(tasks[k:k + 1000], cigar=cig, w=3)
            assert np.array_equal(out[k:k + 1000], part)
            if cig:
                assert all(np.array_equal(a, b) for a, b in zip(cigars[k:k + 1000], pc))
    check(lib, oracle, tasks[:120], w=3)
