"""Scorings under which a mismatch scores above a match: a path then gains the mismatch on every column, so its gaps may
run over more rows than the match would pay for.  The scan's tiles and the search for a maximum's column start that many
rows early: scores and first places against the oracle, and whole alignments, whose recursion rounds take the same
scan."""
import numpy as np
import pytest

from dcns_gb300 import workloads as W

pytestmark = pytest.mark.gpu

A, C = 0, 1


def runs(*parts):
    return np.concatenate([np.full(n, c, np.int8) for c, n in parts])


def check(eng, oracle, tasks, **kw):
    out = eng.SmithWaterman(tasks, **kw)
    okw = {{"open1": "open", "ext1": "ext"}.get(k, k): v for k, v in kw.items()}
    for k, (a, b) in enumerate(tasks):
        assert tuple(int(v) for v in out[k]) == tuple(int(v) for v in oracle.sw(a, b, **okw)[:3]), k


@pytest.mark.parametrize("mismatch", [2, 4, 10, 60])
@pytest.mark.parametrize("gap", [1, 3])
def test_long_gaps_inside_a_window(lib, oracle, mismatch, gap):
    """Half a read on either side of a run that costs about what the mismatches gain; references of one run; both also
    behind enough rows to fall into several chunks."""
    read = runs((A, 38))
    tasks = []
    for long in (20, 50, 38 * mismatch // (2 * gap), 38 * mismatch // gap):
        ref = runs((C, 19), (A, long), (C, 19))
        tasks += [(ref, read), (np.concatenate([runs((A, 700)), ref, runs((A, 333))]), read)]
    tasks += [(runs((A, n)), read) for n in (150, 400, 1000)]
    check(lib, oracle, tasks, match=1, mismatch=mismatch, open1=-gap, ext1=-gap)


@pytest.mark.parametrize("mismatch,open1", [(100, -27), (100, -28), (100, -100), (127, -1), (64, -64)])
def test_scores_beyond_the_table(lib, oracle, mismatch, open1):
    """The fast scan holds a score less the opening in eight bits: up to 127 of it, and beyond."""
    read = runs((A, 38))
    tasks = [(runs((C, 300)), read), (runs((A, 40), (C, 3), (A, 40)), read),
             (runs((C, 19), (A, 50), (C, 19)), read[:21])]
    check(lib, oracle, tasks, match=1, mismatch=mismatch, open1=open1, ext1=-1)


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("kw", [dict(open1=-9, min_score=60), dict(open1=-3, min_score=80)], ids=["9", "3"])
def test_whole_alignments(lib, oracle, mode, kw):
    rng = np.random.default_rng(11)
    kw = dict(match=1, mismatch=3, ext1=-1, xdrop=10, pvalue=1e300, **kw)
    found = 0
    for n1, n2 in ((300, 120), (90, 61), (500, 40), (2500, 60)):
        a, b = W.random_pair(rng, n1, n2)
        exp = oracle.find(a, b, two_gap=mode == 2, **kw)[0]
        assert [f.key() for f in lib.align_pairs([(a, b)], mode, **kw)[0]] == [f.key() for f in exp], (n1, n2)
        found += len(exp)
    assert found > 10
