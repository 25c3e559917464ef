"""The seed-scan filter on references that hold a short word again and again: 17 bases between A's on one side and C's
on the other score 34, which marks the place (32) and seeds nothing (40).  Words of 27 bases' distance mark everything
(the filter stops computing, the plan's rows pass the whole scan's and every window is scanned), of 60 nearly everything
once the warm-up joins the runs, of 120 a third (many short runs: a list longer than it was made).  With planted matches
among them, for seeds and recursion rounds; references of several segments of the plan's words, with matches around
their borders.  Fragments as from a context that scans every window against its whole reference."""
import numpy as np
import pytest

from test_gpu_scan_filter import engines, same  # noqa: F401

pytestmark = pytest.mark.gpu

WORD = np.array([3, 4, 4, 3, 4, 3, 3, 4, 3, 4, 4, 4, 3, 3, 4, 3, 4], np.int8)


def grid(n, sep, period, phase=0):
    x = np.full(n, sep, np.int8)
    for at in range(phase, n - len(WORD), period):
        x[at:at + len(WORD)] = WORD
    return x


def pair(rng, n1, n2, period, planted, length=60):
    a, b = grid(n1, 0, period), grid(n2, 1, period, period // 3)
    for _ in range(planted):
        m = rng.choice(np.array([0, 1, 3, 4], np.int8), length)
        p, q = int(rng.integers(0, n1 - length + 1)), int(rng.integers(0, n2 - length + 1))
        a[p:p + length], b[q:q + length] = m, m
    return a, b


@pytest.mark.parametrize("period", [27, 60, 120])
@pytest.mark.parametrize("n1,n2", [(1000, 900), (40000, 700), (9000, 9500), (30011, 29999)])
def test_one_pair(engines, period, n1, n2):  # noqa: F811
    rng = np.random.default_rng(n1 + period)
    assert same(engines, None, [pair(rng, n1, n2, period, 0)]) == 0
    assert same(engines, None, [pair(rng, n1, n2, period, 6)]) > 0


def test_one_marked_pair_among_others(engines):  # noqa: F811
    rng = np.random.default_rng(1)
    pairs = [pair(rng, int(rng.integers(500, 3000)), int(rng.integers(500, 3000)), (27, 60, 120, 5000)[k % 4], 2)
             for k in range(40)]
    assert same(engines, None, pairs) > 0


@pytest.mark.parametrize("period", [120, 10 ** 6])
def test_references_of_several_segments(engines, period):  # noqa: F811
    """128 words of 512 rows and their overlap make a segment of the plan: matches every 250 rows cross every border."""
    rng = np.random.default_rng(period)
    a, b = grid(150000, 0, period), grid(420, 1, period, 40)
    m = rng.choice(np.array([0, 1, 3, 4], np.int8), 60)
    b[200:260] = m
    for at in range(100, 149900, 250):
        a[at:at + 60] = m
    assert same(engines, None, [(a, b)]) > 100
