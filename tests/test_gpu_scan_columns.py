"""SmithWaterman and slidingWindowAlignment batches, whose scan finds every maximum's row first and its column after:
score and first place against the oracle at the edges of the tiling (rows split into one to many waves of chunks), with
ties along a row and a column, runs of N, windows narrower than 38, and sequences shorter than the warm-up."""
import numpy as np
import pytest

from dcns_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def check(eng, oracle, tasks, **kw):
    okw = {{"open1": "open", "ext1": "ext"}.get(k, k): v for k, v in kw.items()}
    out = eng.SmithWaterman(tasks, **kw)
    for k, (a, b) in enumerate(tasks):
        exp = oracle.sw(a, b, **okw)
        assert int(out[k, 0]) == exp[0], k
        if exp[0] > 0:
            assert tuple(int(v) for v in out[k]) == tuple(int(v) for v in exp[:3]), k


@pytest.mark.parametrize("n", [1, 3, 64, 700, 6000])
def test_tilings(lib, oracle, n):
    rng = np.random.default_rng(n)
    tasks = []
    for k in range(n):
        n1, n2 = int(rng.integers(1, 60 if n > 1000 else 900)), int(rng.integers(1, 39))
        a, b = W.random_pair(rng, n1, n2)
        if n1 > n2 and k % 2:
            at = int(rng.integers(0, n1 - n2 + 1))
            a[at:at + n2] = b
            if k % 4 == 1 and n1 > 2 * n2:  # the same maximum twice
                a[:n2] = b
        tasks.append((a, b))
    check(lib, oracle, tasks)


def test_few_long_references(lib, oracle):
    rng = np.random.default_rng(5)
    tasks = []
    for n1 in (159, 160, 161, 5000, 20011):
        a, b = W.random_pair(rng, n1, 38)
        tasks.append((a, b))
        c = a.copy()
        c[n1 - 30:] = b[:30]
        tasks.append((c, b))
        c = a.copy()
        c[:38] = 2
        tasks.append((c, np.concatenate([b[:20], b[:18]])))
    check(lib, oracle, tasks)
    check(lib, oracle, tasks, open1=-2, ext1=-1)


def test_ties_along_a_row(lib, oracle):
    a = np.array([0, 0, 0, 1, 0, 0, 0, 3, 0, 0, 0], np.int8)
    tasks = [(a, np.zeros(k, np.int8)) for k in (1, 2, 3, 7, 38)] + [(np.zeros(200, np.int8), np.zeros(38, np.int8))]
    check(lib, oracle, tasks)


@pytest.mark.parametrize("n", [5, 38, 200, 3001])
def test_sliding(lib, oracle, n):
    rng = np.random.default_rng(n)
    seqs = [W.random_pair(rng, n, 1)[0] for _ in range(4)]
    seqs[2][:n // 2] = seqs[0][:n // 2]
    score, most = lib.slidingWindowAlignment(seqs)
    for i in range(1, 4):
        exp_s, exp_m = oracle.sliding(seqs[0], seqs[i])
        assert np.array_equal(most[i - 1], exp_m) and np.array_equal(score[i - 1], exp_s), i
