"""The reverse scan of short windows (its DP row in registers) against the oracle's seeds: windows of every width up to
38 and just above (the general form), queries that end inside a window, matches at the first and last bases, N."""
import numpy as np
import pytest

from dcns_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window,min_score", [(38, 40), (37, 40), (31, 40), (22, 40), (39, 40), (60, 40)])
def test_windows(lib, oracle, window, min_score):
    rng = np.random.default_rng(window)
    pairs = []
    for k in range(12):
        n1, n2 = int(rng.integers(40, 400)), int(rng.integers(22, 300))
        a, b = W.planted_pair(rng, max(n1, 120), max(n2, 60), 4, 25, 55, 0.85, 1.0, 0.03, 0.0)
        a, b = W.prepare(a)[:n1], W.prepare(b)[:n2]
        if k % 3 == 0:
            m = min(len(a), len(b), 30)
            a[:m] = b[:m]          # a match that starts at the first bases
            a[-m:] = b[-m:]        # and one that ends at the last
        if k % 4 == 1:
            a[rng.integers(0, len(a), 3)] = 2
            b[rng.integers(0, len(b), 3)] = 2
        pairs.append((a, b))
    kw = dict(window=window, min_score=min_score, pvalue=1e300)
    got = lib.align_pairs(pairs, **kw)
    found = 0
    for k, (a, b) in enumerate(pairs):
        exp, _ = oracle.find(a, b, **kw)
        assert [f.key() for f in got[k]] == [f.key() for f in exp], k
        found += len(exp)
    assert found > 10
