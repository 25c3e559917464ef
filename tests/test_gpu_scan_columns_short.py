"""SmithWaterman on references around the lengths where the scan changes its form: up to a warm-up of rows whole, up to
four warm-ups with the maximum's column found on the way, beyond that by a second DP; few tasks in chunks, many whole.
Scores and first places against the oracle, with maxima at the start, at the end and twice."""
import numpy as np
import pytest

from dcns_gb300 import workloads as W
from test_gpu_scan_columns import check

pytestmark = pytest.mark.gpu


def tasks_of(rng, rows, n):
    out = []
    for k in range(n):
        n1, n2 = rows[k % len(rows)], (38, 38, 37, 20, 1)[k % 5]
        a, b = W.random_pair(rng, n1, n2)
        if k % 3 == 1 and n1 >= n2:
            a[n1 - n2:] = b
        if k % 3 == 2 and n1 >= 2 * n2:
            a[:n2] = b
            a[n1 - n2:] = b
        out.append((a, b))
    return out


@pytest.mark.parametrize("n", [1, 7, 300, 11000])
@pytest.mark.parametrize("rows", [(79, 80, 81), (119, 120, 121), (160, 161), (319, 320), (319, 320, 321), (322, 90, 5)],
                         ids=lambda r: "-".join(map(str, r)))
def test_lengths_at_the_lines(lib, oracle, rows, n):
    rng = np.random.default_rng(sum(rows) + n)
    check(lib, oracle, tasks_of(rng, rows, n if n < 1000 or rows[0] in (119, 319) else 900))


def test_other_gaps(lib, oracle):
    """Warm-ups of 22 to 1,144 rows."""
    rng = np.random.default_rng(9)
    for kw in (dict(open1=-20, ext1=-20), dict(open1=-1, ext1=-1), dict(match=30, mismatch=-30, open1=-2, ext1=-1),
               dict(open1=0, ext1=0)):
        check(lib, oracle, tasks_of(rng, (60, 120, 500, 1300), 40), **kw)
