"""Extension with CIGARs under device budgets of little more than the codes themselves: the traceback arena takes what the
budget leaves, passes that find it full run again in rounds of as many as fit, and the results are those of a context
without a limit.  The budgets are ones that held when a pass's slot took 4 bits a cell without the lanes' padding
(2.3 times less at a band of 11)."""
import numpy as np
import pytest

import dcns_gb300

pytestmark = pytest.mark.gpu

BASES = np.array([0, 1, 3, 4], np.int8)


@pytest.fixture(scope="module")
def tasks():
    rng = np.random.default_rng(77)
    out = []
    for _ in range(400):
        n = int(rng.integers(200, 3000))
        a = BASES[rng.integers(0, 4, n)]
        b = a.copy()
        m = rng.random(n) > .9
        b[m] = BASES[rng.integers(0, 4, int(m.sum()))]
        out.append((a, b))
    return out


@pytest.mark.parametrize("w,mb", [(10, 60), (11, 64), (22, 80), (50, 96), (100, 150), (300, 380), (400, 700)])
def test_accepted_and_exact(lib, tasks, w, mb):
    e = dcns_gb300.Engine(0, mem_budget=mb << 20)
    try:
        want, want_cigars = lib.SemiGlobal_xextend(tasks, cigar=True, w=w, xdrop=50)
        for _ in range(2):  # the second call on the buffers that the first one grew
            got, cigars = e.SemiGlobal_xextend(tasks, cigar=True, w=w, xdrop=50)
            assert np.array_equal(got, want) and cigars == want_cigars
    finally:
        e.close()
