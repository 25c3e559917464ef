"""A lone served request starts at once: the best of its times lies within 90 us of the best direct call's on the same
pair (a worker that first waits 100 us for company cannot be that close).  A request whose seed scan takes milliseconds
lets others join, and is exact alone and in company."""
import time

import numpy as np
import pytest

from dcns_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def best(f, n):
    f()
    t = []
    for _ in range(n):
        s = time.perf_counter()
        f()
        t.append(time.perf_counter() - s)
    return min(t)


@pytest.mark.parametrize("max_inflight", [1, 64])
def test_lone_request_starts_at_once(lib, max_inflight):
    rng = np.random.default_rng(2)
    a, b = W.planted_pair(rng, 900, 800, 3, 40, 120, 0.85, 0.97, 0.01, 0.0)
    a, b = W.prepare(a), W.prepare(b)
    direct = best(lambda: lib.align_pairs([(a, b)], 1)[0], 200)
    lib.serve_start(1, max_inflight=max_inflight, workers=2)
    try:
        served = best(lambda: lib.wait(lib.submit(a, b)), 200)
    finally:
        lib.serve_stop()
    assert served < direct + 90e-6, (served, direct)


def test_long_request_and_company(lib):
    rng = np.random.default_rng(3)
    x, y = W.planted_pair(rng, 150000, 150000, 20, 60, 300, 0.8, 0.95, 0.01, 0.0)
    big = (W.prepare(x), W.prepare(y))
    small = []
    for _ in range(3):
        a, b = W.planted_pair(rng, 1500, 1200, 3, 40, 120, 0.85, 0.97, 0.01, 0.0)
        small.append((W.prepare(a), W.prepare(b)))
    want = lib.align_pairs([big] + small, 1)
    lib.serve_start(1, max_inflight=8, workers=2)
    try:
        alone = lib.wait(lib.submit(*big))
        tickets = [lib.submit(a, b) for a, b in [big] + small]
        mixed = [lib.wait(t) for t in tickets]
    finally:
        lib.serve_stop()
    assert alone == want[0] and len(alone) > 0
    for k, m in enumerate(mixed):
        assert m == want[k], k


def test_two_gap_requests_share_a_batch(lib):
    """Admission by predicted bytes: a 2-piece DP keeps checkpoints of 28 bytes per 128 cells, not a byte a cell, so
    requests of 4 kb (16 MB of cells, 11 MB predicted in all, 21 with a byte a cell) share a batch of 100 MB by more than five."""
    rng = np.random.default_rng(4)
    x, y = W.planted_pair(rng, 60000, 60000, 60, 60, 300, 0.8, 0.95, 0.01, 0.0)
    first = (W.prepare(x), W.prepare(y))
    reqs = []
    for _ in range(24):
        a, b = W.planted_pair(rng, 4000, 4000, 3, 40, 120, 0.85, 0.97, 0.01, 0.0)
        reqs.append((W.prepare(a), W.prepare(b)))
    lib.serve_start(2, max_inflight=64, workers=1, batch_cells=10 ** 15, admit_bytes=100 << 20)
    try:
        tickets = [lib.submit(a, b) for a, b in [first] + reqs]  # the first keeps the worker while the others queue
        got = [lib.wait(t) for t in tickets]
        st = lib.serve_stats()
    finally:
        lib.serve_stop()
    assert st["max_batch"] > 5, st
    want = lib.align_pairs([first] + reqs, 2)
    for k, g in enumerate(got):
        assert g == want[k], k
