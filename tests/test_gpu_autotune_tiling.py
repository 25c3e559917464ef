"""The autotuner times the seed scan's tiling target only where some scan runs without the filter: with it the target and
its per-bin values stay the default's, whatever the trials' noise; results are the untuned context's either way."""
import numpy as np
import pytest

from dcns_gb300 import workloads as W
from test_gpu_knobs import engine_with, flat

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pairs():
    rng = np.random.default_rng(12)
    out = []
    for _ in range(4200):
        a, b = W.planted_pair(rng, int(rng.integers(150, 700)), int(rng.integers(150, 700)), int(rng.integers(0, 3)), 30,
                              120, 0.8, 0.95, 0.01, 0.0)
        out.append((W.prepare(a), W.prepare(b)))
    return out


@pytest.mark.parametrize("filter", [0, 1])
def test_target(lib, pairs, filter):
    e = engine_with({"DCNS_SCAN_FILTER": str(filter)})
    try:
        before = e.tuning()["scan_tiles_per_thread"]
        batch = e.upload(pairs)
        tuned = e.autotune(batch)
        got = flat(e.align_resident(batch))
        e.free_batch(batch)
    finally:
        e.close()
    assert got == flat(lib.align_pairs(pairs, 1))
    values = {tuned["scan_tiles_per_thread"], *(b["scan_tiles"] for b in tuned["xdrop_per_bin"])}
    assert values == {before} if filter else values <= {4, 8, 16}
