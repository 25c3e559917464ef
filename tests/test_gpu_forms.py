"""Every form of the scan and the two-piece DPs that a setting or the autotuner chooses gives the default's results:
without the filter (whole windows, in few and in many tiles), the stripe flow on one block per SM, and one CTA per DP
with two, four and eight warps."""
import pytest

from test_gpu_knobs import defaults, engine_with, flat, sample, short_pairs  # noqa: F401

pytestmark = pytest.mark.gpu

FORMS = [
    {"DCNS_SCAN_FILTER": "0"},
    {"DCNS_SCAN_FILTER": "0", "DCNS_SCAN_TILES": "1"},
    {"DCNS_SCAN_FILTER": "0", "DCNS_SCAN_TILES": "16"},
    {"DCNS_SG_FLOW_BLOCKS": "1"},
    {"DCNS_SG_FLOW": "0", "DCNS_SG_WARPS": "2"},
    {"DCNS_SG_FLOW": "0", "DCNS_SG_WARPS": "4"},
    {"DCNS_SG_FLOW": "0", "DCNS_SG_WARPS": "8"},
]


@pytest.mark.parametrize("env", FORMS, ids=lambda e: ",".join(f"{k}={v}" for k, v in e.items()))
def test_forms_give_the_default_results(env, sample, defaults):  # noqa: F811
    e = engine_with(env)
    try:
        t = e.tuning()
        if "DCNS_SCAN_TILES" in env:
            assert t["scan_tiles_per_thread"] == int(env["DCNS_SCAN_TILES"])
        if "DCNS_SG_FLOW_BLOCKS" in env:
            assert t["sg_flow_blocks"] == int(env["DCNS_SG_FLOW_BLOCKS"])
        if "DCNS_SG_WARPS" in env:
            assert not t["sg_flow"] and t["sg_warps"] == int(env["DCNS_SG_WARPS"])
        assert flat(e.align_pairs(sample, 1)) == defaults["one"]
        assert flat(e.align_pairs(sample[:200], 2)) == defaults["two"]
        if "DCNS_SCAN_FILTER" in env:
            assert flat(e.align_pairs(sample[:1], 1)) == defaults["one"][:1]
    finally:
        e.close()
