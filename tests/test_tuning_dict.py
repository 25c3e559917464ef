"""Tuning.as_dict reports what the library sets; the x-drop forms that no longer exist have no value, not a zero."""
import dcns_gb300


def test_forms_without_a_value():
    t = dcns_gb300.Tuning()
    t.n_bins_tuned = 3
    for b in range(3):
        t.scan_tiles[b] = 4 + b
    bins = t.as_dict()["xdrop_per_bin"]
    assert [x["scan_tiles"] for x in bins] == [4, 5, 6]
    for x in bins:
        assert set(x) == {"warp_from", "wave_max_w", "row_interleaved", "handoff_rows", "handoff_lanes",
                          "groups_from_band", "scan_tiles"}
        assert all(v is None for k, v in x.items() if k != "scan_tiles")
