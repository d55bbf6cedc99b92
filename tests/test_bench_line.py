"""The benchmark's roofline is that of the kernel that ran."""
import bench


def test_roofline_names_and_measures_the_kernel_that_ran():
    # 31 ms for 2e8 crossings: at the tree searches' 3,262 bytes each it would be
    # three times the memory's rate
    r = bench.roofline("clustered_2m", "list", 198_903_587, 31.0)
    assert r["kernel"].startswith("k_list") and "tree" not in r["bytes"]
    assert 0.0 < r["frac"] < 1.0 and r["traffic"] < 100 * 198_903_587
    # the list walk's traffic is not known there
    assert bench.roofline("nested_16m", "list", 1_000_000_000, 150.0) is None
    r = bench.roofline("nested_16m", "thread_fp32", 785_000_000, 585.0)
    assert r["kernel"].startswith("k_batched") and r["bytes_per_crossing"] == bench.BX["nested_16m"]
    assert bench.roofline("clustered_2m", "list", 198_903_587, None) is None
