"""The denominator of the bench's multiply-add fractions: a bound that no kernel
passes."""

import bench


def test_the_peak_is_the_issue_bound_at_the_sampled_clock():
    peak = bench.imad_peak(152, {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0})
    assert abs(peak - 152 * 32 * 2.070e9 / 1e12) < 1e-9
    # chains of products in the kernels' form reach 9.25 TMAC/s
    assert peak > 9.25
    assert bench.imad_peak(152, {"sm_mhz": 1035.0, "sm_max_mhz": 2070.0}) == peak / 2
    assert bench.imad_peak(152, {"sm_mhz": None, "sm_max_mhz": 2070.0}) == peak
    assert bench.imad_peak(152, None) is None and bench.imad_peak(152, {}) is None
