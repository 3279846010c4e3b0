"""bench.py names the force kernel that its settings run and reports DRAM traffic for
the captured kernel alone."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


@pytest.mark.parametrize("n,lanes,form,kernel", [
    (32000, 0, "", "k_force_mixed"), (32000, 4, "", "k_force_mixed"), (32000, 0, "staged", "k_force_staged"),
    (108000, 1, "", "k_force<mixed>"), (108000, 2, "", "k_force_lanes"), (4000000, 0, "thread", "k_force_walk"),
    (4000000, 2, "", "k_force_lanes"), (4000000, 0, "staged", "k_force_staged"),
])
def test_force_record(n, lanes, form, kernel):
    assert bench.mixed_force_kernel(n, lanes, form) == kernel
    r = bench.force_traffic(kernel, n, 2.0)
    if kernel == "k_force_walk":
        assert r["traffic"] == bench.FORCE_DRAM_BYTES_PER_ATOM * n
        assert r["hbm"]["achieved_gbs"] == pytest.approx(r["traffic"] / 2e-3 / 1e9)
    else:
        assert r["traffic"] is None and r["hbm"] is None


@pytest.mark.parametrize("n,fits", [(20, True), (100, False)])
def test_flush_text_follows_the_state(n, fits):
    assert ("stays in L2" in bench.config_of(n, 4 * n**3)["flush"]) == fits
