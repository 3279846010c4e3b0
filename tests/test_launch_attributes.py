"""Kernel attributes belong to the kernel, not to a launch or a thread, and setting one
clears the thread's last error: the sources set them through set_attribute (which
keeps an error that is there), and raise the shared-memory limit to constants."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "exanbody_gb300", "csrc")


def sources():
    return {os.path.basename(p): open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu*"))}


def test_set_in_one_place():
    sites = {f: s.count("cudaFuncSetAttribute(") for f, s in sources().items() if "cudaFuncSetAttribute(" in s}
    # the allocation-free entry point sets constants and returns their errors itself
    assert sites == {"xnb_launch.cuh": 1, "xnb_static_scratch.cu": 2}


def test_limits_do_not_follow_a_launch():
    calls = [a for s in sources().values() for a in re.findall(r"raise_smem_limit\(\w+(?:<[^>]*>)?, (.*?)\);", s)]
    assert len(calls) >= 6
    constant = re.compile(r"(k[A-Z]\w*|sizeof\(\w+\)|sub_stage_offset\(4\)|warps|\d+u?|[ *+()])+$")
    assert all(constant.match(a) or a == "smem" for a in calls), calls
    # the one named `smem` is the size of a fixed struct
    assert "const size_t smem = 4 * sizeof(RowsWarp);" in sources()["xnb_build_rows.cu"] and calls.count("smem") == 1
