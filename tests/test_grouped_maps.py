"""The host side of the grouped products on tcgen05 (csrc/gemm_grouped_tc.cu): no launch without all of its tensor maps."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm-rs_b200", "csrc")


def test_every_tensor_map_is_checked_before_the_launch():
    """A map that the driver refuses leaves its variable unset: a kernel that reads it would fault, so this is read, not run."""
    with open(os.path.join(CSRC, "gemm_grouped_tc.cu")) as f:
        body = f.read().split("int launch_grouped_tc(", 1)[1].split("<<<", 1)[0]
    calls = re.findall(r"^.*gt_map\(&.*$", body, re.M)
    assert len(calls) == 3
    assert all(re.search(r"if \(\(rc = gt_map\(&.*\)\) != 0\) return rc;", c) for c in calls), calls
