"""Bounded waits of the one-launch stage: the block leaves together or not at
all, since the barriers and tile stores after the wait need every thread (read
from the source: no wait is made to run out on a GPU that others share)."""
import os
import re

from conftest import ROOT


def test_one_launch_stage_leaves_as_a_block():
    src = open(os.path.join(ROOT, "flurrypp_b200", "csrc", "kernels", "stage_fused.cu")).read()
    guards = re.findall(r"if \(!([^\n]*mbar_wait_bounded[^\n]*)\) \{", src)
    assert guards
    for g in guards:
        assert g.startswith("__syncthreads_and("), g
