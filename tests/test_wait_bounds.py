"""Bounded waits of the one-launch stage: no thread leaves its block early, since
the barriers and tile stores after the wait need every thread; a wait that ran
out is flagged for the host (read from the source: no wait is made to run out on
a GPU that others share)."""
import os
import re

from conftest import ROOT


def test_one_launch_stage_stays_together():
    src = open(os.path.join(ROOT, "flurrypp_b200", "csrc", "kernels", "stage_fused.cu")).read()
    body = src[src.index("    k_fused_stage("):src.index("// Thread-order copies")]
    guard = re.search(r"if \(!mbar_wait_bounded\([^\n]*\) \{(.*?)\n    \}", body, re.S)
    assert guard and "atomicOr(a.err" in guard[1] and "mbar_wait_bounded" in guard[1] and "return" not in guard[1]
    # the only exit is the residual's, which all threads of a launch take
    assert re.findall(r"[^\n]*\breturn;", body) == ["  if (residual) return;"]
