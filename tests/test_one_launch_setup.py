"""One-launch stages are an optimisation: whatever their setup lacks (memory,
tensor maps), the case is set up in the two-kernel form and never refused (read
from the source: neither can be made to fail here)."""
import os
import re

from conftest import ROOT


def test_setup_never_refuses_a_case():
    src = open(os.path.join(ROOT, "flurrypp_b200", "csrc", "fr_case.cu")).read()
    outer = src[src.index("bool setup_fused() {"):src.index("bool setup_fused_as(")]
    inner = src[src.index("bool setup_fused_as("):src.index("bool fused_ok()")]
    assert "fail(" not in inner and "fail(" not in outer
    assert re.search(r"if \(!ok\) \{[^}]*return true;", outer, re.S)
    # what was taken before the maps are known to fit is given back
    assert inner.index("alloc(pool") < inner.index("drop_last()") < inner.index("launch_fused_pack")
