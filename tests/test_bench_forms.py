"""bench.py reports the form a case's steps run in: an explicit tile shape (or
short memory) leaves the two-kernel form, whose kernels are then the ones named."""
import sys
from types import SimpleNamespace

import pytest

import flurrypp_b200 as fb
from conftest import ROOT

CASE = SimpleNamespace(nSpts=64, nFpts=96, nFields=5, nDims=3, nEles=1000)


@pytest.mark.parametrize("wbytes", [4, 8])
@pytest.mark.parametrize("one_launch", [True, False])
def test_kernels_of_both_forms(wbytes, one_launch):
    sys.path.insert(0, ROOT)
    import bench

    def time_ms(kernel):
        if kernel == "stage" and not one_launch:
            raise fb.FrError(fb.FR_ERR_UNSUPPORTED, "this case's stages are two launches")
        return {"stage": 3.0, "element_stage": 2.0, "faces": 1.0}[kernel]

    kms, top = bench.stage_kernels(fb, CASE, wbytes, time_ms)
    words = 5 * 320 + 2 * 480 + 640
    if one_launch:
        assert kms == {"stage": 3.0, "two_kernel_form": {"element_stage": 2.0, "faces": 1.0}}
        assert "k_fused_stage" in top["kernel"] and top["kernel_ms"] == 3.0
        assert top["algorithmic_bytes"] == 1000 * (wbytes * (words + 4 * 96) + 4 * 96)
    else:
        assert kms == {"element_stage": 2.0, "faces": 1.0}
        assert "k_elem_tma" in top["kernel"] and top["kernel_ms"] == 2.0
        assert top["algorithmic_bytes"] == 1000 * wbytes * words


def test_other_errors_are_not_hidden():
    sys.path.insert(0, ROOT)
    import bench

    def time_ms(kernel):
        raise fb.FrError(fb.FR_ERR_CUDA, "launch failed")

    with pytest.raises(fb.FrError):
        bench.stage_kernels(fb, CASE, 8, time_ms)
