"""The residual norm reduced on the device against the same sum in numpy.

Both add up to 6e3 non-negative terms of a few roundings each: they agree to
1e-12 relative (6e3 * 2^-53 = 7e-13); maxima to a few ulps."""
import numpy as np
import pytest

import flurrypp_b200 as fb
from flurrypp_b200.decks import write_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [fb.FR_PREC_FP64, fb.FR_PREC_MIXED])
@pytest.mark.parametrize("order,size", [(0, (3, 3)), (1, (3, 3)), (3, (17, 23)), (2, (5, 4, 3)), (3, (5, 5, 4))])
@pytest.mark.parametrize("res_type", [1, 2, 3])
def test_norm_matches_numpy(tmp_path, prec, order, size, res_type):
    o = dict(nDims=len(size), order=order, meshType=1, dt=0.001)
    for name, n in zip("xyz", size):
        o.update({"n" + name: n, name + "min": 0, name + "max": 1.0})
    s = fb.Solver(write_deck(str(tmp_path / "n.deck"), **o), precision=prec)
    u = np.array([1.0] + [0.3, 0.1, 0.2][:s.nDims] + [2.0])
    s.set_state(u * (1 + np.random.default_rng(5).uniform(-0.05, 0.05, s.shape)))
    s.calc_residual(0)
    got = s.residual_norm(res_type)
    again = s.residual_norm(res_type)
    d = np.abs(s.get_residual(0))
    J = s.get_array("detJac_spts").reshape(s.nSpts, s.nEles, 1)
    x, w1 = np.polynomial.legendre.leggauss(order + 1)
    w = w1
    for _ in range(s.nDims - 1):
        w = np.multiply.outer(w, w1)
    w = w.reshape(-1, 1, 1)
    want = {1: lambda: (d * w).sum((0, 1)), 2: lambda: np.sqrt((d * d / J * w).sum((0, 1))),
            3: lambda: (d / J).max((0, 1))}[res_type]()
    assert np.array_equal(got, again)  # the counter is ready for the next call
    assert np.max(np.abs(got - want) / np.maximum(want, 1e-300)) <= 1e-12
