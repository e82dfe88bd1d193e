"""One-launch stages give the two-kernel form's bits where both add the same
terms in the same order: in 2-D, and in FP32 3-D with rows that allow TMA tiles
(element counts that are multiples of 4) and rows that do not.  FP64 3-D adds
the correction line by line and is held to a tolerance elsewhere."""
import numpy as np
import pytest

import flurrypp_b200 as fb
from flurrypp_b200.decks import write_deck

pytestmark = pytest.mark.gpu

WALLS = dict(create_bcBottom="slip_wall", create_bcTop="slip_wall", create_bcLeft="char", create_bcRight="char")
FORMS = ([(fb.FR_PREC_FP64, s) for s in ((5, 3), (16, 8))] +
         [(fb.FR_PREC_MIXED, s) for s in ((5, 3), (16, 8), (6, 4, 4), (7, 5, 3), (5, 5, 3), (3, 3, 2))])


@pytest.mark.parametrize("prec,size", FORMS)
@pytest.mark.parametrize("order", range(6))
@pytest.mark.parametrize("walls", [{}, WALLS])
def test_arrays_equal(tmp_path, prec, size, order, walls):
    nd = len(size)
    o = dict(nDims=nd, order=order, meshType=1, dt=0.002, uBound=0.35, pBound=0.7142857143, **walls)
    for name, n in zip("xyz", size):
        o.update({"n" + name: n, name + "min": 0, name + "max": 1.0})
    d = write_deck(str(tmp_path / "b.deck"), **o)
    v = np.array([0.35, 0.1, 0.05])[:nd]
    u = np.concatenate([[1.0], v, [0.7142857143 / 0.4 + 0.5 * (v @ v)]])
    got = []
    for variant in (-1, 0):
        s = fb.Solver(d, precision=prec, tile_variant=variant)
        s.set_state(u * (1 + np.random.default_rng(7).uniform(-0.01, 0.01, s.shape)))
        s.calc_residual(0)
        first = [s.get_array("divF_0"), s.get_array("Fn_fpts"), s.residual_norm(2)]
        s.run(3)
        got.append(first + [s.get_array(n) for n in ("U_spts", "U0", "U_fpts", "Fn_fpts", "waveSp_fpts", "divF_0")])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
