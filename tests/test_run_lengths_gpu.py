"""fr_run replays graphs captured per number of steps; whatever was captured
when, a run equals update (and the P-multigrid cycle) step by step, bit for
bit, also after a new state, a residual evaluation or an output in between."""
import numpy as np
import pytest

import flurrypp_b200 as fb
from conftest import deck_path, has_pmg, load_golden, perturb_opts
from flurrypp_b200.decks import write_deck

pytestmark = pytest.mark.gpu

PRECS = [fb.FR_PREC_FP64, fb.FR_PREC_MIXED]


def steps(s, pmg, n):
    for _ in range(n):
        s.update()
        if pmg:
            s.pmg_cycle()


# calls on one solver: ("run", n), ("state", factor), ("residual",), ("csv",)
SEQUENCES = {
    "new state": [("run", 10), ("state", 1.01), ("run", 5), ("run", 5), ("run", 5)],
    "residual": [("run", 10), ("state", 1.01), ("run", 1), ("residual",), ("run", 5), ("run", 5), ("run", 5), ("residual",)],
    "output": [("run", 25), ("csv",), ("run", 25), ("state", 1.01), ("run", 3), ("run", 3), ("residual",)],
    # lengths that come back often enough for a graph of their own, and one more
    "returning": [("run", 2), ("run", 3)] * 5 + [("residual",)] + [("run", 2), ("run", 3)] * 40 + [("residual",), ("run", 2)],
    "chunks": [("run", 1), ("state", 1.01), ("run", 10), ("run", 10), ("residual",), ("run", 20), ("residual",)],
}


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("case", ["pmg_vortex2d_p3_8", "pmg_tgv3d_p3_3", "vortex2d_p3_8", "pmg_ns_vortex2d_p3"])
@pytest.mark.parametrize("sequence", SEQUENCES)
def test_run_equals_steps(tmp_path, prec, case, sequence):
    a, meta = load_golden(case)
    equal(tmp_path, lambda: fb.Solver(deck_path(meta), precision=prec, **perturb_opts(meta)), a["U_init"], has_pmg(meta), sequence)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("sequence", ["new state", "residual"])
def test_one_launch_levels(tmp_path, prec, sequence):
    """P-multigrid above the size up to which its cases keep two launches a stage."""
    d = write_deck(str(tmp_path / "p.deck"), nDims=2, order=2, meshType=1, nx=132, ny=130, xmin=0, xmax=1, ymin=0, ymax=1,
                   dtType=2, CFL=0.3, PMG=1, lowOrder=0, smoothSteps=2, uBound=0.35)
    make = lambda v=-1: fb.Solver(d, precision=prec, tile_variant=v)
    s = make()
    U = np.array([1.0, 0.35, 0.1, 2.0]) * (1 + np.random.default_rng(7).uniform(-0.001, 0.001, s.shape))
    assert launches(make, U) < launches(lambda: make(0), U)
    equal(tmp_path, make, U, True, sequence)


@pytest.mark.parametrize("prec", PRECS)
def test_small_levels_keep_two_launches(prec):
    a, meta = load_golden("pmg_vortex2d_p3_8")
    n = [launches(lambda: fb.Solver(deck_path(meta), precision=prec, tile_variant=v), a["U_init"]) for v in (-1, 0)]
    assert n[0] == n[1]


def launches(make, U):
    s = make()
    s.set_state(U)
    s.run(2)
    n = s.info().launches
    s.run(1)
    return s.info().launches - n


def equal(tmp_path, make, U, pmg, sequence):
    both = []
    for graph in (True, False):
        s = make()
        s.set_state(U)
        seen = []
        for call in SEQUENCES[sequence]:
            if call[0] == "run":
                s.run(call[1]) if graph else steps(s, pmg, call[1])
                seen.append(s.get_state())
            elif call[0] == "state":
                s.set_state(call[1] * U)
            elif call[0] == "residual":
                s.calc_residual(0)
                seen += [s.get_residual(0), s.get_array("Fn_fpts")]
            else:
                s.write_data(str(tmp_path / "out"))
        assert np.isfinite(seen[-1]).all()
        both.append(seen)
    for x, y in zip(*both):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("prec", PRECS)
def test_member_runs_on_after_a_batch(prec):
    """A batch member whose graphs were built before the batch stepped its state."""
    a, meta = load_golden("vortex2d_p3_8")
    ends = []
    for graph in (True, False):
        s = fb.Solver(deck_path(meta), precision=prec)
        s.set_state(a["U_init"])
        s.run(3)
        s.run(2)
        s.run(2)
        b = fb.Batch([s])
        b.set_form(fb.FR_BATCH_GROUPS)  # the other form rounds differently, and the choice is timed
        b.run(4)
        b.gather()
        s.run(2) if graph else steps(s, False, 2)
        ends.append(s.get_state())
    assert np.array_equal(*ends)
