"""fr_run replays graphs captured per number of steps; whatever was captured
when, a run equals update (and the P-multigrid cycle) step by step, bit for
bit, also after a new state, a residual evaluation or an output in between."""
import numpy as np
import pytest

import flurrypp_b200 as fb
from conftest import deck_path, has_pmg, load_golden, perturb_opts

pytestmark = pytest.mark.gpu

PRECS = [fb.FR_PREC_FP64, fb.FR_PREC_MIXED]


def steps(s, meta, n):
    for _ in range(n):
        s.update()
        if has_pmg(meta):
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
    both = []
    for graph in (True, False):
        s = fb.Solver(deck_path(meta), precision=prec, **perturb_opts(meta))
        s.set_state(a["U_init"])
        seen = []
        for call in SEQUENCES[sequence]:
            if call[0] == "run":
                s.run(call[1]) if graph else steps(s, meta, call[1])
                seen.append(s.get_state())
            elif call[0] == "state":
                s.set_state(call[1] * a["U_init"])
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
        b.run(4)
        b.gather()
        s.run(2) if graph else steps(s, meta, 2)
        ends.append(s.get_state())
    assert np.array_equal(*ends)
