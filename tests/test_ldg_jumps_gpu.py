"""The LDG jumps dUc_fpts of FP32 3-D viscous cases, which the gradient kernel
forms (rows with TMA tiles) and stores only where a caller can look at them.

A jump 0.5 (ul + ur) - pen (ul - ur) - u has at most five roundings of values
below 2 max|U|: 5 * 2 * 2^-24 < 6e-7 of the largest trace.  After steps the two
forms' traces differ by the state's own rounding, at most 50 roundings a stage
over 16 stages: 50 * 16 * 2^-24 = 5e-5."""
import numpy as np
import pytest

import flurrypp_b200 as fb
from flurrypp_b200.decks import write_deck

pytestmark = pytest.mark.gpu

WALLS = dict(create_bcBottom="adiabatic_noslip", create_bcTop="slip_wall", create_bcLeft="char", create_bcRight="char")


@pytest.mark.parametrize("order", range(1, 6))
@pytest.mark.parametrize("walls", [{}, WALLS])
def test_jumps(tmp_path, order, walls):
    d = write_deck(str(tmp_path / "v.deck"), nDims=3, order=order, meshType=1, nx=4, ny=3, nz=3, xmin=0, ymin=0, zmin=0,
                   xmax=1, ymax=1, zmax=1, viscous=1, Re=100, MachBound=0.3, prandtl=0.71, fixVis=1, LDG_tau=0.1,
                   LDG_penFact=0.5, TBound=291.15, TGas=291.15, MachWall=0, CFL=0.1, **walls)
    both, dt = [], None
    for opts in ({}, {"no_tma": 1}):
        s = fb.Solver(d, precision=fb.FR_PREC_MIXED, **opts)
        assert s.info().tensor_kernels == (1 if opts else 2)
        s.initialize_solution(fb.IC_UNIFORM)  # the free stream, disturbed by 1 % of each value
        s.set_state(s.get_state() * (1 + np.random.default_rng(7).uniform(-0.01, 0.01, s.shape)))
        dt = dt or 0.1 * s.calc_dt()
        s.set_dt(dt)
        s.calc_residual(0)
        E, nPF = s.nEles, (order + 1) ** 2
        U = s.get_array("U_fpts").reshape(-1, 5)
        J = s.get_array("dUc_fpts").reshape(-1, 5)
        n = s.get_array("norm_fpts").reshape(-1, 3)
        eL, locL, eR = (s.get_array("face_" + k).astype(int) for k in ("eL", "locL", "eR"))
        fR = s.get_array("face_fptR").astype(int).reshape(-1, nPF)
        inner = eR >= 0
        sL = ((locL[inner, None] * nPF + np.arange(nPF)) * E + eL[inner, None]).ravel()
        sR = (fR[inner] * E + eR[inner, None]).ravel()
        pen = np.where(n[sL, 0] + n[sL, 1] + np.sqrt(2) * n[sL, 2] < 0, -0.5, 0.5)[:, None]
        uc = 0.5 * (U[sL] + U[sR]) - pen * (U[sL] - U[sR])
        tol = 6e-7 * np.abs(U).max()
        assert np.abs(J[sL] - (uc - U[sL])).max() <= tol and np.abs(J[sR] - (uc - U[sR])).max() <= tol
        seen = [J]
        for call in (lambda: s.run(3), s.update, lambda: s.run(2), lambda: s.calc_residual(0)):
            call()
            seen.append(s.get_array("dUc_fpts").reshape(-1, 5))
        assert np.isfinite(seen[-1]).all()
        assert not any(np.array_equal(a, b) for a, b in zip(seen, seen[1:]))  # the steps move them
        both.append(seen)
    scale = np.abs(U).max()
    for a, b in zip(*both):
        assert np.abs(a - b).max() <= 5e-5 * scale
