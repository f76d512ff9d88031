"""Reduced-rank extrapolation for every number of snapshots (GPU): the Gram
kernel is compiled per number of differences, and a lane takes whole 16-byte
vectors of a ragged velocity count.  The coefficients must minimise
|sum gamma_j u_j| (against a float64 solve on the same snapshots) and the state
must be max(sum gamma_j x_j, 0) of the coefficients returned."""
import numpy as np
import pytest

from dgbgk import Solver, channel_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", range(2, 12))
@pytest.mark.parametrize("prec", [64, 32])
def test_extrapolation_of_n_snapshots(n, prec):
    c = channel_case(-2.0, 4.0, -2.0, 2.0, 21, 14, 5, 7, mach=2.0, kn=0.05, obstacle_side=1.0)
    s = Solver.from_case(c, precision=prec)
    s.init_case()
    x = []
    for k in range(n):
        s.advance(7)
        s.snapshot(k)
        x.append(s.get_state().ravel())
    g = s.extrapolate(n)
    u = np.diff(np.array(x), axis=0)
    G = u @ u.T
    ref = np.linalg.solve(G + 1e-14 * np.trace(G) * np.eye(n - 1), np.ones(n - 1))
    ref /= ref.sum()
    assert abs(g.sum() - 1.0) <= 1e-12
    # the objective at both solutions: the sums of the Gram matrix agree to 1e-12, its
    # condition enters the coefficients but not the minimum they reach
    got, best = np.linalg.norm(g @ u), np.linalg.norm(ref @ u)
    assert got <= best * (1 + 1e-6) + 1e-12 * np.linalg.norm(u)
    want = np.maximum(g @ np.array(x[:-1]), 0.0)
    tol = 1e-13 if prec == 64 else 1e-7
    assert np.linalg.norm(s.get_state().ravel() - want) <= tol * (1 + np.abs(g).sum()) * np.linalg.norm(want)
