"""The residual's flux arithmetic (reciprocals and roots by one third-order step, logarithmic means on
both sides of their series threshold) against the CPU oracle, where it can go wrong: neighbouring nodes
that differ by less and by more than the threshold, a vanishing field (zero roots), a uniform state."""
import numpy as np
import pytest

from conftest import rel_l1
from test_gpu_parity import _perturbed

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("field", [True, False])
@pytest.mark.parametrize("scale", [0.004, 0.02, 0.2])
def test_residual_of_rough_states(pkg, ora, p, field, scale):
    """tolerance: nodal values that differ by the fraction `scale` make differences of fluxes whose
    rounding errors, a few EPS of the flux each, are 1/scale times larger relative to the difference;
    20 roundings of one sign and 2 for the oracle's own"""
    prob = pkg.problems.make("ot2pi")
    nx, ny = 17, 11
    u = prob.initial_state(nx, ny, p)
    if not field:
        u[7] -= 0.5 * (u[4] ** 2 + u[5] ** 2 + u[6] ** 2)
        u[4:7] = 0.0
    u = np.asfortranarray(_perturbed(u, 11, scale, prob.gamma))
    if not field:
        u[7] -= 0.5 * (u[4] ** 2 + u[5] ** 2 + u[6] ** 2)
        u[4:7] = 0.0
    o = ora.OracleSolver(nx, ny, p, p, 3, *prob.domain, prob.gamma, prob.bc_kind, prob.bc_state)
    o.apply_bc(u)
    want, dl_o = o.semidiscretize(u)
    with pkg.DGSolver.for_problem(prob, nx, ny, p) as g:
        g.upload_state(0, u)
        dl = g.semidiscretize(1, 0)
        got = g.download_ut(1)
    assert rel_l1(got, want, floor_frac=1e-2).max() <= 22 * EPS / scale
    assert abs(dl - dl_o) <= 20 * EPS * dl_o


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("b", [0.0, 3.0])
def test_residual_of_a_uniform_state(pkg, p, b):
    """the exact residual is zero; what is left is rounding: the largest flux (velocity times the total
    energy density, 1 * 40) times 2/h times the largest coefficient (6), a few EPS"""
    prob = pkg.problems.make("ot2pi")
    nx, ny = 9, 7
    u = np.full((8, p + 1, p + 1, nx + 2, ny + 2), np.nan, order="F")
    w = np.array([1.3, 0.7, -0.9, 0.2, b, -0.5 * b, 0.25 * b, 20.0])
    u[...] = w[:, None, None, None, None]
    with pkg.DGSolver.for_problem(prob, nx, ny, p) as g:
        g.upload_state(0, u)
        g.semidiscretize(1, 0)
        got = g.download_ut(1)
    assert np.abs(got).max() <= 16 * EPS * 40 * 6 * 2 / (2 * np.pi / max(nx, ny))
