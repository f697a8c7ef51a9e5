"""dt_lim of states that hold an inadmissible density (GPU).  The residual forms a node's exact speeds only where a bound of
them could lower dt_lim; a node of negative density, whose bound is NaN, and one of density zero, whose speed
is infinite, count all the same (DG_solver.f90:776-789: the clamped speed |v| + c).  On meshes of more items than
run at once, so that the last ones find dt_lim set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(pkg, ora, nx, ny, p, w):
    prob = pkg.problems.make("ot2pi")
    u = prob.initial_state(nx, ny, p)
    u[:, 1, 1, nx, ny] = w
    u = np.asfortranarray(u)
    o = ora.OracleSolver(nx, ny, p, p, 3, *prob.domain, prob.gamma, prob.bc_kind, prob.bc_state)
    o.apply_bc(u)
    return prob, u, o


SIZES = [(1, 300, 260), (2, 200, 121), (3, 160, 145)]


@pytest.mark.parametrize("p,nx,ny", SIZES)
def test_negative_density(pkg, ora, p, nx, ny):
    """the node's gas pressure is at its clamp, 1e-11, so its speeds are |v| = 50, 30 to 4e-6, by far the largest.
    Tolerance: 20 roundings"""
    prob, u, o = _state(pkg, ora, nx, ny, p, [-1.0, 50.0, 30.0, 0.0, 0.0, 0.0, 0.0, -1.0e6])
    want = o.semidiscretize(u)[1]
    with pkg.DGSolver.for_problem(prob, nx, ny, p) as g:
        g.upload_state(0, u)
        got = g.semidiscretize(1, 0)
    assert abs(got - want) <= 20 * np.finfo(float).eps * want, (got, want)


@pytest.mark.parametrize("p,nx,ny", SIZES)
def test_density_zero(pkg, ora, p, nx, ny):
    prob, u, _ = _state(pkg, ora, nx, ny, p, [0.0, 50.0, 30.0, 0.0, 0.0, 0.0, 0.0, 1.0])
    with pkg.DGSolver.for_problem(prob, nx, ny, p) as g:
        g.upload_state(0, u)
        assert g.semidiscretize(1, 0) == 0.0
