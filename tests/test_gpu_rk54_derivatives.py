"""The time derivatives of an SSP-RK(5,4) run (GPU): after a step ut(2..5) hold L of the stage states, also where the
next stage is formed inside the residual (from 1024 nodes on, and in batches)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,nx,ny", [(1, 8, 7), (1, 23, 12), (2, 5, 6), (2, 13, 10), (3, 4, 5), (3, 11, 9)])
@pytest.mark.parametrize("batch", [False, True])
def test_derivatives_of_the_stages(pkg, p, nx, ny, batch):
    """bit for bit: the residual's arithmetic is the same in every kernel"""
    prob = pkg.problems.make("rotor")
    with pkg.DGSolver.for_problem(prob, nx, ny, p, 5) as g:
        g.upload_state(0, prob.initial_state(nx, ny, p))
        g.solve_begin(prob.final_T, 0.5 * prob.cfl, True, True, True)
        if batch:
            with pkg.Batch() as b:
                b.add(g)
                b.advance(2)
                b.remove(g)
        else:
            g.advance(2)
        assert g.status()["steps"] == 2
        got = [g.download_ut(s) for s in range(1, 6)]
        for s in range(1, 5):  # ut(s+1) = L(stage s), whose state and ghost ring are still in its slot
            g.semidiscretize(1, s)
            np.testing.assert_array_equal(got[s], g.download_ut(1), err_msg=str(s))
