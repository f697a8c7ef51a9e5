"""OEDG damping of states whose wave speeds overflow (GPU): an infinite speed damps its element to the average, as in
the oracle."""
import numpy as np
import pytest

from conftest import rel_l1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("node", [dict(b=1.0e80, e=1.0e161), dict(b=0.0, e=1.0e200), dict(b=3.0e100, e=1.0e202)])
def test_overflowing_speed(pkg, ora, p, node):
    """the square of the squared speeds overflows from 1e154 on (a field of 1e80, a pressure of 1e200).  Tolerance:
    as the one-step parity of test_gpu_parity, per variable"""
    nx, ny = 9, 7
    prob = pkg.problems.make("ot2pi")
    u = prob.initial_state(nx, ny, p)
    u[:, 0, 1, 4, 3] = [1.0, 0.3, 0.2, 0.1, node["b"], 0.4, 0.1, node["e"]]
    u = np.asfortranarray(u)
    o = ora.OracleSolver(nx, ny, p, p, 3, *prob.domain, prob.gamma, prob.bc_kind, prob.bc_state)
    o.apply_bc(u)
    want = u.copy(order="F")
    avg = np.full((8, nx + 2, ny + 2), np.nan, order="F")
    ro = o.post_process(want, avg, 1, 0, 1.0e-3, 0, 0)
    with pkg.DGSolver.for_problem(prob, nx, ny, p) as g:
        g.upload_state(0, u)
        rg = g.post_process(0, 1, 0, 1.0e-3, 0, 0)
        got = g.download_state(0)
    assert rg["neg_avg"] == ro["neg_avg"] == 0 and rg["num_negcell"] == ro["num_negcell"]
    inner = (slice(None), slice(None), slice(None), slice(1, -1), slice(1, -1))
    a, b = got[inner], want[inner]
    far = np.ones(a.shape[3:], bool)
    far[3, 2] = False  # the element itself, on its own scale; the others on theirs
    assert rel_l1(a[:, :, :, far], b[:, :, :, far]).max() <= 1e-12
    assert rel_l1(a[:, :, :, 3, 2], b[:, :, :, 3, 2]).max() <= 1e-12
