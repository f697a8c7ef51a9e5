"""The residual of states that hold an inadmissible node (GPU): what has no value is NaN (or infinite) and nothing else,
as in the oracle, also at faces where the densities of both sides are negative and their ratio and product are
not; the rest of the mesh and dt_lim are those of the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
INF, NAN = np.inf, np.nan
OK = [1.0, 0.3, 0.2, 0.1, 0.5, 0.4, 0.1, 3.0]


def _bad(**kw):
    names = ["rho", "mx", "my", "mz", "bx", "by", "bz", "e"]
    return np.array([kw.get(n, v) for n, v in zip(names, OK)])


NODES = {"negative density": _bad(rho=-1.0), "density zero": _bad(rho=0.0), "negative pressure": _bad(e=-5.0),
         "NaN density": _bad(rho=NAN), "NaN field": _bad(bx=NAN), "NaN energy": _bad(e=NAN),
         "infinite density": _bad(rho=INF), "infinite momentum": _bad(mx=INF), "infinite field": _bad(bx=INF)}


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("node", list(NODES))
@pytest.mark.parametrize("where", ["corner", "both sides of a face", "inside", "a line"])
def test_inadmissible_node(pkg, ora, p, node, where):
    """tolerance: as test_gpu_residual_terms, of smooth states at this mesh"""
    nx, ny = 9, 7
    prob = pkg.problems.make("ot2pi")
    u = prob.initial_state(nx, ny, p)
    bad = NODES[node]
    if where == "inside":
        u[:, 1, 1, 4, 3] = bad
    elif where == "a line":
        u[:, :, 0, 4, 3] = bad[:, None] * np.linspace(1.0, 1.2, p + 1)
    else:
        u[:, p, 0, 4, 3] = bad
        if where == "both sides of a face":
            u[:, 0, 0, 5, 3] = 0.9 * bad
    u = np.asfortranarray(u)
    o = ora.OracleSolver(nx, ny, p, p, 3, *prob.domain, prob.gamma, prob.bc_kind, prob.bc_state)
    o.apply_bc(u)
    want, dt_want = o.semidiscretize(u)
    with pkg.DGSolver.for_problem(prob, nx, ny, p) as g:
        g.upload_state(0, u)
        dt = g.semidiscretize(1, 0)
        got = g.download_ut(1)
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(want))
    ok = np.isfinite(want)
    assert np.abs(got[ok] - want[ok]).max() <= 200 * EPS * (p + 1) ** 2 * np.abs(want[ok]).max()
    assert abs(dt - dt_want) <= 20 * EPS * abs(dt_want)
