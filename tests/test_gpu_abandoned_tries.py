"""What a try leaves behind that is abandoned in a stage formed inside the residual (GPU): an element whose average is
inadmissible keeps the values of the SSP-RK combination and the average of the stage before, as when its loops
1 and 3 are launches of their own; nothing of it is projected, limited or written."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _combination(R, s, u0, u, L, dt):
    """stage s of SSP-RK(2,2) and (3,3) as the device rounds it, and stages 2 to 4 of SSP-RK(5,4)"""
    if R < 5:
        ca, cb = {2: {2: (0.5, 0.5)}, 3: {2: (0.75, 0.25), 3: (1.0 / 3.0, 2.0 / 3.0)}}[R][s]
        return ca * u0 + cb * (u + dt * L)
    a, b, c = {2: (0.444370493651235, 0.555629506348765, 0.368410593050371),
               3: (0.620101851488403, 0.379898148511597, 0.251891774271694),
               4: (0.178079954393132, 0.821920045606868, 0.544974750228521)}[s]
    return (a * u0 + b * u) + (c * dt) * L


SIZES = {1: (15, 14), 2: (11, 10), 3: (7, 9)}


@pytest.mark.parametrize("R,p", [(2, 1), (2, 2), (3, 1), (3, 2), (3, 3), (5, 1), (5, 2), (5, 3)])
def test_abandoned_stage(pkg, R, p):
    nx, ny = SIZES[p]
    prob = pkg.problems.make("blast")
    u0 = prob.initial_state(nx, ny, p)
    w = 0.5 * pkg.problems.gll_nodes(p)[1]
    inner = (Ellipsis, slice(1, -1), slice(1, -1))
    found = 0
    for k in range(25, 50):  # from steps that pass to steps that fail at once: some fail in a later stage
        with pkg.DGSolver.for_problem(prob, nx, ny, p, R) as g, pkg.Batch() as b:
            g.set_log(64)
            g.upload_state(0, u0)
            g.solve_begin(1.0e6, 0.3 * 1.1 ** k, k % 2, 1, k % 3 == 0)
            b.add(g)
            b.advance(1)
            last = g.read_log()[0][-1]
            b.remove(g)
            s = last["stage"]
            if not last["neg_avg"] or s == 1 or s == 5:
                continue
            before, stage, avg = g.download_state(s - 1), g.download_state(s), g.download_avg()[inner]
            g.semidiscretize(1, s - 1)
            want = _combination(R, s, g.download_state(0)[inner], before[inner], g.download_ut(1), last["dt"])
            a = np.einsum("vklij,k,l->vij", want, w, w)
            prs = (prob.gamma - 1) * (a[7] - 0.5 * ((a[1] ** 2 + a[2] ** 2 + a[3] ** 2) / a[0] + (a[4] ** 2 + a[5] ** 2 + a[6] ** 2)))
            bad = (a[0] < -1e-9) | (prs < -1e-9)  # clearly inadmissible
            if not bad.any():
                continue
            found += 1
            np.testing.assert_array_equal(stage[inner][..., bad], want[..., bad], err_msg=str((k, s)))
            old = np.einsum("vklij,k,l->vij", before[inner], w, w)
            np.testing.assert_allclose(avg[:, bad], old[:, bad], rtol=1e-11, atol=1e-11, err_msg=str((k, s)))
    assert found > 0
