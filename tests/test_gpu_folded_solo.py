"""Runs of 1024 nodes and more alone (GPU): their stages after the first are formed inside the residual, by other kernels
than a batch's.  State, averages, derivatives, times and limiter counts equal the batch member's bit for bit, which
test_gpu_folded_stages compares with separate launches; and the try's graph has the kernels that leaves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = {1: (30, 13), 2: (20, 7), 3: (10, 8)}
KERNELS = {2: 12, 3: 14, 5: 18}  # begin, re-try, dt; loop 1; two a stage; sum, indicators, limiter; end


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("R", [2, 3, 5])
@pytest.mark.parametrize("name", ["ot2pi", "blast", "rotor", "cloud_shock", "jet"])
@pytest.mark.parametrize("flags", [(1, 1, 0), (1, 1, 1), (0, 0, 1)])
def test_solo_equals_batch_member(pkg, p, R, name, flags):
    prob = pkg.problems.make(name)
    nx, ny = SIZES[p]
    assert nx * ny * (p + 1) ** 2 >= 1024
    runs = []
    for batch in (False, True):
        with pkg.DGSolver.for_problem(prob, nx, ny, p, R) as g:
            g.upload_state(0, prob.initial_state(nx, ny, p))
            g.solve_begin(prob.final_T, 0.5 * prob.cfl, *flags)
            if batch:
                with pkg.Batch() as b:
                    b.add(g)
                    for _ in range(40):  # tries; re-tries among them
                        if b.status(g)["steps"] < 3:
                            b.advance(1)
                    b.remove(g)
            else:
                g.advance(3)
                assert g.step_graph_kernels() == KERNELS[R] - (0 if flags[0] else 2)
            inner = (Ellipsis, slice(1, -1), slice(1, -1))
            runs.append((g.status(), [g.download_state(s)[inner] for s in range(R + 1)], g.download_avg()[inner],
                         [g.download_ut(s) for s in range(1, R + 1)]))
    (sa, ua, aa, ka), (sb, ub, ab, kb) = runs
    for key in ("t", "dt", "dt_lim", "tot_ent", "steps", "retries", "num_negcell_total", "flags"):
        np.testing.assert_equal(sa[key], sb[key], err_msg=key)
    for q in range(R + 1):
        np.testing.assert_array_equal(ua[q], ub[q], err_msg=f"slot {q}")
    np.testing.assert_array_equal(aa, ab)
    for q in range(R):
        np.testing.assert_array_equal(ka[q], kb[q], err_msg=f"ut {q + 1}")
