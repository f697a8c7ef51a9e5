"""Stages formed inside the residual (GPU): stages after the first take their combination, ghost ring and
loop 1 from the previous stage's residual, in a batch always, alone from 1024 nodes on.  Below that an
instance keeps a launch per procedure, so a small run alone and as a batch member takes the two routes with
the same arithmetic: the states, the averages (ghost elements included), times and limiter counts are equal
bit for bit, over every boundary kind, ragged and smallest meshes, and combinations of the limiters."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = {1: [(15, 14), (2, 3)], 2: [(13, 6), (2, 2)], 3: [(7, 5), (3, 2)]}
FLAGS = [(1, 1, 0), (0, 1, 1), (1, 0, 1), (0, 0, 0)]  # OEDG, LDF, entropy offset


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("R", [2, 3, 5])
@pytest.mark.parametrize("name", ["ot2pi", "blast", "rotor", "cloud_shock", "jet", "xextrap"])
def test_folded_stages_equal_separate_launches(pkg, p, R, name):
    prob = pkg.problems.make("blast" if name == "xextrap" else name)
    if name == "xextrap":
        prob = dataclasses.replace(prob, bc_kind=pkg.capi.BC_XEXTRAP_YPER)
    sizes = [(10, 6)] if name == "jet" else SIZES[p]
    runs = [(nx, ny, fl) for nx, ny in sizes for fl in FLAGS]

    def make(nx, ny, fl):
        g = pkg.DGSolver.for_problem(prob, nx, ny, p, R)
        g.upload_state(0, prob.initial_state(nx, ny, p))
        g.solve_begin(prob.final_T, 0.5 * prob.cfl, *fl)
        return g

    alone = [make(*r) for r in runs]
    members = [make(*r) for r in runs]
    with pkg.Batch() as b:
        for m in members:
            b.add(m)
        b.advance(4)
        together = [b.status(m) for m in members]
        for m in members:
            b.remove(m)
    for g, m, st, (nx, ny, fl) in zip(alone, members, together, runs):
        assert nx * ny * (p + 1) ** 2 < 1024
        for _ in range(4):
            sg = g.advance(1) if g.status()["steps"] < st["steps"] else sg
        assert st["steps"] > 0, (nx, ny, fl)
        for k in ("t", "dt", "dt_lim", "tot_ent", "steps", "num_negcell_total"):
            np.testing.assert_equal(st[k], sg[k], err_msg=str((k, nx, ny, fl)))
        np.testing.assert_array_equal(m.download_state(0), g.download_state(0), err_msg=str((nx, ny, fl)))
        a, r = m.download_avg(), g.download_avg()
        np.testing.assert_array_equal(a[:, 1:-1, :], r[:, 1:-1, :])
        np.testing.assert_array_equal(a[:, :, 1:-1], r[:, :, 1:-1])
        g.close()
        m.close()
