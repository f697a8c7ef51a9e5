"""Residuals of meshes with more rows than a grid has in y (65,535): a state that repeats every eight rows has the residual
of the eight-row mesh in each of them, bit for bit (both meshes have hy = 1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,ny", [(1, 131072 + 8), (2, 65536 + 8), (3, 65536 + 8)])
def test_residual_of_a_tall_mesh(pkg, p, ny):
    nx, few, n = 2, 8, p + 1
    rng = np.random.default_rng(p)
    w = rng.uniform(0.5, 1.5, (8, n, n, nx, few))
    w[7] += 20.0
    small = np.full((8, n, n, nx + 2, few + 2), np.nan, order="F")
    small[:, :, :, 1:-1, 1:-1] = w
    tall = np.full((8, n, n, nx + 2, ny + 2), np.nan, order="F")
    tall[:, :, :, 1:-1, 1:-1] = np.tile(w, (1, 1, 1, 1, ny // few))
    out = []
    for u, rows in ((small, few), (tall, ny)):
        with pkg.DGSolver(nx, rows, p, 1, (0.0, float(nx), 0.0, float(rows))) as g:
            g.upload_state(0, u)
            g.apply_bc(0)
            out.append((g.semidiscretize(1, 0), g.download_ut(1)))
    (dt_small, ut_small), (dt_tall, ut_tall) = out
    assert dt_small == dt_tall
    for j in range(0, ny, few):
        if not np.array_equal(ut_tall[:, :, :, :, j:j + few], ut_small):
            raise AssertionError(f"rows {j} to {j + few - 1}")
