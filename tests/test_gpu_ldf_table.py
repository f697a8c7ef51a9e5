"""The LDF projection as loop 1 applies it (between even and odd parts) against the dense nodal
operator, on elements that are not square: at every degree, with and without the fused limiter
(no OEDG and OEDG), on sizes that leave partial chunks and idle lanes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("oedg", [0, 1])
@pytest.mark.parametrize("p,nx,ny", [(1, 2, 2), (1, 37, 5), (2, 2, 3), (2, 19, 7), (3, 3, 2), (3, 13, 6)])
def test_projection_matches_dense_operator(pkg, p, nx, ny, oedg):
    """tolerance: 2n^2 products an output and 8 sums around them, which can double a value twice, relative
    to the operator's largest row sum and the largest field value"""
    n = p + 1
    rng = np.random.default_rng(100 * p + nx)
    u = np.zeros((8, n, n, nx + 2, ny + 2), order="F")
    u[0], u[7] = 1.0, 100.0  # far from every bound of the limiter
    u[4:6] = 2.0 + rng.uniform(-0.5, 0.5, u[4:6].shape)
    hx, hy = 0.7 / nx, 1.9 / ny
    w = 0.5 * pkg.problems.gll_nodes(p)[1]
    with pkg.DGSolver(nx, ny, p, 3, (0.0, 0.7, 0.0, 1.9)) as g:
        g.upload_state(0, u)
        g.post_process(0, oedg, 1, 0.0, 0, 0)
        got = g.download_state(0)
    A = pkg.ldf_operator(p, hx, hy)
    tol = EPS * (2 * n * n + 8) * 4 * np.abs(A).sum(1).max() * np.abs(u[4:6]).max()
    for i in range(1, nx + 1):
        for j in range(1, ny + 1):
            b = u[4:6, :, :, i, j]
            avg = np.einsum("vkl,k,l->v", b, w, w)
            x = (b - avg[:, None, None]).reshape(2, n * n, order="F").reshape(-1)
            want = (A @ x).reshape(2, n, n, order="C").transpose(0, 2, 1) + avg[:, None, None]
            np.testing.assert_allclose(got[4:6, :, :, i, j], want, rtol=0, atol=tol)
