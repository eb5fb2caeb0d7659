"""The fused Arnoldi step behind the AMEn solvers, over its forms: one CTA (up
to 128 unknowns a local problem), a grid, several rows per thread; a Krylov
space that ends early.  The solves' FP64 residuals, against the dense operator,
meet the tolerance the solver was given, as before."""
import numpy as np
import pytest

from oracle.ksl import tt_full
from test_oracle import tt_matrix_full
from ttgpu.operators import amen_operator, laplace_tt, pack_tt_matrix, random_tt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,r", [(2, 9, 1), (3, 12, 2), (4, 7, 3), (2, 60, 4)])
@pytest.mark.parametrize("method", ["plain", "split"])
def test_solves(ctx, d, n, r, method):
    import ttgpu
    tol = 1e-8
    nn, mm, ra, crA = amen_operator(d=d, n=n)
    _, ry, y = random_tt(d, n, r, seed=11)
    _, rx, x0 = random_tt(d, n, 2, seed=12)
    c, rx1 = ttgpu.dtt_amen_solve(d, nn, mm, ry, ra, crA, y, x0, rx, tol, nswp=40, method=method, ctx=ctx)
    A = tt_matrix_full(d, nn, ra, crA)
    yf = tt_full(d, nn, ry, y)
    assert np.linalg.norm(A @ tt_full(d, nn, rx1, c) - yf) <= 2 * tol * np.linalg.norm(yf)


def test_krylov_space_ends_early(ctx):
    """A right-hand side that is an eigenvector: one Arnoldi step spans the
    space, the second vector is rounding noise."""
    import ttgpu
    d, n = 3, 14
    nn, mm, ra, crA = pack_tt_matrix(laplace_tt(d, n))
    v = np.sin(np.pi * np.arange(1, n + 1) / (n + 1))
    lam = d * (2 - 2 * np.cos(np.pi / (n + 1)))
    y = np.concatenate([v] * d)
    ry = [1] * (d + 1)
    _, rx, x0 = random_tt(d, n, 1, seed=3)
    c, rx1 = ttgpu.dtt_amen_solve(d, nn, mm, ry, ra, crA, y, x0, rx, 1e-10, ctx=ctx)
    yf = tt_full(d, nn, ry, y)
    xf = tt_full(d, nn, rx1, c)
    assert np.linalg.norm(xf - yf / lam) <= 1e-9 * np.linalg.norm(yf / lam)


def test_reproducible(ctx):
    import ttgpu
    d, n = 4, 16
    nn, mm, ra, crA = amen_operator(d=d, n=n)
    _, ry, y = random_tt(d, n, 3, seed=1)
    _, rx, x0 = random_tt(d, n, 2, seed=2)
    a = ttgpu.dtt_amen_solve(d, nn, mm, ry, ra, crA, y, x0, rx, 1e-8, ctx=ctx)
    b = ttgpu.dtt_amen_solve(d, nn, mm, ry, ra, crA, y, x0, rx, 1e-8, ctx=ctx)
    assert a[1] == b[1] and np.array_equal(a[0], b[0])
