"""Truncation SVD: the block sweeps (rows in registers, 1 to 8 a thread), the
pair sweeps behind them (more than 1024 rows in fewer than 16 columns), odd and
tiny widths, degenerate and extreme columns.

Bounds as in test_dgesvd_jacobi: singular values to 1e-14 max(p, q) ||M||, the
product to 1e-13 max(p, q) ||M|| (Jacobi's backward error, a few u per sweep and
column)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def svd(torch, ctx, M):
    import ttgpu
    p, q = M.shape
    r = min(p, q)
    m = torch.from_numpy(np.ravel(M, order="F").copy()).cuda()
    U = torch.zeros(p * r, dtype=torch.float64, device="cuda")
    s = torch.zeros(r, dtype=torch.float64, device="cuda")
    Vt = torch.zeros(r * q, dtype=torch.float64, device="cuda")
    ttgpu.dgesvd(p, q, m, U, s, Vt)
    ctx.synchronize()
    return (U.cpu().numpy().reshape(p, r, order="F"), s.cpu().numpy(),
            Vt.cpu().numpy().reshape(r, q, order="F"))


@pytest.mark.parametrize("p,q", [(2, 2), (5, 1), (6, 5), (17, 16), (40, 17), (128, 127), (129, 129),
                                 (300, 255), (260, 257), (600, 511), (520, 513), (1100, 15),
                                 (1024, 9), (1025, 4), (1300, 2), (900, 700)])
def test_sizes(torch_cuda, ctx, p, q):
    rng = np.random.default_rng(p + q)
    r = min(p, q)
    U0, V0 = np.linalg.qr(rng.standard_normal((p, r)))[0], np.linalg.qr(rng.standard_normal((q, r)))[0]
    s0 = np.logspace(0, -13, r)
    M = (U0 * s0) @ V0.T
    U, s, Vt = svd(torch_cuda, ctx, M)
    big = max(p, q)
    assert (np.diff(s) <= 0).all()
    assert abs(s - np.linalg.svd(M, compute_uv=False)).max() <= 1e-14 * big
    assert np.linalg.norm((U * s) @ Vt - M) <= 1e-13 * big
    assert np.linalg.norm(U.T @ U - np.eye(r)) <= 1e-14 * big * np.sqrt(r)
    assert np.linalg.norm(Vt @ Vt.T - np.eye(r)) <= 1e-14 * big * np.sqrt(r)


@pytest.mark.parametrize("p,q", [(90, 30), (400, 150)])
def test_small_singular_values_keep_their_relative_accuracy(torch_cuda, ctx, p, q):
    """Orthonormal columns scaled over 30 decades: the singular values are the
    scales, each to a relative q u times a small constant (one-sided Jacobi on
    the triangular factor of column-sorted data)."""
    rng = np.random.default_rng(q)
    Q = np.linalg.qr(rng.standard_normal((p, q)))[0]
    d = np.logspace(10, -20, q)
    s = svd(torch_cuda, ctx, Q[:, rng.permutation(q)] * rng.permutation(d))[1]
    assert (abs(s - d) <= 50 * q * 2.0 ** -53 * d).all()


def test_degenerate_columns(torch_cuda, ctx):
    rng = np.random.default_rng(1)
    M = rng.standard_normal((200, 61))
    M[:, 5] = 0.0
    M[:, 9] = M[:, 8]
    M[:, 20] = -2.0 * M[:, 8]
    for scale in (1.0, 1e100, 1e-120):
        U, s, Vt = svd(torch_cuda, ctx, M * scale)
        ref = np.linalg.svd(M, compute_uv=False)
        assert abs(s / scale - ref).max() <= 1e-14 * 200 * ref[0]
        assert np.linalg.norm((U * (s / scale)) @ Vt - M) <= 1e-13 * 200 * ref[0]
    U, s, Vt = svd(torch_cuda, ctx, np.zeros((70, 33)))
    assert (s == 0).all() and np.isfinite(U).all() and np.isfinite(Vt).all()


def test_nan_is_not_lost(torch_cuda, ctx):
    M = np.random.default_rng(3).standard_normal((64, 40))
    M[7, 11] = np.nan
    assert np.isnan(svd(torch_cuda, ctx, M)[1]).any()


def test_reproducible(torch_cuda, ctx):
    M = np.random.default_rng(4).standard_normal((500, 260))
    a = svd(torch_cuda, ctx, M)
    for _ in range(3):
        b = svd(torch_cuda, ctx, M)
        assert all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("q", [12, 63, 128, 200])
@pytest.mark.parametrize("kind", ["random", "clusters", "nearly equal", "orthogonal"])
def test_last_sweep_left_out(torch_cuda, ctx, q, kind):
    """The sweeps end without a look at the result where the last rotations were
    small enough: no pair of columns may be left above the level at which a
    sweep would have counted it, q 2^-52, whatever the spectrum (equal values
    turn by large angles at tiny cosines); the SVD's bounds as above."""
    rng = np.random.default_rng(q + len(kind))
    p = 2 * q
    U0, V0 = np.linalg.qr(rng.standard_normal((p, q)))[0], np.linalg.qr(rng.standard_normal((q, q)))[0]
    s0 = {"random": rng.random(q) + 0.01, "clusters": np.repeat(rng.random(q // 3 + 1) + 0.1, 3)[:q],
          "nearly equal": 1 + 1e-10 * rng.standard_normal(q), "orthogonal": np.ones(q)}[kind]
    M = (U0 * s0) @ V0.T
    U, s, Vt = svd(torch_cuda, ctx, M)
    # plus the rounding of U's own dot products
    assert abs(U.T @ U - np.eye(q)).max() <= q * 2.0 ** -52 + 2 * p * 2.0 ** -53
    assert abs(s - np.sort(s0)[::-1]).max() <= 1e-14 * p
    assert np.linalg.norm((U * s) @ Vt - M) <= 1e-13 * p
