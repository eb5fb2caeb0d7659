"""Householder QR over many SMs (ttg_qr.cu): the cluster form (small blocks),
the grid form (large ones), real and complex, at sizes around the row deal
(rows below, at and above a multiple of the CTAs), thin, square and wide.

Householder QR is backward stable: ||A - Q R|| <= c r u ||A|| and ||Q^H Q - I||
<= c r u with u = 2^-53; c = 10 covers the length of the sums (numpy's own
check included).  R equals LAPACK's up to cond(A) times that."""
import numpy as np
import pytest
import scipy.linalg as sla

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def run(torch, ctx, A):
    import ttgpu
    n, m = A.shape
    z = np.iscomplexobj(A)
    a = torch.from_numpy(np.ravel(A, order="F").copy()).cuda()
    R = torch.zeros(min(n, m) * m, dtype=a.dtype, device="cuda")
    ttgpu.dqr(n, m, a, R, complex_=z)
    ctx.synchronize()
    k = min(n, m)
    return (a.cpu().numpy()[:n * k].reshape(n, k, order="F"),
            R.cpu().numpy().reshape(k, m, order="F"))


SIZES = [(1, 1), (2, 1), (1, 4), (7, 5), (8, 8), (16, 9), (33, 32), (5, 40), (129, 64), (64, 129),
         (255, 128), (1000, 24), (301, 200), (1217, 77), (1216, 300), (2049, 3), (5000, 86)]


@pytest.mark.parametrize("n,m", SIZES)
@pytest.mark.parametrize("cplx", [False, True])
def test_qr_sizes(torch_cuda, ctx, n, m, cplx):
    rng = np.random.default_rng(n * 7 + m)
    A = rng.standard_normal((n, m))
    if cplx:
        A = A + 1j * rng.standard_normal((n, m))
    Q, R = run(torch_cuda, ctx, A)
    r = min(n, m)
    assert np.linalg.norm(Q @ R - A) <= 10 * r * U * np.linalg.norm(A)
    assert np.linalg.norm(Q.conj().T @ Q - np.eye(r)) <= 10 * r * U * np.sqrt(r)
    assert (np.tril(R, -1) == 0).all()
    Rl = sla.qr(A, mode="economic")[1]
    cond = np.linalg.cond(A[:, :r])
    assert np.linalg.norm(R - Rl) <= 20 * r * U * cond * np.linalg.norm(A)


@pytest.mark.parametrize("n,m", [(40, 12), (3000, 60)])
def test_qr_degenerate_columns(torch_cuda, ctx, n, m):
    """Zero columns, repeated columns and a triangular start: the reflector of
    a column that is zero below its diagonal is the identity (its sign stays)."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, m))
    A[:, 3] = 0.0
    A[:, 5] = A[:, 1]
    A[:, 7] *= 1e-200
    A[:, 9] *= 1e120
    Q, R = run(torch_cuda, ctx, A)
    scale = np.linalg.norm(A, axis=0)
    err = np.linalg.norm(Q @ R - A, axis=0)
    assert (err <= 10 * m * U * scale).all()
    assert np.linalg.norm(Q.T @ Q - np.eye(m)) <= 10 * m * U * np.sqrt(m)
    T = np.zeros((n, m))
    T[:m] = np.triu(rng.standard_normal((m, m)))
    T[np.arange(m), np.arange(m)] = np.where(np.arange(m) % 2, 2.0, -3.0)
    Q, R = run(torch_cuda, ctx, T)
    assert np.array_equal(R, T[:m]) and np.array_equal(Q, np.eye(n, m))


def test_qr_nan_stays_nan(torch_cuda, ctx):
    A = np.ones((2000, 40)) + np.eye(2000, 40)
    A[1500, 7] = np.nan
    Q, R = run(torch_cuda, ctx, A)
    assert np.isnan(R[7:, 7:]).any() and np.isnan(Q[:, 7:]).any()
    assert np.isfinite(R[:, :7]).all()


def test_qr_is_reproducible(torch_cuda, ctx):
    rng = np.random.default_rng(2)
    A = rng.standard_normal((4100, 70))
    a = run(torch_cuda, ctx, A)
    for _ in range(3):
        b = run(torch_cuda, ctx, A)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("n,m", [(700, 7), (700, 8), (700, 9), (40, 15), (40, 17), (900, 33),
                                 (300, 129), (1500, 140), (2500, 40), (100, 150), (1344, 30)])
@pytest.mark.parametrize("cplx", [False, True])
def test_qr_panels(torch_cuda, ctx, n, m, cplx):
    """Q is formed a panel of 8 reflectors at a time: columns below, at and above
    a multiple of it, in the cluster and the grid form; columns above the grid
    form's limit of directly added parts.  Tolerance as above."""
    test_qr_sizes(torch_cuda, ctx, n, m, cplx)


@pytest.mark.parametrize("n", [64, 2000])
def test_qr_nan_leaves_earlier_columns(torch_cuda, ctx, n):
    """Column c of Q is the product of reflectors 0..c with e_c: a NaN in
    column 11, the middle of a panel, does not reach the columns before it."""
    A = np.random.default_rng(n).standard_normal((n, 20))
    A[n // 2, 11] = np.nan
    Q, R = run(torch_cuda, ctx, A)
    assert np.isfinite(Q[:, :11]).all() and np.isfinite(R[:, :11]).all()
    assert np.isnan(Q[:, 11:]).all()
