"""The chosen local eigensolver's CG step in one kernel (ttg_chosen.cu): every
split of rows and columns over its CTAs, and the five kernels behind it.

The local operator P (x) I (x) I + I (x) B (x) I + I (x) I (x) Q has the sums of
the three spectra for eigenvalues.  A Ritz value lies within its residual's norm
of an eigenvalue, and the solver stops at tol times the largest |theta|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def problem(r1, r2, seed):
    """phi1, A, phi2 and the spectrum of a local problem of size r1 x 2 x r2."""
    rng = np.random.default_rng(seed)

    def sym(n, low):
        w = np.concatenate([low, rng.uniform(2.0, 4.0, n - len(low))])
        V = np.linalg.qr(rng.standard_normal((n, n)))[0]
        return (V * w) @ V.T, w
    P, wp = sym(r1, [-3.0, -1.9])
    Q, wq = sym(r2, [-2.0, -1.5])
    B = np.array([[0.3, 0.4], [0.4, -0.3]])                     # -0.5, 0.5
    phi1 = np.zeros((r1, r1, 2), order="F")                     # [c, b, a]
    phi1[:, :, 0], phi1[:, :, 1] = np.eye(r1), P
    phi2 = np.zeros((r2, 2, r2), order="F")                     # [b, a, c]
    phi2[:, 0], phi2[:, 1] = np.eye(r2), Q
    A = np.zeros((2, 2, 2, 2), order="F")                       # [a1, i, j, a2]
    A[0, :, :, 0], A[1, :, :, 0], A[0, :, :, 1] = B, np.eye(2), np.eye(2)
    w = (wp[:, None, None] + np.array([-0.5, 0.5])[:, None] + wq).ravel()
    return phi1, A, phi2, np.sort(w)


@pytest.mark.parametrize("r1,r2,B", [(16, 16, 1), (20, 21, 5), (49, 50, 4), (64, 64, 5),
                                     (72, 80, 8), (100, 96, 3), (104, 100, 5), (144, 150, 4),
                                     (208, 200, 2), (40, 40, 9)])
def test_local_problem(ctx, torch_cuda, r1, r2, B):
    import ttgpu
    torch = torch_cuda
    phi1, A, phi2, w = problem(r1, r2, r1 + r2)
    dev = lambda a: torch.from_numpy(np.ravel(a, order="F").copy()).cuda()
    rng = np.random.default_rng(B)
    X0 = np.linalg.qr(rng.standard_normal((2 * r1 * r2, B)))[0]
    tol = 1e-9
    lam, res, nmv = ttgpu.local_eig(r1, 2, r2, 2, 2, dev(phi1), dev(A), dev(phi2), dev(X0), B, tol,
                                    method="split", ctx=ctx)
    assert ctx.capped() == 0
    assert abs(np.sort(lam) - w[:B]).max() <= tol * abs(lam).max()
