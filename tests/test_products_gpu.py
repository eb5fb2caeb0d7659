"""FP64 and complex products of the local operators at the edges of their
tiles: sizes just below, at and above the 16 and 32 tiles and the warp blocks
(4 x 8, 8 x 16), K below, at and above one K step and in several cluster
chunks, and batches.

Bound: each entry is a sum of K products, so GPU and numpy each lie within
(K + 2) u |A| |B| of the exact value, u = 2^-53 (complex: 4 real products per
term, sqrt(2) per component); two chained products add their bounds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _t(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _f(a, *shape):
    return np.reshape(a, shape, order="F")


@pytest.mark.parametrize("rx1,n,rx2,ry1,ry2", [
    (1, 1, 1, 1, 1), (4, 2, 3, 9, 8), (15, 1, 16, 17, 31), (16, 2, 17, 16, 32), (33, 1, 4, 5, 33),
    (7, 5, 64, 8, 65), (10, 1, 200, 96, 16), (24, 43, 31, 24, 47), (8, 3, 1500, 8, 8),
    (100, 40, 13, 90, 7), (17, 64, 80, 19, 80),
])
def test_real_products_at_tile_edges(torch_cuda, ctx, rx1, n, rx2, ry1, ry2):
    """phi2_right: (rx1 n x rx2)(rx2 x ry2), then (rx1 x n ry2)(n ry2 x ry1);
    phi2_left runs the same sizes through the other operand orders."""
    import ttgpu
    rng = np.random.default_rng(rx1 * 1000 + rx2 + ry1)
    x, y = rng.standard_normal(rx1 * n * rx2), rng.standard_normal(ry1 * n * ry2)
    p2, p1 = rng.standard_normal(rx2 * ry2), rng.standard_normal(ry1 * rx1)
    X, Y = _f(x, rx1 * n, rx2), _f(y, ry1, n * ry2)
    P2, P1 = _f(p2, rx2, ry2), _f(p1, ry1, rx1)
    out = torch_cuda.zeros(rx1 * ry1, dtype=torch_cuda.float64, device="cuda")
    ttgpu.phi2_right(rx1, rx2, ry1, n, ry2, _t(torch_cuda, p2), _t(torch_cuda, x),
                     _t(torch_cuda, y), out)
    ctx.synchronize()
    ref = _f(np.ravel(X @ P2, order="F"), rx1, n * ry2) @ Y.T
    bound = _f(np.ravel(abs(X) @ abs(P2), order="F"), rx1, n * ry2) @ abs(Y).T
    err = abs(_f(out.cpu().numpy(), rx1, ry1) - ref)
    assert (err <= 2 * (rx2 + n * ry2 + 4) * U * bound).all()
    out = torch_cuda.zeros(ry2 * rx2, dtype=torch_cuda.float64, device="cuda")
    ttgpu.phi2_left(rx1, rx2, ry1, n, ry2, _t(torch_cuda, p1), _t(torch_cuda, x),
                    _t(torch_cuda, y), out)
    ctx.synchronize()
    ref = _f(np.ravel(P1.T @ Y, order="F"), rx1 * n, ry2).T @ X
    bound = _f(np.ravel(abs(P1).T @ abs(Y), order="F"), rx1 * n, ry2).T @ abs(X)
    err = abs(_f(out.cpu().numpy(), ry2, rx2) - ref)
    assert (err <= 2 * (ry1 + rx1 * n + 4) * U * bound).all()


@pytest.mark.parametrize("r1,n,r2,ra,nvec", [
    (1, 2, 1, 1, 1), (3, 5, 4, 2, 3), (8, 32, 8, 6, 1), (8, 32, 8, 6, 4), (9, 8, 7, 3, 2),
    (16, 17, 17, 2, 1), (5, 16, 33, 4, 2), (4, 3, 2, 5, 9),
])
def test_complex_local_products_at_tile_edges(torch_cuda, ctx, r1, n, r2, ra, nvec):
    import ttgpu
    rng = np.random.default_rng(r1 * 100 + n)
    z = lambda k: rng.standard_normal(k) + 1j * rng.standard_normal(k)
    p1, A, p2 = z(r1 * r1 * ra), z(ra * n * n * ra), z(r2 * ra * r2)
    x = z(r1 * n * r2 * nvec)
    out = torch_cuda.zeros(x.size, dtype=torch_cuda.complex128, device="cuda")
    outt = torch_cuda.zeros(x.size, dtype=torch_cuda.complex128, device="cuda")
    args = [_t(torch_cuda, v) for v in (p1, A, p2, x)]
    ttgpu.zbfun3(r1, n, r2, r1, n, r2, ra, ra, *args, out, nvec)
    ttgpu.zbfun3(r1, n, r2, r1, n, r2, ra, ra, *args, outt, nvec, transp=True)
    ctx.synchronize()
    P1, AA, P2 = _f(p1, r1, r1, ra), _f(A, ra, n, n, ra), _f(p2, r2, ra, r2)
    X = _f(x, r1, n, r2, nvec)

    def fwd(P1, AA, P2, X):
        t = np.einsum("eac,bjev->bjacv", P2, X)
        t = np.einsum("dija,bjacv->bdicv", AA, t)
        return np.einsum("zbd,bdicv->zicv", P1, t)

    def adj(P1, AA, P2, X):
        t = np.einsum("zbd,zicv->bdicv", P1.conj(), X)
        t = np.einsum("dija,bdicv->bjacv", AA.conj(), t)
        return np.einsum("eac,bjacv->bjev", P2.conj(), t)

    K = r2 + n * ra + r1 * ra
    for got, f in ((out, fwd), (outt, adj)):
        bound = f(abs(P1), abs(AA), abs(P2), abs(X))
        err = abs(_f(got.cpu().numpy(), *bound.shape) - f(P1, AA, P2, X))
        assert (err <= 2 * 4 * np.sqrt(2) * (K + 6) * U * bound).all()
