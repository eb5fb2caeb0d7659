"""The forms for problems that do not fit the chip's shared memory: the QR kernel of
one block on global memory and the panels of the SVD's factorisation (blocks above
25 MB), and the Arnoldi steps of separate products (above 1.2 million unknowns).

Bounds as for the forms on shared memory: ||A - Q R|| <= 10 r u ||A||, ||Q^H Q - I||
<= 10 r u sqrt(r), singular values to 10 q u of the largest, the solver's residual
below what it was asked for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("n,m,cplx", [(40000, 90, False), (21000, 83, True)])
def test_qr_on_global_memory(torch_cuda, ctx, n, m, cplx):
    import ttgpu
    dt = torch_cuda.complex128 if cplx else torch_cuda.float64
    g = torch_cuda.Generator(device="cuda")
    g.manual_seed(n)
    a0 = torch_cuda.randn(n * m, dtype=dt, device="cuda", generator=g)
    a, r = a0.clone(), torch_cuda.zeros(m * m, dtype=dt, device="cuda")
    ttgpu.dqr(n, m, a, r, complex_=cplx, ctx=ctx)
    ctx.synchronize()
    A, Q, R = (t.view(m, -1).T for t in (a0, a, r))
    norm = torch_cuda.linalg.norm
    assert float(norm(Q @ R - A)) <= 10 * m * U * float(norm(A))
    assert float(norm(Q.mH @ Q - torch_cuda.eye(m, dtype=dt, device="cuda"))) <= 10 * m * U * np.sqrt(m)
    assert float(norm(torch_cuda.tril(R, -1))) == 0.0


def test_svd_by_panels(torch_cuda, ctx):
    import ttgpu
    p, q = 38000, 97
    rng = np.random.default_rng(p)
    G = rng.standard_normal((p, q)) * 10.0 ** -np.linspace(0, 9, q)
    M = torch_cuda.from_numpy(np.ravel(G, order="F").copy()).cuda()
    u, s, vt = (torch_cuda.zeros(k, dtype=torch_cuda.float64, device="cuda") for k in (p * q, q, q * q))
    ttgpu.dgesvd(p, q, M, u, s, vt, ctx=ctx)
    ctx.synchronize()
    Um, S, V = u.view(q, p).T, s, vt.view(q, q).T
    A = M.view(q, p).T
    norm = torch_cuda.linalg.norm
    eye = torch_cuda.eye(q, dtype=torch_cuda.float64, device="cuda")
    assert float(norm((Um * S) @ V - A)) <= 20 * q * U * float(norm(A))
    assert float(norm(Um.T @ Um - eye)) <= 20 * q * U * np.sqrt(q)
    assert float(norm(V @ V.T - eye)) <= 20 * q * U * np.sqrt(q)
    ref = np.linalg.svd(G, compute_uv=False)
    assert abs(S.cpu().numpy() - ref).max() <= 10 * q * U * ref[0]


def test_gmres_beyond_a_resident_grid(ctx):
    """Middle core of 30 x 1500 x 30 = 1.35 million unknowns, which the right-hand
    side's ranks keep."""
    import ttgpu
    from ttgpu.operators import pack_tt_matrix, random_tt
    n = [30, 1500, 30]
    tri = [4.0 / 3 * np.eye(k) + 0.2 * (2 * np.eye(k) - np.eye(k, k=1) - np.eye(k, k=-1)) for k in n]
    eye = [np.eye(k) for k in n]
    first, mid, last = np.zeros((1, 30, 30, 2)), np.zeros((2, 1500, 1500, 2)), np.zeros((2, 30, 30, 1))
    first[0, :, :, 0], first[0, :, :, 1] = tri[0], eye[0]
    mid[0, :, :, 0], mid[1, :, :, 0], mid[1, :, :, 1] = eye[1], tri[1], eye[1]
    last[0, :, :, 0], last[1, :, :, 0] = eye[2], tri[2]
    n_, m_, ra, A = pack_tt_matrix([first, mid, last])
    rng = np.random.default_rng(9)
    core = lambda a, k, b: rng.standard_normal(a * k * b) / np.sqrt(k * b)
    ry = rx = [1, 30, 30, 1]
    y = np.concatenate([core(ry[k], n[k], ry[k + 1]) for k in range(3)])
    x0 = np.concatenate([core(rx[k], n[k], rx[k + 1]) for k in range(3)])
    cores, r = ttgpu.dtt_amen_solve(3, n_, m_, ry, ra, A, y, x0, rx, 1e-8, ctx=ctx)
    assert min(r[1], r[2]) >= 30

    def full(ranks, c):
        T, off = np.ones((1, 1)), 0
        for k in range(3):
            w = c[off:off + ranks[k] * n[k] * ranks[k + 1]].reshape(ranks[k], -1, order="F")
            off += w.size
            T = (T @ w).reshape(-1, ranks[k + 1], order="F")
        return T[:, 0].reshape(n, order="F")
    X, Y = full(r, cores), full(ry, y)
    AX = (np.tensordot(tri[0], X, (1, 0)) + np.tensordot(tri[1], X, (1, 1)).transpose(1, 0, 2) +
          np.tensordot(X, tri[2], (2, 1)))
    assert np.linalg.norm(AX - Y) <= 1e-7 * np.linalg.norm(Y)


def test_svd_of_a_square_block_by_panels(torch_cuda, ctx):
    """1900 x 1900: panels of 1024 rows and more on a grid, the last ones in one block
    of threads, in both factorisations."""
    import ttgpu
    q = 1900
    rng = np.random.default_rng(q)
    G = rng.standard_normal((q, q)) * 10.0 ** -np.linspace(0, 6, q)
    M = torch_cuda.from_numpy(np.ravel(G, order="F").copy()).cuda()
    u, s, vt = (torch_cuda.zeros(k, dtype=torch_cuda.float64, device="cuda") for k in (q * q, q, q * q))
    ttgpu.dgesvd(q, q, M, u, s, vt, ctx=ctx)
    ctx.synchronize()
    Um, S, V, A = u.view(q, q).T, s, vt.view(q, q).T, M.view(q, q).T
    norm = torch_cuda.linalg.norm
    eye = torch_cuda.eye(q, dtype=torch_cuda.float64, device="cuda")
    assert float(norm((Um * S) @ V - A)) <= 20 * q * U * float(norm(A))
    assert float(norm(Um.T @ Um - eye)) <= 20 * q * U * np.sqrt(q)
    assert float(norm(V @ V.T - eye)) <= 20 * q * U * np.sqrt(q)
    ref = np.linalg.svd(G, compute_uv=False)
    assert abs(S.cpu().numpy() - ref).max() <= 10 * q * U * ref[0]
