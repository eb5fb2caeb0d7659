"""Split FP64 products (ttg_oz.cu) on operands whose parts differ in scale.

A product's two factors hold an operator's parts in opposite scales where its K
runs over the operator rank (1 and 1/h^2 for a Laplacian), and a row then spans
more than the 55 bits a split row has.  Every product must be as accurate as the
FP64 kernels whatever the scale: within 4e-15 of numpy in the norm (the FP64
kernels' own errors here are below 2e-15), for each operator rank block of the
result by itself, since the next product weighs the blocks by the other scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 4e-15
SCALES = [1.0, 1e2, 1e4, 1e8, 1e12]


def _t(torch, a):
    return torch.from_numpy(np.ravel(a, order="F").copy()).cuda()


def _close(got, ref, what):
    err, size = np.linalg.norm(got - ref), np.linalg.norm(ref)
    assert err <= TOL * size, f"{what}: {err / size:.2e}"


def _orthonormal(rng, rows, cols, cplx):
    A = rng.standard_normal((rows, cols))
    if cplx:
        A = A + 1j * rng.standard_normal((rows, cols))
    return np.linalg.qr(A)[0]


def laplace_interfaces(n, s, r, cplx=False, sites=2):
    """Core of s * sum_k I x .. x L_k x .. x I and its interfaces at a middle site:
    Phi1[c1, b1, a1] and Phi2[b2, a2, c2] from random orthonormal cores."""
    from ttgpu.operators import laplace_tt
    rng = np.random.default_rng(n + int(np.log2(s)))
    cores = laplace_tt(2 * sites + 1, n, s)
    dt = complex if cplx else float
    P1 = np.ones((1, 1, 1), dtype=dt)
    for C in cores[:sites]:
        k = min(P1.shape[0] * n, r)
        Q = _orthonormal(rng, P1.shape[0] * n, k, cplx).reshape(P1.shape[0], n, k)
        T = np.einsum("cba,bjx->cajx", P1, Q)
        T = np.einsum("cajx,aije->cixe", T, C)
        P1 = np.einsum("cixe,ciy->yxe", T, Q.conj())
    P2 = np.ones((1, 1, 1), dtype=dt)
    for C in cores[:sites:-1]:
        k = min(P2.shape[0] * n, r)
        Q = _orthonormal(rng, P2.shape[0] * n, k, cplx).reshape(P2.shape[0], n, k)
        T = np.einsum("eac,ejx->acjx", P2, Q)
        T = np.einsum("acjx,dija->cixd", T, C)
        P2 = np.einsum("cixd,ciy->xdy", T, Q.conj())
    return cores[sites], P1, P2


def apply(P1, C, P2, X):
    T = np.einsum("bjev,eac->bjacv", X, P2, optimize=True)
    T = np.einsum("dija,bjacv->bdicv", C, T, optimize=True)
    return np.einsum("cbd,bdiev->ciev", P1, T, optimize=True)


def adjoint(P1, C, P2, X):
    T = np.einsum("zbd,zicv->bdicv", P1.conj(), X, optimize=True)
    T = np.einsum("dija,bdicv->bjacv", C.conj(), T, optimize=True)
    return np.einsum("eac,bjacv->bjev", P2.conj(), T, optimize=True)


@pytest.mark.parametrize("s", SCALES)
@pytest.mark.parametrize("n,r", [(24, 60), (33, 41)])
def test_laplace_operator(torch_cuda, ctx, n, r, s):
    import ttgpu
    C, P1, P2 = laplace_interfaces(n, s, r)
    nv = 3
    x = np.random.default_rng(1).standard_normal((r, n, r, nv)) * np.array([1.0, 1e-9, 1e5])
    y = torch_cuda.zeros(x.size, dtype=torch_cuda.float64, device="cuda")
    l0 = ttgpu.launch_count()
    ttgpu.dbfun3(r, n, r, r, n, r, 2, 2, _t(torch_cuda, P1), _t(torch_cuda, C), _t(torch_cuda, P2),
                 _t(torch_cuda, x), y, nvec=nv)
    assert ttgpu.launch_count() - l0 > 3, "no split product was taken"
    ctx.synchronize()
    got, ref = y.cpu().numpy().reshape(x.shape, order="F"), apply(P1, C, P2, x)
    for v in range(nv):
        _close(got[..., v], ref[..., v], f"vector {v}")


@pytest.mark.parametrize("s", SCALES)
def test_laplace_complex_operator_and_adjoint(torch_cuda, ctx, s):
    import ttgpu
    n, r, nv = 24, 48, 2
    C, P1, P2 = laplace_interfaces(n, s, r, cplx=True)
    rng = np.random.default_rng(2)
    x = rng.standard_normal((r, n, r, nv)) + 1j * rng.standard_normal((r, n, r, nv))
    t = [_t(torch_cuda, v) for v in (P1, C.astype(complex), P2, x)]
    y = torch_cuda.zeros(x.size, dtype=torch_cuda.complex128, device="cuda")
    for f, kw in ((apply, {}), (adjoint, {"transp": True})):
        l0 = ttgpu.launch_count()
        ttgpu.zbfun3(r, n, r, r, n, r, 2, 2, *t, y, nv, **kw)
        assert ttgpu.launch_count() - l0 > 3
        ctx.synchronize()
        got, ref = y.cpu().numpy().reshape(x.shape, order="F"), f(P1, C, P2, x)
        for v in range(nv):
            _close(got[..., v], ref[..., v], f.__name__)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("s", SCALES)
def test_laplace_interface_updates(torch_cuda, ctx, s, cplx):
    import ttgpu
    n, r = 24, 60
    C, P1, P2 = laplace_interfaces(n, s, r, cplx)
    rng = np.random.default_rng(3)
    x = _orthonormal(rng, r * n, r, cplx).reshape(r, n, r, order="F")
    y = _orthonormal(rng, r * n, r, cplx).reshape(r, n, r, order="F")
    t = lambda v: _t(torch_cuda, v.astype(complex if cplx else float))
    dt = torch_cuda.complex128 if cplx else torch_cuda.float64
    L = torch_cuda.zeros(r * r * 2, dtype=dt, device="cuda")
    R = torch_cuda.zeros(r * r * 2, dtype=dt, device="cuda")
    l0 = ttgpu.launch_count()
    ttgpu.phi_left(r, n, r, r, n, r, 2, 2, t(P1), t(C), t(x), t(y), L, complex_=cplx)
    ttgpu.phi_right(r, n, r, r, n, r, 2, 2, t(P2), t(C), t(x), t(y), R, complex_=cplx)
    assert ttgpu.launch_count() - l0 > 6
    ctx.synchronize()
    T = np.einsum("cba,ciy->baiy", P1, y.conj(), optimize=True)
    T = np.einsum("aije,baiy->bjey", C, T, optimize=True)
    ref = np.einsum("bjey,bjx->yxe", T, x, optimize=True)
    got = L.cpu().numpy().reshape(r, r, 2, order="F")
    for a in range(2):
        _close(got[:, :, a], ref[:, :, a], f"left block {a}")
    T = np.einsum("bje,eac->bjac", x, P2, optimize=True)
    T = np.einsum("dija,bjac->bdic", C, T, optimize=True)
    ref = np.einsum("bdic,yic->bdy", T, y.conj(), optimize=True)
    got = R.cpu().numpy().reshape(r, 2, r, order="F")
    for a in range(2):
        _close(got[:, a], ref[:, a], f"right block {a}")


@pytest.mark.parametrize("M,N,K", [(640, 96, 257), (130, 400, 300), (64, 200, 4097)])
@pytest.mark.parametrize("decades", [4, 13])
def test_opposite_scales_along_k(torch_cuda, ctx, M, N, K, decades):
    """X S times S^-1 P: every k gives the same share, the rows span `decades`."""
    import ttgpu
    rng = np.random.default_rng(M + K)
    S = 10.0 ** (-decades * rng.permutation(np.linspace(0, 1, K)))
    X, P = rng.standard_normal((M, K)) * S, rng.standard_normal((K, N)) / S[:, None]
    one = torch_cuda.ones(1, dtype=torch_cuda.float64, device="cuda")
    y = torch_cuda.zeros(M * N, dtype=torch_cuda.float64, device="cuda")
    l0 = ttgpu.launch_count()
    ttgpu.dbfun3(1, 1, K, 1, 1, N, 1, 1, one, one, _t(torch_cuda, P), _t(torch_cuda, X.T), y, nvec=M)
    assert ttgpu.launch_count() - l0 > 3
    ctx.synchronize()
    _close(y.cpu().numpy().reshape(M, N), X @ P, "product")


@pytest.mark.parametrize("what", ["phi1", "core", "phi2", "x"])
def test_zero_blocks(torch_cuda, ctx, what):
    """A zero operator rank block, or a zero vector beside others, at scale 1e8."""
    import ttgpu
    n, r, nv = 24, 60, 2
    C, P1, P2 = laplace_interfaces(n, 1e8, r)
    x = np.random.default_rng(4).standard_normal((r, n, r, nv))
    if what == "phi1":
        P1[:, :, 0] = 0
    elif what == "core":
        C[1, :, :, 0] = 0
    elif what == "phi2":
        P2[:, 1] = 0
    else:
        x[..., 0] = 0
    y = torch_cuda.zeros(x.size, dtype=torch_cuda.float64, device="cuda")
    ttgpu.dbfun3(r, n, r, r, n, r, 2, 2, _t(torch_cuda, P1), _t(torch_cuda, C), _t(torch_cuda, P2),
                 _t(torch_cuda, x), y, nvec=nv)
    ctx.synchronize()
    got, ref = y.cpu().numpy().reshape(x.shape, order="F"), apply(P1, C, P2, x)
    for v in range(nv):
        _close(got[..., v], ref[..., v], f"{what}, vector {v}")


@pytest.mark.parametrize("r1,r2,nvec", [(64, 64, 5), (101, 90, 3)])
def test_chain_with_a_large_coupling(torch_cuda, ctx, r1, r2, nvec):
    """n = 2: the core contracted into Phi2 first; one operator rank block 1e10
    times the others, its partner in the other interface 1e-10 times."""
    import ttgpu
    rng = np.random.default_rng(r1)
    n, ra = 2, 5
    w = np.array([1.0, 1e10, 1.0, 1e-10, 1e3])
    P1 = rng.standard_normal((r1, r1, ra)) * w
    C = rng.standard_normal((ra, n, n, ra)) / w[:, None, None, None] / w[::-1]
    P2 = rng.standard_normal((r2, ra, r2)) * w[::-1, None]
    x = rng.standard_normal((r1, n, r2, nvec))
    y = torch_cuda.zeros(x.size, dtype=torch_cuda.float64, device="cuda")
    l0 = ttgpu.launch_count()
    ttgpu.dbfun3(r1, n, r2, r1, n, r2, ra, ra, _t(torch_cuda, P1), _t(torch_cuda, C),
                 _t(torch_cuda, P2), _t(torch_cuda, x), y, nvec=nvec)
    assert ttgpu.launch_count() - l0 > 3
    ctx.synchronize()
    _close(y.cpu().numpy().reshape(x.shape, order="F"), apply(P1, C, P2, x), "product")


@pytest.mark.parametrize("rows", ["one", "many"])
def test_large_elements_that_do_not_meet(torch_cuda, ctx, rows):
    """Both factors' largest elements stand where the other one's are small: in the
    rows of one vector, or of one operator rank block of many rows; the product has
    the FP64 kernels' accuracy in each block all the same."""
    import ttgpu
    rng = np.random.default_rng(11)
    r, n, ra, nv = 40, 24, 2, 4
    P1, P2 = rng.standard_normal((r, r, ra)), rng.standard_normal((r, ra, r))
    C = rng.standard_normal((ra, n, n, ra))
    x = rng.standard_normal((r, n, r, nv))
    if rows == "one":
        x[:, :, ::2, 1] *= 1e-9
        P2[::2] *= 1e9
    else:
        C[1, :, ::3] *= 1e11
        x[:, ::3] *= 1e-11
    y = torch_cuda.zeros(x.size, dtype=torch_cuda.float64, device="cuda")
    ttgpu.dbfun3(r, n, r, r, n, r, ra, ra, _t(torch_cuda, P1), _t(torch_cuda, C), _t(torch_cuda, P2),
                 _t(torch_cuda, x), y, nvec=nv)
    ctx.synchronize()
    got, ref = y.cpu().numpy().reshape(x.shape, order="F"), apply(P1, C, P2, x)
    for v in range(nv):
        _close(got[..., v], ref[..., v], f"vector {v}")


@pytest.mark.parametrize("s", [1.0, 1e4, 1e8])
def test_linear_solve_does_not_depend_on_the_scale(ctx, s):
    """dtt_amen_solve of s A x = s y: the solution of s = 1 to the accuracy asked for
    (ranks may differ by rounding at the truncation, with the FP64 kernels alone too)."""
    import ttgpu
    from ttgpu.operators import laplace_tt, pack_tt_matrix, random_tt
    d, n, tol = 3, 24, 1e-8
    _, ry, y = random_tt(d, n, 2, seed=5)
    _, rx, x0 = random_tt(d, n, 2, seed=6)
    runs = []
    for scale in (1.0, s):
        n_, m_, ra, A = pack_tt_matrix(laplace_tt(d, n, scale))
        b = y.copy()
        b[:ry[0] * n * ry[1]] *= scale
        cores, r = ttgpu.dtt_amen_solve(d, n_, m_, ry, ra, A, b, x0, rx, tol, ctx=ctx)
        T = np.ones((1, 1))
        off = 0
        for k in range(d):
            c = cores[off:off + r[k] * n * r[k + 1]].reshape(r[k], n * r[k + 1], order="F")
            off += c.size
            T = (T @ c).reshape(-1, r[k + 1], order="F")
        runs.append((r, T[:, 0]))
    (r1, x1), (r2, x2) = runs
    assert np.linalg.norm(x1 - x2) <= 1e-6 * np.linalg.norm(x1)
