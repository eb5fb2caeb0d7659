"""FP64 products on the tensor cores by error-free splitting (ttg_oz.cu).

Bound of one split product C = A B (K terms): an operand element is rounded to
2^-56 2^e <= 2^-55 of its row's (column's) largest, twice, and the dropped
digit products sum to at most 6.1 2^-56 K 2^(ea + eb) <= 24.4 2^-56 K amax bmax;
together below 2^-51 K amax bmax, plus the last rounding u |C| (u = 2^-53).
numpy's own product lies within (K + 2) u |A| |B|.  Chained products add the
bound of the first, carried through the absolute values of the next.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _t(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def oz_bound(A, B):
    K = A.shape[1]
    return K * 2.0 ** -51 * np.outer(abs(A).max(1), abs(B).max(0))


def plain_product(torch, ctx, X, P2):
    """X (M x K) P2 (K x N) as the first product of nvec = M local problems of
    size 1 x 1 x K, and the launches it took (three on the FP64 kernels)."""
    import ttgpu
    M, K = X.shape
    N = P2.shape[1]
    one = torch.ones(1, dtype=torch.float64, device="cuda")
    y = torch.zeros(M * N, dtype=torch.float64, device="cuda")
    l0 = ttgpu.launch_count()
    ttgpu.dbfun3(1, 1, K, 1, 1, N, 1, 1, one, one, _t(torch, np.ravel(P2, order="F")),
                 _t(torch, X.ravel()), y, nvec=M)
    ctx.synchronize()
    return y.cpu().numpy().reshape(M, N), ttgpu.launch_count() - l0


@pytest.mark.parametrize("M,N,K", [
    (128, 640, 512), (127, 1281, 257), (129, 1023, 255), (513, 321, 241), (2000, 63, 529),
    (1025, 65, 1000), (96, 77, 5248), (300, 200, 4097), (4096, 640, 64),
])
def test_split_product_at_tile_edges(torch_cuda, ctx, M, N, K):
    rng = np.random.default_rng(M + N + K)
    X, P2 = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    got, launches = plain_product(torch_cuda, ctx, X, P2)
    assert launches > 3, "the split product was not taken"
    err = abs(got - X @ P2)
    assert (err <= oz_bound(X, P2) + (K + 4) * U * (abs(X) @ abs(P2))).all()
    # and no less exact than the FP64 chain in the norm: against sums in extended
    # precision of a sample of rows
    rows = rng.integers(0, M, 4)
    ref = (X[rows].astype(np.longdouble)[:, :, None] * P2.astype(np.longdouble)[None]).sum(1)
    rel = np.linalg.norm((got[rows] - ref).astype(float)) / np.linalg.norm(ref.astype(float))
    assert rel <= 6e-16


@pytest.mark.parametrize("value", [1.0 / 3, 0.5019607843137, 1.0 - 2.0 ** -53, -0.998046875])
def test_constant_digits_stay_exact(torch_cuda, ctx, value):
    """Equal elements give every digit product the same sign: the largest
    sums tensor memory has to hold exactly."""
    M, N, K = 256, 512, 512
    got, launches = plain_product(torch_cuda, ctx, np.full((M, K), value), np.full((K, N), value))
    assert launches > 3
    ref = float(np.longdouble(value) * np.longdouble(value) * K)
    assert (abs(got - ref) <= 2 * U * abs(ref)).all()


def test_special_values_as_the_fp64_chain(torch_cuda, ctx):
    """Infinities, NaN, zeros, subnormal and extreme rows and columns: where
    the FP64 chain gives a non-finite value so does the split product, and
    the same one; finite sums of positive terms agree to 2 (K + 2) u."""
    rng = np.random.default_rng(5)
    M, N, K = 300, 513, 320
    X, P2 = rng.random((M, K)) + 0.1, rng.random((K, N)) + 0.1
    X[3, 17], X[40, 0], X[41, 5], X[41, 6] = np.nan, np.inf, np.inf, -np.inf
    X[128] *= 1e200
    X[129] *= 1e-200
    X[130] = 0.0
    X[131] = 5e-324
    X[132, 1:] = 0.0
    X[133, ::2] *= 1e-30
    P2[9, 64], P2[11, 130] = -np.inf, np.nan
    P2[:, 200] *= 1e-250
    P2[:, 201] *= 1e180
    P2[:, 202] = 0.0
    got, launches = plain_product(torch_cuda, ctx, X, P2)
    assert launches > 3
    with np.errstate(all="ignore"):
        ref = X @ P2
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    inf = np.isinf(ref)
    assert np.array_equal(got[inf], ref[inf])
    fin = np.isfinite(ref)
    assert (abs(got[fin] - ref[fin]) <= 2 * (K + 2) * U * abs(ref[fin]) + 1e-320).all()


@pytest.mark.parametrize("r1,r2,nvec", [(64, 64, 5), (101, 90, 3), (128, 77, 6), (37, 200, 4)])
def test_spin_chain_operator(torch_cuda, ctx, r1, r2, nvec):
    """n = 2: the core contracted into Phi2 first, against the FP64 kernels
    (ttg_dbfun3_noalloc), each within the chained bounds."""
    import ctypes as C
    import ttgpu
    rng = np.random.default_rng(r1)
    n, ra = 2, 5
    p1, A, p2 = (rng.standard_normal(k) for k in (r1 * r1 * ra, ra * n * n * ra, r2 * ra * r2))
    x = rng.standard_normal(r1 * n * r2 * nvec)
    args = [_t(torch_cuda, v) for v in (p1, A, p2, x)]
    y = torch_cuda.zeros(x.size, dtype=torch_cuda.float64, device="cuda")
    z = torch_cuda.zeros_like(y)
    l0 = ttgpu.launch_count()
    ttgpu.dbfun3(r1, n, r2, r1, n, r2, ra, ra, *args, y, nvec=nvec)
    assert ttgpu.launch_count() - l0 > 3
    ctx.check(ttgpu.lib().ttg_dbfun3_noalloc(
        ctx.handle, *[C.c_int64(v) for v in (r1, n, r2, r1, n, r2, ra, ra)],
        *[C.c_void_p(t.data_ptr()) for t in (*args, z)], C.c_int64(nvec)))
    ctx.synchronize()
    P1 = p1.reshape(r1, r1, ra, order="F")
    AA = A.reshape(ra, n, n, ra, order="F")
    P2 = p2.reshape(r2, ra, r2, order="F")
    X = x.reshape(r1, n, r2, nvec, order="F")
    Q = np.einsum("dija,eac->icdje", abs(AA), abs(P2)).reshape(-1, n * r2)
    XX = abs(X).transpose(0, 3, 1, 2).reshape(r1 * nvec, n * r2)
    T = Q @ XX.T                                     # (i c2 a1) x (b1 v)
    eT = oz_bound(Q, XX.T) + (n * r2 + 8) * U * T    # (the core's own rounding: ra + 1 terms)
    shape = (n, r2, ra, r1, nvec)
    T, eT = T.reshape(shape), eT.reshape(shape)
    Tm = T.transpose(3, 2, 0, 1, 4).reshape(r1 * ra, -1)
    eTm = eT.transpose(3, 2, 0, 1, 4).reshape(r1 * ra, -1)
    P1m = P1.reshape(r1, r1 * ra)
    P1m = np.abs(P1m)
    bound = P1m @ eTm + oz_bound(P1m, Tm) + (r1 * ra + n * ra + r2 + 8) * U * (P1m @ Tm)
    got = y.cpu().numpy().reshape(r1, n, r2, nvec, order="F").reshape(r1, -1)
    ref = z.cpu().numpy().reshape(r1, n, r2, nvec, order="F").reshape(r1, -1)
    assert (abs(got - ref) <= 2 * bound).all()
    assert np.linalg.norm(got - ref) <= 4e-15 * np.linalg.norm(ref)


@pytest.mark.parametrize("r1,n,r2,nvec", [(48, 32, 48, 1), (33, 17, 40, 4), (64, 20, 9, 3)])
def test_complex_operator_and_adjoint(torch_cuda, ctx, r1, n, r2, nvec):
    """Complex products run as real ones with rows and K doubled: operator and
    adjoint against numpy to the FP64 kernels' tolerance, and adjoint to each
    other."""
    import ttgpu
    rng = np.random.default_rng(n)
    ra = 6
    c = lambda k: rng.standard_normal(k) + 1j * rng.standard_normal(k)
    p1, A, p2 = c(r1 * r1 * ra), c(ra * n * n * ra), c(r2 * ra * r2)
    x, w = c(r1 * n * r2 * nvec), c(r1 * n * r2 * nvec)
    args = [_t(torch_cuda, v) for v in (p1, A, p2)]
    y = torch_cuda.zeros(x.size, dtype=torch_cuda.complex128, device="cuda")
    yt = torch_cuda.zeros_like(y)
    l0 = ttgpu.launch_count()
    ttgpu.zbfun3(r1, n, r2, r1, n, r2, ra, ra, *args, _t(torch_cuda, x), y, nvec)
    ttgpu.zbfun3(r1, n, r2, r1, n, r2, ra, ra, *args, _t(torch_cuda, w), yt, nvec, transp=True)
    assert ttgpu.launch_count() - l0 > 6
    ctx.synchronize()
    P1, AA = p1.reshape(r1, r1, ra, order="F"), A.reshape(ra, n, n, ra, order="F")
    P2, X = p2.reshape(r2, ra, r2, order="F"), x.reshape(r1, n, r2, nvec, order="F")
    t = np.einsum("eac,bjev->bjacv", P2, X, optimize=True)
    t = np.einsum("dija,bjacv->bdicv", AA, t, optimize=True)
    ref = np.einsum("zbd,bdicv->zicv", P1, t, optimize=True)
    got, gott = y.cpu().numpy(), yt.cpu().numpy()
    assert np.linalg.norm(got - np.ravel(ref, order="F")) <= 1e-14 * np.linalg.norm(ref)
    a, b = np.vdot(w, got), np.vdot(gott, x)
    assert abs(a - b) <= 1e-13 * np.linalg.norm(w) * np.linalg.norm(got)


@pytest.mark.parametrize("r1,m,r2,ry1,n,ry2", [(60, 40, 51, 45, 33, 70), (82, 64, 77, 82, 64, 77)])
def test_interface_updates(torch_cuda, ctx, r1, m, r2, ry1, n, ry2):
    """Rectangular interface updates with long K (the K-split path)."""
    import ttgpu
    from oracle import ops
    rng = np.random.default_rng(r1 + ry2)
    ra1, ra2 = 3, 2
    A = rng.standard_normal(ra1 * n * m * ra2)
    x, y = rng.standard_normal(r1 * m * r2), rng.standard_normal(ry1 * n * ry2)
    q1, q2 = rng.standard_normal(ry1 * r1 * ra1), rng.standard_normal(r2 * ra2 * ry2)
    L = torch_cuda.zeros(ry2 * r2 * ra2, dtype=torch_cuda.float64, device="cuda")
    R = torch_cuda.zeros(r1 * ra1 * ry1, dtype=torch_cuda.float64, device="cuda")
    l0 = ttgpu.launch_count()
    t = lambda a: _t(torch_cuda, a)
    ttgpu.phi_left(r1, m, r2, ry1, n, ry2, ra1, ra2, t(q1), t(A), t(x), t(y), L)
    ttgpu.phi_right(r1, m, r2, ry1, n, ry2, ra1, ra2, t(q2), t(A), t(x), t(y), R)
    assert ttgpu.launch_count() - l0 > 6
    ctx.synchronize()
    for got, ref in ((L, ops.phi_left(r1, m, r2, ry1, n, ry2, ra1, ra2, q1, A, x, y)),
                     (R, ops.phi_right(r1, m, r2, ry1, n, ry2, ra1, ra2, q2, A, x, y))):
        assert np.linalg.norm(got.cpu().numpy() - ref) <= 1e-14 * np.linalg.norm(ref)


@pytest.mark.parametrize("M,N,K", [
    (256, 120, 256), (256, 120, 400), (250, 120, 512), (256, 120, 560), (200, 128, 700),
    (256, 120, 1000), (1000, 128, 700),
])
def test_k_split_over_clusters(torch_cuda, ctx, M, N, K):
    """K in 4, 5, 8 and 7 chunks of one cluster (no summing kernel), in two and
    three clusters of four (one chunk of the last is empty), with ragged
    columns shared out: bounds as above, flagged rows among them."""
    rng = np.random.default_rng(M + N + K)
    X, P2 = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    X[5, K // 2], X[M - 1, 0] = np.nan, np.inf
    P2[K - 1, N - 1] = np.inf
    got, launches = plain_product(torch_cuda, ctx, X, P2)
    assert launches > 3, "the split product was not taken"
    with np.errstate(all="ignore"):
        ref = X @ P2
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    rows, cols = np.isfinite(X).all(1), np.isfinite(P2).all(0)
    A, B = X[rows], P2[:, cols]
    err = abs(got[rows][:, cols] - A @ B)
    assert (err <= oz_bound(A, B) + (K + 4) * U * (abs(A) @ abs(B))).all()


@pytest.mark.parametrize("M,N,K", [
    (640, 320, 128), (129, 33, 640), (1000, 31, 300), (2000, 97, 256), (2432, 130, 200), (2433, 127, 200),
])
def test_narrow_tiles(torch_cuda, ctx, M, N, K):
    """32 columns a tile where 64 leave more than half of the SMs idle, at the
    edges of a tile and on both sides of the rule (76 tiles of 128 x 64)."""
    rng = np.random.default_rng(M + N + K)
    X, P2 = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    got, launches = plain_product(torch_cuda, ctx, X, P2)
    assert launches > 3, "the split product was not taken"
    err = abs(got - X @ P2)
    assert (err <= oz_bound(X, P2) + (K + 4) * U * (abs(X) @ abs(P2))).all()


@pytest.mark.parametrize("r1,n,r2,ra,nvec", [(40, 24, 17, 6, 3), (17, 30, 40, 5, 2), (24, 16, 24, 2, 1)])
def test_complex_doubled_side(torch_cuda, ctx, r1, n, r2, ra, nvec):
    """Complex products double the rows of the smaller operand: stages with
    either side the smaller, odd columns, an infinite and a NaN element (their
    rows and columns take the FP64 chain), against numpy by einsum to 4 K u of
    the absolute values per stage."""
    import ttgpu
    rng = np.random.default_rng(r1 + n)

    def z(*s):
        return rng.standard_normal(s) + 1j * rng.standard_normal(s)
    p1, A, p2 = z(r1, r1, ra), z(ra, n, n, ra), z(r2, ra, r2)   # [c,b,a] [a,i,j,e] [b,e,c]
    x = z(r1, n, r2, nvec)
    t = [_t(torch_cuda, np.ravel(v, order="F")) for v in (p1, A, p2, x)]
    y = torch_cuda.zeros(r1 * n * r2 * nvec, dtype=torch_cuda.complex128, device="cuda")
    ttgpu.zbfun3(r1, n, r2, r1, n, r2, ra, ra, *t, y, nvec)
    ctx.synchronize()
    got = y.cpu().numpy().reshape(r1, n, r2, nvec, order="F")

    def product(P1, C, P2, X):
        T = np.einsum("xjbv,bec->xjecv", X, P2, optimize=True)
        T = np.einsum("aije,xjecv->xaicv", C, T, optimize=True)
        return np.einsum("cxa,xaidv->cidv", P1, T, optimize=True)
    ref = product(p1, A, p2, x)
    size = product(abs(p1), abs(A), abs(p2), abs(x))
    K = r2 + n * ra + r1 * ra
    # the split stages' bound is relative to row and column maxima: each factor's
    # largest element over its mean square is below 8 at these sizes
    assert (abs(got - ref) <= 8 * 4 * K * U * size.max()).all()
    x[1, 2, 3, 0] = np.inf
    x[0, 1, 2, nvec - 1] = np.nan
    t[3] = _t(torch_cuda, np.ravel(x, order="F"))
    ttgpu.zbfun3(r1, n, r2, r1, n, r2, ra, ra, *t, y, nvec)
    ctx.synchronize()
    bad = y.cpu().numpy().reshape(r1, n, r2, nvec, order="F")
    # every output of those vectors sees the element; the others stay finite
    assert not np.isfinite(bad[..., 0]).any() and not np.isfinite(bad[..., nvec - 1]).any()
    if nvec > 2:
        assert np.isfinite(bad[..., 1]).all()
