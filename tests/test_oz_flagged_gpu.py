"""Split products with flagged rows (ttg_oz.cu): a product that meets an infinity,
a NaN or an extreme row is formed by FP64 FMA chains over all SMs.

Values: against numpy in the pattern of non-finite outputs, and within the FP64
chain's bound (K + 2) u |A| |B| beside them.  Time: a call whose every product
is flagged costs at most twice the FP64 pipe's time for its flops (two FMAs per
clock on 152 SMs, 1.2 TFLOP/s) on top of the unflagged call."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _t(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("r1,n,r2,ra", [(82, 64, 77, 3), (256, 2, 256, 5)])
def test_a_flagged_call_costs_no_more_than_fp64(torch_cuda, ctx, r1, n, r2, ra):
    import ttgpu
    rng = np.random.default_rng(r1)
    A, x, y = (rng.standard_normal(k) for k in (ra * n * n * ra, r1 * n * r2, r1 * n * r2))
    q = rng.standard_normal(r1 * r1 * ra)
    out = torch_cuda.zeros(r2 * r2 * ra, dtype=torch_cuda.float64, device="cuda")
    best = []
    for bad in (False, True):
        if bad:
            q[7] = np.inf
        t = [_t(torch_cuda, v) for v in (q, A, x, y)]
        times = []
        for _ in range(8):
            ctx.synchronize()
            t0 = time.perf_counter()
            ttgpu.phi_left(r1, n, r2, r1, n, r2, ra, ra, *t, out)
            ctx.synchronize()
            times.append(time.perf_counter() - t0)
        best.append(min(times))
    flops = 2.0 * (r1 * ra * n * r2 * r1 + r1 * r2 * (n * ra) ** 2 + r2 * ra * r2 * r1 * n)
    assert best[1] <= 2.0 * flops / 1.2e12 + best[0], (best, flops / 1.2e12)


@pytest.mark.parametrize("M,N,K", [(1, 700, 4000), (129, 33, 640), (2049, 70, 200), (300, 200, 4097),
                                   (96, 77, 5248), (1000, 129, 257)])
@pytest.mark.parametrize("side", ["row", "column"])
def test_tiles_beside_a_flag(torch_cuda, ctx, M, N, K, side):
    """One extreme row (or column) in shapes of one tile, of K splits in one cluster
    and in several: its elements and those beside it."""
    import ttgpu
    rng = np.random.default_rng(M + N + K)
    X, P = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    X[M // 2, K // 3] = np.nan
    if side == "row":
        X[M - 1] *= 1e140
    else:
        P[:, N - 1] *= 1e-140
    one = torch_cuda.ones(1, dtype=torch_cuda.float64, device="cuda")
    y = torch_cuda.zeros(M * N, dtype=torch_cuda.float64, device="cuda")
    ttgpu.dbfun3(1, 1, K, 1, 1, N, 1, 1, one, one, _t(torch_cuda, np.ravel(P, order="F")),
                 _t(torch_cuda, X.ravel()), y, nvec=M)
    ctx.synchronize()
    got = y.cpu().numpy().reshape(M, N)
    rows = np.arange(M) != M // 2
    assert np.isnan(got[~rows]).all() and np.isfinite(got[rows]).all()
    ref, size = X[rows] @ P, abs(X[rows]) @ abs(P)
    # tiles of normal rows: the split product's bound (see test_oz_gpu.py)
    bound = 2 * (K + 4) * U * size + K * 2.0 ** -51 * np.outer(abs(X[rows]).max(1), abs(P).max(0))
    assert (abs(got[rows] - ref) <= bound).all()
    # the extreme row or column itself: chains
    ext = np.s_[-1:, :] if side == "row" else np.s_[:, -1:]
    if side == "column" or M // 2 != M - 1:
        assert (abs(got[rows] - ref)[ext] <= 2 * (K + 4) * U * size[ext]).all()
