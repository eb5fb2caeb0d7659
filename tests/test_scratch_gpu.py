"""Scratch of single calls: what the call uses and no more.  A product whose split
operands would pass the 4 GiB limit stays on the FP64 kernels and reserves nothing
for them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reserved(torch, call):
    """Device bytes that a fresh context's call leaves allocated."""
    import ttgpu
    torch.cuda.synchronize()
    ctx = ttgpu.Context(0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    call(ctx)
    ctx.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    ctx.close()
    return used


def test_no_room_for_products_beyond_the_limit(torch_cuda, ctx):
    """The first product, (rx1 m + ry2) rx2 = 3.2e8 elements, 14 bytes each of digit
    planes: 4.5 GB."""
    import ttgpu
    r1, m, r2, ry2 = 320, 1000, 1000, 8
    rnd = lambda k: torch_cuda.randn(k, dtype=torch_cuda.float64, device="cuda")
    x, A, p1, p2 = rnd(r1 * m * r2), rnd(m), rnd(r1), rnd(r2 * ry2)
    y = torch_cuda.zeros(ry2, dtype=torch_cuda.float64, device="cuda")
    used = _reserved(torch_cuda, lambda c: ttgpu.dbfun3(r1, m, r2, 1, 1, ry2, 1, 1, p1, A, p2, x, y, ctx=c))
    assert used <= 2 * r1 * m * ry2 * 8 + (64 << 20), used   # the two intermediates
    T = p2.view(ry2, r2) @ x.view(r2, m * r1)                # [c2, (j, b1)]
    ref = (T.view(ry2, m, r1) * A[None, :, None]).sum(1) @ p1
    assert torch_cuda.allclose(y, ref, rtol=1e-10, atol=0)


@pytest.mark.parametrize("kind", ["dbfun3", "zbfun3", "phi", "localop"])
def test_a_call_in_its_own_scratch(torch_cuda, ctx, kind):
    """A context whose workspace is exactly one call's: split and unsplit products, the
    spin chain's form, blocks of fewer vectors than were prepared for."""
    import ttgpu
    rng = np.random.default_rng(3)
    for (r1, n, r2, ra, nv) in [(64, 2, 60, 5, 5), (40, 24, 33, 3, 4), (7, 3, 5, 2, 1), (130, 1, 90, 4, 2)]:
        z = kind == "zbfun3"
        g = (lambda k: rng.standard_normal(k) + 1j * rng.standard_normal(k)) if z else rng.standard_normal
        t = lambda a: torch_cuda.from_numpy(a).cuda()
        p1, A, p2 = t(g(r1 * r1 * ra)), t(g(ra * n * n * ra)), t(g(r2 * ra * r2))
        x, w = t(g(r1 * n * r2 * nv)), t(g(r1 * n * r2 * nv))
        outs = []
        big = ttgpu.Context(0)
        fresh = ttgpu.Context(0)
        for c in (fresh, big):
            if c is big:      # a workspace that a larger call left
                s = 300
                a = torch_cuda.zeros(s * s * 4, dtype=torch_cuda.float64, device="cuda")
                b = torch_cuda.zeros(s * s * 4, dtype=torch_cuda.float64, device="cuda")
                ttgpu.dbfun3(s, 2, s, s, 2, s, 2, 2, a, a, a, a, b, nvec=2, ctx=c)
            y = torch_cuda.zeros_like(x)
            if kind == "dbfun3":
                ttgpu.dbfun3(r1, n, r2, r1, n, r2, ra, ra, p1, A, p2, x, y, nvec=nv, ctx=c)
            elif kind == "zbfun3":
                ttgpu.zbfun3(r1, n, r2, r1, n, r2, ra, ra, p1, A, p2, x, y, nv, ctx=c)
                y2 = torch_cuda.zeros_like(x)
                ttgpu.zbfun3(r1, n, r2, r1, n, r2, ra, ra, p1, A, p2, w, y2, nv, transp=True, ctx=c)
                y = torch_cuda.cat([y, y2])
            elif kind == "phi":
                L = torch_cuda.zeros(r2 * r2 * ra, dtype=torch_cuda.float64, device="cuda")
                R = torch_cuda.zeros(r1 * r1 * ra, dtype=torch_cuda.float64, device="cuda")
                ttgpu.phi_left(r1, n, r2, r1, n, r2, ra, ra, p1, A, x, w, L, ctx=c)
                ttgpu.phi_right(r1, n, r2, r1, n, r2, ra, ra, p2, A, x, w, R, ctx=c)
                y = torch_cuda.cat([L, R])
            else:
                op = ttgpu.LocalOp(r1, n, r2, r1, n, r2, ra, ra, p1, A, p2, nvec_max=nv, ctx=c)
                for v in range(nv, 0, -1):
                    op.apply(x, y, v)
                c.synchronize()
                op.close()
            c.synchronize()
            outs.append(y.cpu().numpy())
            c.close()
        assert np.array_equal(outs[0], outs[1])
