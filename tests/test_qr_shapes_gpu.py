"""QR of very wide and very tall, thin blocks: scratch and time."""
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


@pytest.mark.parametrize("cplx", [False, True])
def test_no_words_for_a_wide_qr(torch_cuda, ctx, cplx):
    import ttgpu
    n, m = 8, 200_000
    dt = torch_cuda.complex128 if cplx else torch_cuda.float64
    a = torch_cuda.randn(n * m, dtype=dt, device="cuda")
    r = torch_cuda.zeros(n * m, dtype=dt, device="cuda")
    a0 = a.clone()
    used = _reserved(torch_cuda, lambda c: ttgpu.dqr(n, m, a, r, complex_=cplx, ctx=c))
    assert used <= 16 << 20, used
    Q, R = a[:n * n].view(n, n).T, r.view(m, n).T
    err = torch_cuda.linalg.norm(Q @ R - a0.view(m, n).T) / torch_cuda.linalg.norm(a0)
    assert float(err) <= 10 * n * 2.0 ** -53
