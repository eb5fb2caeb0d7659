"""Pair sweeps with more column pairs a block of threads than it keeps rotations of
(blocks of some tens of thousands of columns on a whole GPU): the same code on a
bounded grid, in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import sys
sys.path.insert(0, %r)
import numpy as np, torch, ttgpu
for p, q in ((150, 150), (400, 131), (90, 200), (1300, 70)):
    rng = np.random.default_rng(p + q)
    U, V = np.linalg.qr(rng.standard_normal((p, min(p, q))))[0], np.linalg.qr(rng.standard_normal((q, min(p, q))))[0]
    s0 = 10.0 ** -np.linspace(0, 12, min(p, q))
    A = (U * s0) @ V.T
    r = min(p, q)
    M = torch.from_numpy(np.ravel(A, order="F").copy()).cuda()
    u, s, vt = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (p * r, r, r * q))
    ttgpu.dgesvd(p, q, M, u, s, vt)
    torch.cuda.synchronize()
    u, s, vt = u.cpu().numpy().reshape(p, r, order="F"), s.cpu().numpy(), vt.cpu().numpy().reshape(r, q, order="F")
    n = np.linalg.norm(A)
    assert np.linalg.norm((u * s) @ vt - A) <= 1e-13 * n
    assert np.linalg.norm(u.T @ u - np.eye(r)) <= 1e-12 and np.linalg.norm(vt @ vt.T - np.eye(r)) <= 1e-12
    assert abs(s - np.linalg.svd(A, compute_uv=False)).max() <= 1e-14
print("fine")
"""


@pytest.mark.parametrize("ctas", [1, 2, 5])
def test_many_pairs_a_block(torch_cuda, ctas):
    root = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tt-fort_gb300")
    r = subprocess.run([sys.executable, "-c", CODE % root], capture_output=True, text=True, timeout=120,
                       env={**os.environ, "TTG_SVD_CTAS": str(ctas)})
    assert r.returncode == 0 and "fine" in r.stdout, r.stderr[-2000:]
