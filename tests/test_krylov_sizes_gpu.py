"""The time stepper's Gram-Schmidt and norm-estimate kernels over their sizes:
local problems below one warp, of 64 and 128 entries, in one and several CTAs
of a cluster, one to four entries a thread, and beyond the cluster (a grid).
Against the CPU restatement, one step, to the 1e-8 each exponential is asked
for."""
import numpy as np
import pytest

from oracle.ksl import ztt_ksl as oracle_ksl, tt_full
from ttgpu.operators import ksl_operator, random_tt_complex, tt_norm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,r", [(3, 3, 2), (3, 8, 4), (2, 16, 8), (2, 33, 31), (3, 20, 11),
                                   (2, 64, 33), (2, 80, 64), (2, 100, 90)])
def test_local_problem_sizes(ctx, d, n, r):
    import ttgpu
    n_, m_, ra, crA = ksl_operator(d=d, n=n, rank=2, seed=n)
    _, ry, y = random_tt_complex(d, n, r, seed=r)
    y = y / tt_norm(d, n, ry, y) ** (1.0 / d)
    c, r1 = ttgpu.ztt_ksl(d, n_, m_, ra, crA, y, ry, 1e-3, 64, ctx=ctx)
    o = oracle_ksl(d, n_, m_, ra, crA, y, ry, 1e-3, 64)
    a, b = tt_full(d, n_, r1, c), tt_full(d, n_, o["ry"], o["cores"])
    assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)
