"""Sums of the multi-step row kernel. T_0's norms (the zeroth moments) of host vectors whose
squares are exact show the sums alone.

FP64: rounding at every addition is 2^-53 of the sum so far, uniform: rms 4.4e-17 of it. A
tree adds up to 4.4e-17 sqrt(1 + 1/2 + 1/4 + ...) = 6.2e-17 of the total, whatever goes
before its last levels; one chain over 152 blocks to 4.4e-17 sqrt(152 / 3) = 3.1e-16. The
bound lies between: 1.5e-16 rms.
"""
import math

import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


def _ring(n):
    """Neighbours at distances 1 to 4 on a ring."""
    i = np.repeat(np.arange(n), 8)
    j = (i + np.tile([-4, -3, -2, -1, 1, 2, 3, 4], n)) % n
    o = np.lexsort((j, i))
    return np.arange(n + 1) * 8, j[o], np.full(8 * n, 0.11)


@pytest.mark.parametrize("n,block", [(5000, 8), (3000, 16), (9001, 8), (12000, 16), (20000, 32), (20000, 64)])
def test_fp64_sums_are_a_tree(n, block):
    x = np.random.default_rng(n + block).standard_normal((64, n)).astype(np.float32).astype(np.float64)
    exact = np.array([math.fsum(v * v) for v in x])
    with L.Context(0) as ctx:
        csr = ctx.upload_csr(*_ring(n))
        cfg = L.kpm_cfg(64, R=64, kind=L.VEC_HOST, precision=L.FP64, block=block)
        assert csr.step_kernel(cfg)[0] == 6
        mu = csr.kpm_dos(cfg, x)
    assert np.sqrt(np.mean(((mu[:, 0] - exact) / exact) ** 2)) <= 1.5e-16


# (400,000 rows of 8 columns, 60,000 of 128: a lane of the panels takes several blocks a step)
@pytest.mark.parametrize("n,R,block", [(3000, 8, 8), (3000, 32, 32), (9001, 16, 16), (12000, 64, 64), (400000, 8, 8),
                                       (60000, 128, 128)])
def test_fp32_sums_of_four_rows(n, R, block):
    """Entries k / 2048 with 1024 <= k < 2048: the sum of four squares is a whole number of
    2^-22 below 2^24 of them, exact in FP32 (of sixteen it is not), and so are the pairs
    and the FP64 sums beyond. So T_0's norms are exact."""
    k = np.random.default_rng(n + block).integers(1024, 2048, (R, n))
    with L.Context(0) as ctx:
        csr = ctx.upload_csr(*_ring(n))
        cfg = L.kpm_cfg(64, R=R, kind=L.VEC_HOST, block=block)
        assert csr.step_kernel(cfg)[0] == 6
        mu = csr.kpm_dos(cfg, k / 2048.0)
    np.testing.assert_array_equal(mu[:, 0], (k * k).sum(1) / 2.0**22)
