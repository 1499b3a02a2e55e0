"""Sums of the multi-step row kernel. T_0's norms (the zeroth moments) of host vectors whose
squares are exact show the sums alone.

FP64: rounding at every addition is 2^-53 of the sum so far, uniform: rms 4.4e-17 of it. A
tree adds up to 4.4e-17 sqrt(1 + 1/2 + 1/4 + ...) = 6.2e-17 of the total, whatever goes
before its last levels; one chain over 152 blocks to 4.4e-17 sqrt(152 / 3) = 3.1e-16. The
bound lies between: 1.5e-16 rms.
"""
import math
from fractions import Fraction

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


@pytest.mark.parametrize("n,block", [(3000, 8), (9001, 8), (9001, 16), (12000, 32)])
def test_fp64_rows_are_not_one_chain(n, block):
    """A row of 64 positive products, alone in the first moment: T_0 is 1 in its row and every
    other row's values are zero. One chain of 64 additions errs by 4.4e-17 sqrt(64 / 3) =
    2.0e-16 of the sum (rms), two of 32 and their sum by 4.4e-17 sqrt(32 / 3 / 2 + 1) =
    1.1e-16. The bound lies between."""
    rng = np.random.default_rng(n + block)
    col = (np.arange(n)[:, None] + np.arange(1, 65)) % n
    val = np.zeros((n, 64))
    val[0] = rng.uniform(0.005, 0.015, 64)
    x = rng.uniform(0.5, 1.5, (128, n))
    x[:, 0] = 1.0
    order = np.argsort(col, axis=1)
    col, val = np.take_along_axis(col, order, 1), np.take_along_axis(val, order, 1)
    with L.Context(0) as ctx:
        csr = ctx.upload_csr(np.arange(n + 1) * 64, col.ravel(), val.ravel())
        cfg = L.kpm_cfg(8, R=128, kind=L.VEC_HOST, precision=L.FP64, block=block)
        assert csr.step_kernel(cfg)[0] == 6
        mu = csr.kpm_dos(cfg, x)
    exact = [sum((Fraction(w) * Fraction(v) for w, v in zip(val[0], r[col[0]])), Fraction(0)) for r in x]
    err = [float((Fraction(m) - e) / e) for m, e in zip(mu[:, 1], exact)]
    assert np.sqrt(np.mean(np.square(err))) <= 1.5e-16


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
