"""Random-phase start vectors of FP32 runs (FP32 pairs and a table) against the
oracle's FP64 functions, through moments that any wrong entry would show.

mu_0 and mu_1 of one step are sums over the entries; entries agree to half an FP32 ulp,
so each moment agrees to 2^-23 of the sum of magnitudes.
"""
import numpy as np
import pytest

import leo2d_gb300 as L
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R,first", [(1, 1, 0), (255, 3, 0), (5000, 16, 7), (40_001, 16, 1 << 33)])
def test_local_products(n, R, first):
    """A diagonal matrix with random entries: mu_k = sum_i d_i^k-like weights times the
    squared magnitude of each entry, and a permutation that pairs cos with sin."""
    rng = np.random.default_rng(n)
    d = rng.uniform(-0.9, 0.9, n)
    with L.Context(0) as ctx:
        csr = ctx.upload_csr(np.arange(n + 1), np.arange(n), d)
        mu = csr.kpm_dos(L.kpm_cfg(8, R=R, kind=L.VEC_PHASE, precision=L.FP32, seed=5, first_vector=first))
    re, im = oracle.phase_vectors(5, first, R, n)
    x2 = re.astype(np.float32).astype(np.float64) ** 2 + im.astype(np.float32).astype(np.float64) ** 2
    t = np.arccos(d)
    ref = np.stack([(np.cos(k * t) * x2).sum(axis=1) for k in range(8)], axis=1)
    # (the FP32 recursion on d adds a few ulp a step to each term)
    assert np.max(np.abs(mu - ref)) <= 32 * 2.0**-23 * n
