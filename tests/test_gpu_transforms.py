"""The FP64 transforms at the edges of their kernels against the oracle.

A density is a sum of P terms of at most |g mu|: its FP64 rounding is within P
2^-53 of the sum of their sizes, times the node's weight. The bound below takes
eight times that.
"""
import numpy as np
import pytest

import leo2d_gb300 as L
from oracle import oracle

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def ctx():
    with L.Context(0) as c:
        yield c


# pairs of nodes (k, P-1-k) in warps of 8: one pair, odd P, edges of a block and of the grid
@pytest.mark.parametrize("P,sets", [(2, 1), (3, 1), (4, 2), (15, 1), (16, 3), (17, 1), (33, 1), (1000, 1), (2433, 1),
                                    (4096, 2), (19460, 1)])
def test_dos_transform(ctx, P, sets):
    mu = np.random.default_rng(P).uniform(-1, 1, (sets, P))
    dos, E = ctx.dos_transform(mu, P, 1.7, 0.2, 0.5)
    if P <= 4096:
        ref, Er = oracle.dos_transform(mu, P, 1.7, 0.2, 0.5)
    else:  # the definition at a few nodes
        i = np.arange(P)
        g = ((P - i) * np.cos(np.pi * i / P) + np.sin(np.pi * i / P) / np.tan(np.pi / P)) / P * mu[0]
        Er = 0.2 + 1.7 * np.cos((i + 0.5) * np.pi / P)
        ref = dos.copy()
        for k in (0, 1, P // 2 - 1, P // 2, P - 2, P - 1):
            m = (i * (2 * k + 1)) % (4 * P)
            acc = g[0] + 2 * np.sum(g[1:] * np.cos(np.pi * m[1:] / (2 * P)))
            ref[k] = 0.5 * acc / (np.pi * np.sqrt(1.7 ** 2 - (Er[k] - 0.2) ** 2))
    w = 0.5 / (np.pi * 1.7 * np.abs(np.sin((np.arange(P) + 0.5) * np.pi / P)))
    tol = 8 * P * EPS * 2 * np.abs(mu).sum() / sets
    # (the weight itself loses bits where E comes near the band edge)
    assert np.all(np.abs(dos - ref) <= tol * w * (1 + P * P * EPS) + np.abs(ref) * 16 * P * P * EPS)
    np.testing.assert_allclose(E, Er, rtol=0, atol=8 * EPS)


# 32 energies a block, rows in groups of 32 per block row, chunks of energies
@pytest.mark.parametrize("M,n", [(2, 1), (3, 31), (4, 33), (31, 32), (33, 100), (64, 1001), (130, 65), (513, 40),
                                 (40, 300000)])
def test_cond_sigma(ctx, M, n):
    mu = np.random.default_rng(M).uniform(-1, 1, (M, M))
    E = np.linspace(-1.3, 1.3, n) if n > 1 else np.array([0.1])
    got = ctx.cond_sigma(mu, E, 1.2, 0.05, 0.7)
    pick = np.unique(np.r_[np.arange(min(n, 40)), np.arange(0, n, max(1, n // 60)), n - 1])
    ref = oracle.cond_sigma(mu, E[pick], 1.2, 0.05, 0.7)
    x = (E[pick] - 0.05) / 1.2
    inside = np.abs(x) < 1
    assert np.all(got[pick][~inside] == 0)
    # T_n by its recurrence loses up to n^2 2^-53; M^2 products of such terms
    tol = 8 * (M * M + 2 * M) * EPS * 4 * np.abs(mu).sum() * 0.7 / np.pi ** 2
    assert np.all(np.abs(got[pick] - ref)[inside] <= tol / (1 - x[inside] ** 2))


@pytest.mark.parametrize("P", [2, 3, 7, 64, 129])
def test_cond_transform(ctx, P):
    M = np.random.default_rng(P).uniform(-1, 1, (P, P))
    got, ref = ctx.cond_transform(M), oracle.cond_transform(M)
    assert np.max(np.abs(got - ref)) <= 8 * 2 * P * EPS * 8 * np.abs(M).sum()


def test_scratch_is_reused_and_given_back(ctx):
    """Calls of growing and shrinking size on one context: the same results as on
    a fresh one."""
    mu = np.random.default_rng(0).uniform(-1, 1, 512)
    first = ctx.dos_transform(mu, 512, 1.0, 0.0)[0]
    ctx.cond_sigma(np.ones((900, 900)), np.linspace(-0.9, 0.9, 9000), 1.0, 0.0)  # past the kept size
    np.testing.assert_array_equal(ctx.dos_transform(mu, 512, 1.0, 0.0)[0], first)
    with L.Context(0) as other:
        np.testing.assert_array_equal(other.dos_transform(mu, 512, 1.0, 0.0)[0], first)
