"""The limit on one allocation (alloc_cap_mb) holds for each array of a call by itself: work
space that a call takes in one piece, or in larger pieces for speed, does not make it
fail where every array that it needs is within the limit.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    with L.Context(0) as c:
        yield c


def _limited(ctx, mb, run):
    ref = run()
    ctx.set_option("alloc_cap_mb", mb)
    try:
        return ref, run()
    finally:
        ctx.set_option("alloc_cap_mb", 0)


@pytest.mark.parametrize("P,sets", [(20000, 1), (40000, 1), (4000, 32)])  # (40000: the cosine table alone is 1.28 MB)
def test_density_transform(ctx, P, sets):
    mu = np.random.default_rng(P).normal(0, 1, (sets, P)) / np.arange(1, P + 1)
    (a, _), (b, _) = _limited(ctx, 1, lambda: ctx.dos_transform(mu, P, 10.0, 0.5))
    # (cosines to 2 ulp either way, P of them in FP64)
    assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(a)) * np.sqrt(P)


def test_reconstruction(ctx):
    mu = np.random.default_rng(1).normal(0, 1, 500)
    E = np.linspace(-9.9, 9.9, 100000)
    a, b = _limited(ctx, 1, lambda: ctx.dos_reconstruct(mu, E, 10.0, 0.0))
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("M,energies", [(300, 2001), (8, 50000), (360, 40000)])
def test_conductivity(ctx, M, energies):
    mu = np.random.default_rng(M).normal(0, 1, (M, M))
    E = np.linspace(-9.9, 9.9, energies)
    a, b = _limited(ctx, 1, lambda: ctx.cond_sigma(mu, E, 10.0, 0.0))
    assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(a))


@pytest.mark.parametrize("fused", [1, 0])
def test_site_sum(ctx, fused):
    csr = ctx.build_csr(ctx.prepare(L.make_geom(model=L.MODEL_SIMPLE, size=57, angles_deg=(0.0, 2.0),
                                                energy_rescale=10.5)))
    assert 7000 < csr.n < 8000
    net = L.Mlp(ctx, seed=3)
    ctx.set_option("mlp_fused", fused)
    a, b = _limited(ctx, 1 if fused else 8, lambda: net.site_sum(csr, 2.0))
    np.testing.assert_array_equal(a, b)


def test_kubo_moments(ctx):
    """The FP64 tiles of the moment product's K ranges: one for each SM would take 40 MB, the
    T_n vectors 20."""
    csr = ctx.build_csr(ctx.prepare(L.make_geom(model=L.MODEL_SIMPLE, size=66, max_R=63.0, angles_deg=(0.0, 2.0),
                                                energy_rescale=10.5)))
    assert 9300 < csr.n <= 9728  # (64 k-blocks of 32 products a range)
    ctx.set_option("reorder", 1)
    ctx.set_option("kubo_chunk", 4)
    a, b = _limited(ctx, 24, lambda: csr.kpm_cond(L.kpm_cfg(16, R=16, seed=3)))
    # the FP32 sums do not depend on the K ranges, which FP64 adds up
    assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(a))
