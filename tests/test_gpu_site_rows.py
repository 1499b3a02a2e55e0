"""The network's sum over all sites: features from fixed-point phases in FP32
pairs, chunks of sites through one work space.

The sum is compared with the network's outputs on the FP64 features of the same
sites (predict on site_features). Both round the features to BF16; a value whose
two forms straddle a rounding boundary differs by one BF16 step. The forms agree
to 2^-24, so about one value in 2^14 may: a relative change of the sum far below
the 1e-6 of the sum of magnitudes allowed here.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


def _expected(net, x):
    s, a = np.zeros(256), np.zeros(256)
    for r in range(0, len(x), 200_000):
        y = net.predict(x[r:r + 200_000]).astype(np.float64)
        s += y.sum(axis=0)
        a += np.abs(y).sum(axis=0)
    return s, a


# sizes: a handful of sites, odd counts, more sites than one chunk (2M)
@pytest.mark.parametrize("size,theta", [(4, 0.0), (30, -1.3), (301, 7.0), (1000, 1.05)])
@pytest.mark.parametrize("fused", [1, 0])
def test_site_sum_matches_predict(size, theta, fused):
    with L.Context(0) as ctx:
        ctx.set_option("mlp_fused", fused)
        g = L.make_geom(model=L.MODEL_SIMPLE, size=size, angles_deg=(0.3, 0.3 + theta), energy_rescale=1.0)
        csr = ctx.build_csr(ctx.prepare(g))
        if size == 1000:
            assert csr.n > 2_000_000
        net = L.Mlp(ctx, seed=5)
        s, a = _expected(net, csr.site_features(theta))
        got = net.site_sum(csr, theta)
        np.testing.assert_array_less(np.abs(got - s), 1e-6 * a + 1e-12)
        np.testing.assert_array_equal(got, net.site_sum(csr, theta))  # fixed order
        net.close()


def test_site_sum_respects_the_allocation_cap():
    with L.Context(0) as ctx:
        g = L.make_geom(model=L.MODEL_SIMPLE, size=400, angles_deg=(0.0, 1.05), energy_rescale=1.0)
        csr = ctx.build_csr(ctx.prepare(g))
        net = L.Mlp(ctx, seed=5)
        ref = net.site_sum(csr, 1.05)
        ctx.set_option("alloc_cap_mb", 1)
        with pytest.raises(L.Leo2dError, match="alloc_cap_mb"):
            net.site_sum(csr, 1.05)
        ctx.set_option("alloc_cap_mb", 0)
        np.testing.assert_array_equal(ref, net.site_sum(csr, 1.05))
        net.close()
