"""Values beyond FP32's range, where sums that are FP64 to the caller run in pairs of FP32
numbers: a diverging recursion's moments are infinite (as in the tiled step, whose sums
are FP64), not undefined, and the network's loss is that of FP64.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


def _growing(n):
    """A diagonal matrix of 100 with small off-diagonal pairs: T_k grows by 200 a step."""
    i = np.arange(n)
    r, c = np.concatenate([i, i]), np.concatenate([i, i ^ 1])
    v = np.concatenate([np.full(n, 100.0), np.full(n, 1e-3)])
    o = np.lexsort((c, r))
    return np.arange(n + 1) * 2, c[o], v[o], np.stack([1.2 * (i % 100), 1.2 * (i // 100), 0.0 * i], 1)


# (rows: the row kernel's exact form and its panels; the 4-row and the 8-row step)
@pytest.mark.parametrize("n,options", [(600, {}), (9000, {}), (9000, {"step_kernel": 3, "reorder": 1}),
                                       (9000, {"step_kernel": 5, "reorder": 1})])
def test_diverging_moments(n, options):
    rp, col, val, pos = _growing(n)
    cfg = L.kpm_cfg(64, block=32)
    targets = [0, 1, 7, n - 1]
    with L.Context(0) as ctx:
        csr = ctx.upload_csr(rp, col, val, pos=pos)
        for k, v in options.items():
            ctx.set_option(k, v)
        got = csr.kpm_ldos(cfg, targets)
        ctx.set_option("step_kernel", 0)
        ref = csr.kpm_ldos(cfg, targets)
    # T_k^2 leaves FP32 at k = 9, T_k itself at k = 17 (what follows is undefined in every form)
    finite, beyond = np.arange(2, 16), np.arange(20, 32)
    assert np.isposinf(ref[:, beyond]).all()
    np.testing.assert_array_equal(got[:, beyond], ref[:, beyond])
    np.testing.assert_allclose(got[:, finite], ref[:, finite], rtol=1e-5)


@pytest.mark.parametrize("size", [1e25, 1e-25, 3e-17, 1.0])
@pytest.mark.parametrize("weight", [1.0, 1e-6, 1e12])
def test_loss(size, weight):
    rng = np.random.default_rng(2)
    x = rng.uniform(-1, 1, (192, 16)).astype(np.float32)
    t = (size * rng.normal(0, 1, (192, 256))).astype(np.float32)
    w = (weight * rng.uniform(0.5, 1.5, 256)).astype(np.float32)
    with L.Context(0) as ctx:
        net = L.Mlp(ctx, seed=1)
        net.set_params(np.zeros(net.n_params, np.float32))  # every output is zero
        net.set_loss_weights(w)
        loss, _ = net.grad(x, t)
        net.close()
    ref = np.sum(w.astype(np.float64) * t.astype(np.float64) ** 2) / 192
    # 49,152 terms of one sign: pairs to 2^-45 relative, FP64 sums
    assert abs(loss - ref) <= 1e-12 * ref


def test_infinite_loss():
    with L.Context(0) as ctx:
        net = L.Mlp(ctx, seed=1)
        t = np.zeros((64, 256), np.float32)
        t[3, 5] = np.inf
        assert net.grad(np.zeros((64, 16), np.float32), t)[0] == np.inf
        net.close()
