"""A batch, a network and a matrix may be destroyed after the context that made them (as
Python's garbage collector does); the next context works."""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


def _flake(ctx):
    return ctx.build_csr(ctx.prepare(L.make_geom(model=L.MODEL_SIMPLE, size=20, angles_deg=(0.0, 2.0), energy_rescale=10.5)))


def test_handles_destroyed_after_their_context():
    cfg = L.kpm_cfg(16, R=4, seed=1)
    for _ in range(20):
        ctx = L.Context(0)
        csr, net = _flake(ctx), L.Mlp(ctx, seed=1)
        batch = L.Batch(ctx, [csr], cfg)
        ref = batch.run()[0]
        ctx.close()
        held = [np.full(400 // 8 * k, 7, np.int64) for k in range(1, 40)]  # the context's memory, in use again
        batch.close()
        net.close()
        csr.close()
        del held
        with L.Context(0) as other:
            np.testing.assert_allclose(_flake(other).kpm_dos(cfg), ref, rtol=0, atol=1e-5 * np.abs(ref).max())
