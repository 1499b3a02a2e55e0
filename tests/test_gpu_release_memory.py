"""Kept device memory goes back to the device when asked for, with contexts open, and
the context works on."""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


def test_release_memory():
    torch = pytest.importorskip("torch")

    def job(ctx):
        csr = ctx.build_csr(ctx.prepare(L.make_geom(model=L.MODEL_SIMPLE, size=400, angles_deg=(0.0, 2.0),
                                                    energy_rescale=11.0)))
        try:
            return csr.kpm_dos(L.kpm_cfg(64, R=4, seed=1)), ctx.dos_transform(np.ones(64), 64, 10.0, 0.0)[0]
        finally:
            csr.close()

    with L.Context(0) as ctx:
        first = job(ctx)
        ctx.set_option("release_memory", 1)
        free = torch.cuda.mem_get_info()[0]
        job(ctx)
        kept = free - torch.cuda.mem_get_info()[0]
        assert kept > 128 << 20  # (a job of 384k orbitals leaves some hundreds of MB)
        ctx.set_option("release_memory", 1)
        assert free - torch.cuda.mem_get_info()[0] < 32 << 20
        for a, b in zip(first, job(ctx)):
            np.testing.assert_array_equal(np.asarray(a), np.asarray(b))
        with pytest.raises(L.Leo2dError):
            ctx.set_option("release_memory", 0)
