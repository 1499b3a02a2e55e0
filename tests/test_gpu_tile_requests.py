"""A shape of the tiled step that the caller asks for (rows per warp slot, warps, stages,
tiles per block) reaches the tiled step: the same bits as with that step kernel named.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu
DEFAULTS = {"tile_warps": 0, "tile_stages": 2, "tile_chunk": 4, "step_kernel": -1}


@pytest.mark.parametrize("precision", [L.FP32, L.FP64])
@pytest.mark.parametrize("size,request_", [(40, {"rows_per_warp": 2}), (70, {"rows_per_warp": 4}), (40, {"tile_warps": 8}),
                                           (40, {"tile_warps": 24}), (70, {"tile_stages": 3}), (40, {"tile_chunk": 1})])
def test_the_tiled_step_runs(size, request_, precision):
    with L.Context(0) as ctx:
        csr = ctx.build_csr(ctx.prepare(L.make_geom(model=L.MODEL_SIMPLE, size=size, angles_deg=(0.0, 2.0),
                                                    energy_rescale=10.5)))
        plain = L.kpm_cfg(64, R=8, seed=3, precision=precision)
        assert csr.step_kernel(plain)[0] == 6
        cfg = L.kpm_cfg(64, R=8, seed=3, precision=precision, rows_per_warp=request_.get("rows_per_warp", 0))
        for k, v in request_.items():
            if k != "rows_per_warp":
                ctx.set_option(k, v)
        assert csr.step_kernel(cfg)[0] == 0
        ctx.reset_stats()
        got = csr.kpm_dos(cfg)
        assert ctx.kernel_stats("cheb_steps")[0] == 0 and ctx.kernel_stats("cheb_step")[0] == 32
        ctx.set_option("step_kernel", 0)
        np.testing.assert_array_equal(csr.kpm_dos(cfg), got)
        for k, v in DEFAULTS.items():
            ctx.set_option(k, v)
        assert csr.step_kernel(plain)[0] == 6
