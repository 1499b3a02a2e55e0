"""The 8-row step's forms with the number of warps left to the library, on a matrix of
more than 1M rows: every staging of the rows, 16-row blocks and the depths that 16
warps take run, in the form asked for, and agree to rounding.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def flake():
    with L.Context(0) as ctx:
        csr = ctx.build_csr(ctx.prepare(L.make_geom(model=L.MODEL_SIMPLE, size=440, max_R=650.0,
                                                    angles_deg=(0.0, 1.1), energy_rescale=10.5)))
        assert csr.n >= 1000000
        yield ctx, csr, csr.kpm_dos(L.kpm_cfg(16, R=16, seed=5))


@pytest.mark.parametrize("opts", [{"rt_stage": 0}, {"rt_stage": 0, "rt_depth": 2}, {"rt_stage": 0, "rt_depth": 4},
                                  {"rt_stage": 1}, {"rt_stage": 2}, {"rt_rows": 16}, {"rt_depth": 3}])
def test_forms_without_a_number_of_warps(flake, opts):
    ctx, csr, base = flake
    off = {"rt_stage": -1, "rt_depth": 0, "rt_rows": 0}
    try:
        for k, v in opts.items():
            ctx.set_option(k, v)
        cfg = L.kpm_cfg(16, R=16, seed=5)
        assert csr.step_kernel(cfg)[0] == 5
        got = csr.kpm_dos(cfg)
        rows = opts.get("rt_rows", 8)
        assert csr.rt_info()[0] == (csr.n + rows - 1) // rows  # ran on blocks of this height
        assert np.max(np.abs(got - base)) <= 1e-6 * np.max(np.abs(base))
    finally:
        for k, v in off.items():
            ctx.set_option(k, v)
