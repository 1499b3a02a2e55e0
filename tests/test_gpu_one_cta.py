"""Every step of a small complex matrix in one launch of one CTA against the step of
a launch each: the same FP32 arithmetic, so the moments agree to 1e-13 of the largest
(FP64 sums alone differ). Matrices on both sides of what one CTA's memory holds.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mn", [(2, 1), (3, 2), (4, 3), (5, 4), (6, 5)])
@pytest.mark.parametrize("model", [L.MODEL_SIMPLE, L.MODEL_REF])
@pytest.mark.parametrize("P,R", [(4, 1), (64, 16), (402 // 4 * 4, 7), (128, 33)])
def test_matches_single_steps(mn, model, P, R):
    g = L.make_geom(model=model, boundary_condition=1, size=3 * mn[0] + 6, supercell_mn=mn, energy_rescale=13.0,
                    k_vec=(0.05, -0.03))
    with L.Context(0) as ctx:
        csr = ctx.build_csr(ctx.prepare(g))
        cfg = L.kpm_cfg(P, R=R, seed=P)
        t = [0, csr.n // 3, csr.n - 1]
        ctx.reset_stats()
        got, loc = csr.kpm_dos(cfg), csr.kpm_ldos(cfg, t)
        one = ctx.kernel_stats("cheb_steps")[0]
        assert one > 0 if mn[0] <= 3 else one >= 0
        np.testing.assert_array_equal(got, csr.kpm_dos(cfg))
        ctx.set_option("step_kernel", 3)
        ref, lref = csr.kpm_dos(cfg), csr.kpm_ldos(cfg, t)
        assert ctx.kernel_stats("cheb_step")[0] > 0
    assert np.max(np.abs(got - ref)) <= 1e-13 * np.max(np.abs(ref))
    assert np.max(np.abs(loc - lref)) <= 1e-13 * np.max(np.abs(lref))
