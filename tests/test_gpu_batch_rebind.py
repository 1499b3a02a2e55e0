"""A batch stays right when other calls build its matrices' arrays again: single runs
on a member (which order it for another step kernel), local moments, FP64 runs, a
rescale, with other jobs taking the memory that those released. The replay after them
has the bits of the first.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


def _flake(ctx, size, twist):
    csr = ctx.build_csr(ctx.prepare(L.make_geom(model=L.MODEL_SIMPLE, size=size, angles_deg=(0.0, twist),
                                                energy_rescale=10.5)))
    return csr


OPTIONS = {"rows_of_8": {}, "rows_of_4": {"step_kernel": 3}, "tiles": {"reorder": 1}}


@pytest.mark.parametrize("form,block", [("rows_of_8", 0), ("rows_of_4", 32), ("tiles", 16)])
def test_replay_after_other_calls_on_its_matrices(form, block):
    with L.Context(0) as ctx:
        flakes = [_flake(ctx, s, t) for s, t in ((62, 1.4), (100, 2.0), (12, 3.0))]
        assert flakes[0].n > 8000 and flakes[1].n > 8000
        for k, v in OPTIONS[form].items():
            ctx.set_option(k, v)
        b = L.Batch(ctx, flakes, L.kpm_cfg(64, R=5, seed=3, block=block))
        for k in OPTIONS[form]:
            ctx.set_option(k, -1)
        mu = b.run()
        others = [
            lambda c: c.kpm_dos(L.kpm_cfg(128, R=4, seed=9)),
            lambda c: c.kpm_ldos(L.kpm_cfg(128), [0, 5, c.n - 1]),
            lambda c: c.kpm_dos(L.kpm_cfg(64, R=2, seed=1, precision=L.FP64)),
            lambda c: c.rescale(1.0, 0.0),
            lambda c: ctx.set_option("tile_stages", 3),
            lambda c: c.rescale(1.0, 0.0),
        ]
        keep = []
        for other in others:
            for c in flakes:
                other(c)
            keep.append(_flake(ctx, 62, 2.2))  # takes released memory of the same sizes
            keep[-1].kpm_dos(L.kpm_cfg(64, R=16, seed=2))
            np.testing.assert_array_equal(b.run(), mu)
            np.testing.assert_array_equal(b.run(), mu)
        b.close()


def test_two_batches_share_a_matrix():
    with L.Context(0) as ctx:
        flakes = [_flake(ctx, s, 1.7) for s in (62, 80, 20)]
        a = L.Batch(ctx, flakes[:2], L.kpm_cfg(64, R=5, seed=3))
        b = L.Batch(ctx, flakes[1:], L.kpm_cfg(64, R=5, seed=4, block=16))
        c = L.Batch(ctx, flakes, L.kpm_cfg(64, R=16, seed=5))
        ref = [x.run() for x in (a, b, c)]
        for _ in range(2):
            for x, mu in zip((a, b, c), ref):
                np.testing.assert_array_equal(x.run(), mu)
        for x in (a, b, c):
            x.close()
