"""Panels of 4 rows in the multi-step row kernel (FP32, more than 8000 rows or a
locality-ordered matrix): ragged ends of blocks and slices, every column width,
tiles that one window cannot hold, rows without entries. Against the tiled step, to
the step bar (2e-5 of the largest moment: FP32 sums in another order).
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu
ROW = 6


def _band(n, per_row, reach, seed, empty=0):
    """Symmetric, distinct columns in a row, spectral radius below 1."""
    rng = np.random.default_rng(seed)
    i = rng.integers(empty, n, n * per_row // 2)
    j = i + rng.integers(1, reach, len(i))
    keep = j < n
    key = np.unique(i[keep] * n + j[keep])
    i, j = key // n, key % n
    v = rng.uniform(-1, 1, len(i))
    r, c, v = np.concatenate([i, j]), np.concatenate([j, i]), np.concatenate([v, v])
    o = np.lexsort((c, r))
    r, c, v = r[o], c[o], v[o]
    return (np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]), c,
            v / (1.01 * np.bincount(r, np.abs(v), n).max()))


# columns of a slice 8, 16, 32 and four slices; row counts off 4, 16 and 64; windows
# wider than one tile holds
@pytest.mark.parametrize("n,R,reach,empty", [
    (8001, 2, 40, 0), (8064, 4, 300, 0), (8065, 8, 40, 9), (9003, 16, 40, 70), (8191, 30, 900, 0),
    (12289, 64, 40, 3), (30011, 3, 2500, 0), (30000, 16, 1200, 1)])
def test_panels_match_the_tiled_step(n, R, reach, empty):
    with L.Context(0) as ctx:
        csr = ctx.upload_csr(*_band(n, 30, reach, n + R, empty))
        cfg = L.kpm_cfg(400, R=R, seed=n)
        assert csr.step_kernel(cfg)[0] == ROW
        ctx.reset_stats()
        got = csr.kpm_dos(cfg)
        assert ctx.kernel_stats("cheb_steps")[0] > 0
        np.testing.assert_array_equal(got, csr.kpm_dos(cfg))
        ctx.set_option("step_kernel", 0)
        ref = csr.kpm_dos(cfg)
    assert np.max(np.abs(got - ref)) <= 2e-5 * np.max(np.abs(ref))


def test_a_column_stored_twice_takes_another_step():
    rp, c, v = _band(9000, 30, 40, 1)
    r = np.repeat(np.arange(9000), np.diff(rp))
    e = np.flatnonzero((r == 17) & (c > 17))[0]
    o = np.argsort(np.concatenate([np.arange(len(c)), [e]]), kind="stable")
    split = v.copy()
    split[e] *= 0.25
    c2, v2 = np.concatenate([c, [c[e]]])[o], np.concatenate([split, [0.75 * v[e]]])[o]
    rp2 = rp + (np.arange(9001) > 17)
    cfg = L.kpm_cfg(400, R=4, seed=2)
    with L.Context(0) as ctx:
        one, two = ctx.upload_csr(rp, c, v), ctx.upload_csr(rp2, c2, v2)
        ref = one.kpm_dos(cfg)
        ctx.reset_stats()
        got = two.kpm_dos(cfg)
        assert ctx.kernel_stats("cheb_steps")[0] == 0
        np.testing.assert_array_equal(got, two.kpm_dos(cfg))
    assert np.max(np.abs(got - ref)) <= 2e-5 * np.max(np.abs(ref))


@pytest.mark.parametrize("P,row", [(60, False), (64, True)])
def test_short_runs(P, row):
    """From 32 steps on a run builds the windows; below it takes the tiled step."""
    with L.Context(0) as ctx:
        csr = ctx.upload_csr(*_band(9001, 30, 60, 4))
        cfg = L.kpm_cfg(P, R=4, seed=3)
        assert (csr.step_kernel(cfg)[0] == ROW) == row
        ctx.reset_stats()
        got = csr.kpm_dos(cfg)
        assert (ctx.kernel_stats("cheb_steps")[0] > 0) == row
        ctx.set_option("step_kernel", 0)
        ref = csr.kpm_dos(cfg)
    assert np.max(np.abs(got - ref)) <= 2e-5 * np.max(np.abs(ref))
