"""The multi-step row kernel where its format cannot be: windows that do not fit, rows of
very uneven length, no memory beside the matrix. The tiled step runs then, with the
bits it gives when asked for, and a search that failed is not repeated. What runs
does not depend on what ran before on the same matrix.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu
ROW = 6


@pytest.fixture()
def ctx():
    with L.Context(0) as c:
        yield c


def _symmetric(i, j, n, rng):
    key = np.unique(np.minimum(i, j)[i != j] * n + np.maximum(i, j)[i != j])
    i, j = key // n, key % n
    v = rng.uniform(-1, 1, len(i))
    r, c, v = np.concatenate([i, j]), np.concatenate([j, i]), np.concatenate([v, v])
    o = np.lexsort((c, r))
    r, c, v = r[o], c[o], v[o]
    return np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]), c, v / (1.01 * np.bincount(r, np.abs(v), n).max())


def _matrix(n, per_row, reach, seed):
    """per_row distinct columns a row on average, within `reach` of the diagonal."""
    rng = np.random.default_rng(seed)
    i = rng.integers(0, n, n * per_row // 2)
    return _symmetric(i, np.clip(i + rng.integers(-reach, reach + 1, len(i)), 0, n - 1), n, rng)


def _uneven(n, seed):
    """Four entries a row, 200 in every 16th."""
    rng = np.random.default_rng(seed)
    i = np.concatenate([rng.integers(0, n, 2 * n), np.repeat(np.arange(0, n, 16), 200)])
    return _symmetric(i, rng.integers(0, n, len(i)), n, rng)


def _tiled(ctx, run):
    ctx.set_option("step_kernel", 0)
    try:
        return run()
    finally:
        ctx.set_option("step_kernel", -1)


@pytest.mark.parametrize("n,R", [(30000, 4), (9000, 64)])
def test_wide_windows_are_searched_for_once(ctx, n, R):
    csr = ctx.upload_csr(*_matrix(n, 120, n, 3))  # (every slice of rows needs most of the vectors)
    cfg = L.kpm_cfg(64, R=R, seed=2)
    first = csr.kpm_dos(cfg)
    assert csr.step_kernel(cfg)[0] != ROW
    ctx.reset_stats()
    np.testing.assert_array_equal(csr.kpm_dos(cfg), first)
    assert ctx.kernel_stats("win_build")[0] == 0 and ctx.kernel_stats("cheb_steps")[0] == 0
    np.testing.assert_array_equal(_tiled(ctx, lambda: csr.kpm_dos(cfg)), first)
    csr.rescale(1.5, 0.0)
    assert np.max(np.abs(csr.kpm_dos(cfg) - first)) > 1e-3


def test_uneven_rows_in_fp64(ctx):
    csr = ctx.upload_csr(*_uneven(20000, 5))
    cfg = L.kpm_cfg(64, R=4, seed=2, precision=L.FP64)
    first = csr.kpm_dos(cfg)
    assert csr.step_kernel(cfg)[0] != ROW
    ctx.reset_stats()
    np.testing.assert_array_equal(csr.kpm_dos(cfg), first)
    assert ctx.kernel_stats("sell_build")[0] == 0 and ctx.kernel_stats("cheb_steps")[0] == 0
    np.testing.assert_array_equal(_tiled(ctx, lambda: csr.kpm_dos(cfg)), first)


@pytest.mark.parametrize("precision", [L.FP32, L.FP64])
def test_no_room_for_the_format(ctx, precision):
    """8 MiB an allocation: every array of the CSR matrix fits, the format's values do not."""
    rp, col, val = _matrix(30011, 30, 1250, 7)
    assert len(val) * 8 < 8 << 20
    csr = ctx.upload_csr(rp, col, val)
    cfg = L.kpm_cfg(64, R=4, seed=2, precision=precision)
    ctx.set_option("alloc_cap_mb", 8)
    ctx.reset_stats()
    got = csr.kpm_dos(cfg)
    assert ctx.kernel_stats("cheb_steps")[0] == 0
    np.testing.assert_array_equal(got, csr.kpm_dos(cfg))
    np.testing.assert_array_equal(got, _tiled(ctx, lambda: csr.kpm_dos(cfg)))
    ctx.set_option("alloc_cap_mb", 0)  # room again: the row kernel runs
    ctx.reset_stats()
    more = csr.kpm_dos(cfg)
    assert ctx.kernel_stats("cheb_steps")[0] > 0
    assert np.max(np.abs(more - got)) <= (2e-5 if precision == L.FP32 else 1e-12) * np.max(np.abs(got))


@pytest.mark.parametrize("n,precision", [(2000, L.FP32), (9000, L.FP32), (2000, L.FP64), (9000, L.FP64)])
def test_sums_of_a_run_in_small_pieces(ctx, n, precision):
    """1 MiB an allocation: the CTAs' sums of 500 steps are reduced in several pieces."""
    csr = ctx.upload_csr(*_matrix(n, 10, 40, n))
    cfg = L.kpm_cfg(1000, R=4, seed=2, precision=precision)
    ref = csr.kpm_dos(cfg)
    ctx.set_option("alloc_cap_mb", 1)
    ctx.reset_stats()
    np.testing.assert_array_equal(csr.kpm_dos(cfg), ref)
    assert ctx.kernel_stats("cheb_steps")[0] > 1


def test_a_short_run_does_not_depend_on_a_longer_one_before(ctx):
    csr = ctx.upload_csr(*_matrix(9001, 30, 60, 4))
    short, long = L.kpm_cfg(60, R=4, seed=3), L.kpm_cfg(400, R=4, seed=3)
    before = csr.kpm_dos(short)
    csr.kpm_dos(long)
    ctx.reset_stats()
    np.testing.assert_array_equal(csr.kpm_dos(short), before)
    assert ctx.kernel_stats("cheb_steps")[0] == 0
