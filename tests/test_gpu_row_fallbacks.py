"""The multi-step row kernel: what runs does not depend on what ran before on the same
matrix.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


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


def test_a_short_run_does_not_depend_on_a_longer_one_before(ctx):
    csr = ctx.upload_csr(*_matrix(9001, 30, 60, 4))
    short, long = L.kpm_cfg(60, R=4, seed=3), L.kpm_cfg(400, R=4, seed=3)
    before = csr.kpm_dos(short)
    csr.kpm_dos(long)
    ctx.reset_stats()
    np.testing.assert_array_equal(csr.kpm_dos(short), before)
    assert ctx.kernel_stats("cheb_steps")[0] == 0
