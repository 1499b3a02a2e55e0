"""Processing order and epilogue staging of the tensor-core row-block step.

The blocks after the last whole round are dealt evenly over the warps, and the
epilogue's rows are staged in shared memory per block: sizes with fewer blocks
than warps, exactly one round, one block more or less than a round, blocks
shorter than the copy pipeline, and a ragged last block. The order changes the
dot sums only, so the moments match the gather kernel's to the FP32 step bar
(2e-5 of the largest) and repeat bit for bit.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with L.Context(0) as c:
        yield c


def _band(n, half, seed):
    """Symmetric band matrix on a line of sites (rows of at most 2 half + 1 entries)."""
    rng = np.random.default_rng(seed)
    d = rng.uniform(-1, 1, (n, half + 1)) / (2 * half + 1)
    rp, col, val = [0], [], []
    for i in range(n):
        for j in range(max(0, i - half), min(n, i + half + 1)):
            col.append(j)
            val.append(d[min(i, j), abs(i - j)])
        rp.append(len(col))
    pos = np.stack([2.5 * np.arange(n), np.zeros(n), np.zeros(n)], 1)
    return np.array(rp), np.array(col), np.array(val), pos


@pytest.mark.parametrize("warps,rows", [(16, 8), (20, 8), (12, 16), (16, 16)])
@pytest.mark.parametrize("n", [5, 8 * 19 + 3, 8 * 20 * 4, 8 * 20 * 4 + 1, 8 * 16 * 152 - 7, 8 * 16 * 152 * 2 + 9])
def test_order_and_epilogue(ctx, n, warps, rows):
    half = 1 if n > 2000 else 3  # short rows: blocks of one or two k-steps
    csr = ctx.upload_csr(*_band(n, half, n)[:3], pos=_band(n, half, n)[3])
    cfg = L.kpm_cfg(16, R=16, seed=9, block=32)
    opts = {"reorder": 1, "rt_warps": warps, "rt_rows": rows, "rt_depth": 3, "rt_stage": 1}
    try:
        for k, v in opts.items():
            ctx.set_option(k, v)
        ctx.set_option("step_kernel", 0)
        ref = csr.kpm_dos(cfg)
        ctx.set_option("step_kernel", 5)
        got = csr.kpm_dos(cfg)
        assert csr.rt_info()[0] == (n + rows - 1) // rows
        np.testing.assert_array_equal(got, csr.kpm_dos(cfg))
    finally:
        for k, v in {"reorder": -1, "rt_warps": 0, "rt_rows": 0, "rt_depth": 0, "rt_stage": -1, "step_kernel": -1}.items():
            ctx.set_option(k, v)
    assert np.max(np.abs(got - ref)) < 2e-5 * np.max(np.abs(ref))
