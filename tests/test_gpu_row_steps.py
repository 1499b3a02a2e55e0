"""The multi-step row kernel (every Chebyshev step in one launch over the CSR
rows, the default where the tensor-core step does not apply) against the tiled
step and the FP64 oracle.

FP32 up to 8000 rows keeps the tiled step's FP32 arithmetic (the order of a row's
entries, the groups of rows whose dots are summed in FP32), so only the FP64 sums
over the groups differ: moments agree to 1e-13 of the largest. Larger FP32 runs
and FP64 runs sum in another order: FP32 moments agree to the step bar (2e-5 of
the largest), FP64 moments to 1e-12. Repeated runs are bit-identical.
"""
import numpy as np
import pytest

import leo2d_gb300 as L
from oracle import oracle

pytestmark = pytest.mark.gpu
ROW = 6


@pytest.fixture(scope="module")
def ctx():
    with L.Context(0) as c:
        yield c


def _random(n, per_row, seed, empty=0, wide=0):
    """Symmetric sparse matrix of spectral radius below 1; the first `empty` rows
    hold nothing and row n - 1 meets `wide` others."""
    rng = np.random.default_rng(seed)
    i = rng.integers(empty, n, n * per_row // 2)
    j = np.clip(i + rng.integers(-40, 41, len(i)), empty, n - 1)
    if wide:
        w = rng.choice(np.arange(empty, n - 1), min(wide, n - 1 - empty), replace=False)
        i, j = np.concatenate([i, np.full(len(w), n - 1)]), np.concatenate([j, w])
    v = rng.uniform(-1, 1, len(i))
    a = np.concatenate([i, j]), np.concatenate([j, i]), np.concatenate([v, v])
    o = np.lexsort((a[1], a[0]))
    r, c, v = a[0][o], a[1][o], a[2][o]
    norm = np.bincount(r, np.abs(v), n).max() if len(v) else 1.0
    return np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]), c, v / (1.01 * norm)


def _both(ctx, csr, cfg, fn=None, other=0):
    fn = fn or (lambda: csr.kpm_dos(cfg))
    got = fn()
    np.testing.assert_array_equal(got, fn())
    ctx.set_option("step_kernel", other)
    try:
        return got, fn()
    finally:
        ctx.set_option("step_kernel", -1)


def _close(got, ref, tol):
    assert np.max(np.abs(got - ref)) <= tol * np.max(np.abs(ref))


# (rows, vectors): one CTA and its edge (92 | 93 rows), rows of a warp, several
# column slices, the edge of the small form (8000 rows x slices)
@pytest.mark.parametrize("n,R", [(1, 1), (2, 3), (91, 4), (92, 4), (93, 4), (500, 8), (700, 20), (1999, 64),
                                 (2003, 64), (4001, 32), (7999, 5), (8001, 5), (12007, 12), (12007, 40)])
def test_fp32(ctx, n, R):
    csr = ctx.upload_csr(*_random(n, 24, n))
    cfg = L.kpm_cfg(384, R=R, seed=n)
    assert csr.step_kernel(cfg)[0] == ROW
    exact = n <= 8000 and R <= 32  # (wider blocks of the tiled step group their rows in another kernel shape)
    _close(*_both(ctx, csr, cfg), 1e-13 if exact else 2e-5)


@pytest.mark.parametrize("n,R", [(1, 1), (92, 4), (93, 5), (1000, 16), (7990, 2), (8010, 2), (9001, 9), (3000, 32)])
def test_fp64(ctx, n, R):
    csr = ctx.upload_csr(*_random(n, 24, n))
    _close(*_both(ctx, csr, L.kpm_cfg(64, R=R, seed=n, precision=L.FP64)), 1e-12)


@pytest.mark.parametrize("n", [60, 900, 9000])
@pytest.mark.parametrize("precision,tol", [(L.FP32, 2e-5), (L.FP64, 1e-12)])
def test_empty_and_wide_rows(ctx, n, precision, tol):
    """Rows without entries, and one that meets most others (its CTA's share
    exceeds the shared memory, or its window does not fit: other forms run)."""
    for empty, wide in ((37, 0), (5, n), (17, 40)):
        csr = ctx.upload_csr(*_random(n, 12, n + empty, empty=empty, wide=wide))
        _close(*_both(ctx, csr, L.kpm_cfg(384, R=6, seed=3, precision=precision)), tol)


@pytest.mark.parametrize("size,targets", [(12, 1), (22, 5), (40, 9), (70, 17)])
def test_flake_ldos_and_order(ctx, size, targets):
    """Local moments with and without the locality ordering, against the oracle."""
    g = L.make_geom(model=L.MODEL_SIMPLE, size=size, angles_deg=(0.0, 2.0), energy_rescale=10.5)
    csr = ctx.build_csr(ctx.prepare(g))
    t = np.arange(targets) * (csr.n // targets)
    cfg = L.kpm_cfg(384)
    got, ref = _both(ctx, csr, cfg, lambda: csr.kpm_ldos(cfg, t))
    _close(got, ref, 2e-5)
    ctx.set_option("reorder", 1)
    try:
        _close(csr.kpm_ldos(cfg, t), ref, 2e-5)
    finally:
        ctx.set_option("reorder", -1)
    if csr.n < 3000:
        rp, col, val = csr.download()
        _close(got, oracle.kpm_ldos(rp, col, val, t, 384), 1e-4)
    csr.rescale(1.3, 0.0)  # the formats go with the values
    again, ref2 = _both(ctx, csr, cfg, lambda: csr.kpm_ldos(cfg, t))
    _close(again, ref2, 2e-5)
    assert np.max(np.abs(again - got)) > 1e-3


@pytest.mark.parametrize("mn,R", [((3, 2), 2), ((4, 3), 4), ((7, 6), 9), ((12, 11), 20), ((20, 19), 16)])
def test_complex(ctx, mn, R):
    """A k point's complex matrix: the 4-row step, whose grid is a few blocks, with
    its dots reduced a warp per value."""
    g = L.make_geom(model=L.MODEL_SIMPLE, boundary_condition=1, size=3 * mn[0] + 6, supercell_mn=mn,
                    energy_rescale=10.5, k_vec=(0.05, 0.02))
    csr = ctx.build_csr(ctx.prepare(g))
    cfg = L.kpm_cfg(384, R=R, seed=4)
    _close(*_both(ctx, csr, cfg, other=3), 1e-13)
    t = [0, csr.n // 2, csr.n - 1]
    _close(*_both(ctx, csr, cfg, lambda: csr.kpm_ldos(cfg, t), other=3), 1e-13)


def test_barrier_gives_up(ctx):
    """A step barrier that waits for one arrival too many runs out, and the
    context keeps working."""
    for n in (600, 9000):
        csr = ctx.upload_csr(*_random(n, 20, n))
        cfg = L.kpm_cfg(384, R=4, seed=1)
        before = csr.kpm_dos(cfg)
        ctx.set_spin_limit(2000)
        ctx.set_option("test_unsatisfied_wait", 1)
        try:
            with pytest.raises(L.Leo2dError) as e:
                csr.kpm_dos(cfg)
            assert e.value.status == L._abi.ERR_TIMEOUT
        finally:
            ctx.set_option("test_unsatisfied_wait", 0)
            ctx.set_spin_limit(0)
        np.testing.assert_array_equal(csr.kpm_dos(cfg), before)
