"""The one padded pass over the rows (without stored zeros) against the count and fill
passes, which the same call takes when its padded arrays would exceed the context's
limit on one allocation: the same hoppings in the same order, so the same bits. The
structure and the values (1e-12, as in test_gpu_assembly) also against the CPU oracle.
"""
import numpy as np
import pytest

import leo2d_gb300 as L
from oracle import oracle

pytestmark = pytest.mark.gpu

REF, SIMPLE = L.MODEL_REF, L.MODEL_SIMPLE


def _build(ctx, gp, dx):
    ctx.set_profiling(True)
    try:
        csr = ctx.build_csr(gp, with_dx=dx)
        counts = [ctx.kernel_stats(k)[0] for k in ("flake_rows_count", "periodic_rows_count")]
    finally:
        ctx.set_profiling(False)
    arrays = list(csr.download(dx=dx))
    return csr, arrays, counts


# pad: entries a row has room for in the single pass. Sizes: 2k to 6k orbitals, a row a
# warp; then runs of a few rows and of the most, whose pairs share rounds (three sheets:
# pairs of both sides in one)
@pytest.mark.parametrize("pad,dx,kw", [
    (144, False, dict(model=REF, size=40, angles_deg=(0.0, 1.05))),
    (144, True, dict(model=REF, size=37, angles_deg=(0.7, -2.2), heights=(0.0, 0.4))),
    (144, False, dict(model=REF, size=40, angles_deg=(0.0, 3.0), b_field=20.0)),
    (144, True, dict(model=REF, size=40, angles_deg=(0.0, 2.0), shifts={1: (1 / 3, 1 / 3)}, e_field=0.1)),
    (224, True, dict(model=REF, num_sheets=3, size=33, heights=(0, 3.35, 6.7), angles_deg=(0, 3.0, -1.5))),
    (224, False, dict(model=REF, num_sheets=4, size=30, heights=(0, 3.35, 6.7, 10.05), angles_deg=(0, 3, -1.5, 1))),
    (144, True, dict(model=REF, size=160, angles_deg=(0.0, 2.6))),
    (144, False, dict(model=REF, size=330, angles_deg=(0.0, 2.6))),
    (224, True, dict(model=REF, num_sheets=3, size=110, heights=(0, 3.35, 6.6), angles_deg=(0, 3.0, -1.5))),
    (96, True, dict(model=SIMPLE, size=190, angles_deg=(0.0, 2.0), shifts={0: (0.2, 0.1)})),
    (96, True, dict(model=SIMPLE, size=50, angles_deg=(0.0, 2.0))),
    (256, False, dict(model=REF, boundary_condition=1, supercell_mn=(13, 12), size=47)),
    (256, False, dict(model=REF, boundary_condition=1, supercell_mn=(13, 12), size=47, k_vec=(0.01, 0.02))),
])
def test_one_pass_and_two(pad, dx, kw):
    g = L.make_geom(energy_rescale=13.0, energy_shift=0.2, **kw)
    with L.Context(0) as ctx:
        gp = ctx.prepare(g)
        a, one, counts = _build(ctx, gp, dx)
        assert counts == [0, 0]
        cap_mb = (a.n * pad * 8 - 1) >> 20
        assert a.nnz * 8 + 256 <= cap_mb << 20
        ctx.set_option("alloc_cap_mb", cap_mb)
        b, two, counts = _build(ctx, gp, dx)
        ctx.set_option("alloc_cap_mb", 0)
        assert sum(counts) == 1
        assert (a.n, a.nnz, a.n_intra, a.n_inter) == (b.n, b.nnz, b.n_intra, b.n_inter)
        if kw.get("b_field") or kw.get("k_vec"):
            one.append(a.download_imag())
            two.append(b.download_imag())
        for x, y in zip(one, two):
            assert np.array_equal(x, y)
        if kw.get("b_field") or kw.get("k_vec"):
            return
        ref = oracle.Built(gp)
    keep = (ref.val != 0) | (ref.col == np.repeat(np.arange(ref.n), np.diff(ref.rowptr)))
    exp = np.concatenate([[0], np.cumsum(np.add.reduceat(keep.astype(np.int64), ref.rowptr[:-1]))])
    assert np.array_equal(one[0], exp) and np.array_equal(one[1], ref.col[keep])
    np.testing.assert_allclose(one[2], ref.val[keep], rtol=0, atol=1e-12)
