"""Rows of a supercell in one padded pass (without stored zeros) and in the count and
fill passes (with them, or when a row overflows the padding), against the CPU oracle:
identical structure and pair counts, values to 1e-12 as in test_gpu_assembly.
"""
import numpy as np
import pytest

import leo2d_gb300 as L
from oracle import oracle

pytestmark = pytest.mark.gpu


def _compact(ref):
    keep = (ref.val != 0) | (ref.col == np.repeat(np.arange(ref.n), np.diff(ref.rowptr)))
    return keep, np.concatenate([[0], np.cumsum(np.add.reduceat(keep.astype(np.int64), ref.rowptr[:-1]))])


# the smallest cells (several images of one orbital in a row), a wider image search
# (its hoppings do not all fit the shared memory a row may hold), layers further apart
@pytest.mark.parametrize("mn,model,kw", [
    ((2, 1), L.MODEL_SIMPLE, {}), ((2, 1), L.MODEL_REF, {}), ((3, 2), L.MODEL_REF, {}),
    ((5, 4), L.MODEL_SIMPLE, {"sc_search_size": 2}), ((5, 4), L.MODEL_REF, {"sc_search_size": 2}),
    ((7, 6), L.MODEL_REF, {"heights": (0.0, 5.2)}), ((13, 12), L.MODEL_REF, {}), ((13, 12), L.MODEL_SIMPLE, {}),
])
def test_supercell_rows(mn, model, kw):
    size = 3 * max(mn) + 8
    g = L.make_geom(model=model, boundary_condition=1, supercell_mn=mn, size=size, energy_rescale=13.0,
                    energy_shift=0.2, **kw)
    with L.Context(0) as ctx:
        gp = ctx.prepare(g)
        ref = oracle.Built(gp)
        full = ctx.build_csr(gp, keep_zeros=True, with_dx=True)
        rp, col, val, dx, dy = full.download(dx=True)
        assert np.array_equal(rp, ref.rowptr) and np.array_equal(col, ref.col)
        assert (full.n_intra, full.n_inter) == (ref.n_intra, ref.n_inter)
        np.testing.assert_allclose(val, ref.val, rtol=0, atol=1e-12)
        c = ctx.build_csr(gp, with_dx=True)
        assert (c.n_intra, c.n_inter) == (ref.n_intra, ref.n_inter)
        crp, ccol, cval, cdx, cdy = c.download(dx=True)
    keep, exp = _compact(ref)
    assert np.array_equal(crp, exp) and np.array_equal(ccol, ref.col[keep])
    np.testing.assert_array_equal(cval, val[keep])
    np.testing.assert_array_equal(cdx, dx[keep])
    np.testing.assert_array_equal(cdy, dy[keep])
