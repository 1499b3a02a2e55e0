"""Device memory kept by a context: results do not depend on what a reused block
holds, memory goes back when a context closes, when an allocation needs it, and a
matrix may outlive its context.
"""
import threading

import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


def _job(ctx, size, seed=1):
    g = L.make_geom(model=L.MODEL_SIMPLE, size=size, angles_deg=(0.0, 2.0), energy_rescale=11.0)
    csr = ctx.build_csr(ctx.prepare(g))
    mu = csr.kpm_dos(L.kpm_cfg(64, R=4, kind=L.VEC_PHASE, precision=L.FP32, seed=seed))
    return csr, mu


def _free():
    torch = pytest.importorskip("torch")
    return torch.cuda.mem_get_info()[0]


def test_reused_blocks_give_the_same_results():
    sizes = [30, 90, 31, 60, 30, 89]
    fresh = []
    for s in sizes:
        with L.Context(0) as ctx:
            csr, mu = _job(ctx, s)
            fresh.append(mu)
            csr.close()
    with L.Context(0) as ctx:
        for s, ref in zip(sizes, fresh):
            csr, mu = _job(ctx, s)
            np.testing.assert_allclose(mu, ref, rtol=1e-6, atol=1e-6 * np.abs(ref).max())
            csr.close()


def test_closing_a_context_gives_memory_back():
    with L.Context(0) as ctx:  # loads the kernels
        _job(ctx, 60)[0].close()
    before = _free()
    with L.Context(0) as ctx:
        csr, _ = _job(ctx, 400)
        csr.close()
    assert _free() >= before - (64 << 20)


def test_matrix_outlives_its_context():
    ctx = L.Context(0)
    csr, mu = _job(ctx, 40)
    other = L.Context(0)
    rp = csr.download()[0]
    ctx.close()
    csr.close()
    again = _job(other, 40)[1]
    np.testing.assert_allclose(again, mu, rtol=1e-6, atol=1e-6 * np.abs(mu).max())
    assert rp[-1] > 0
    other.close()


def test_contexts_in_threads():
    ref = {}
    for s in (30, 45, 60):
        with L.Context(0) as ctx:
            csr, ref[s] = _job(ctx, s)
            csr.close()
    bad = []

    def work(s):
        try:
            with L.Context(0) as ctx:
                for _ in range(4):
                    csr, mu = _job(ctx, s)
                    np.testing.assert_allclose(mu, ref[s], rtol=1e-6, atol=1e-6 * np.abs(ref[s]).max())
                    csr.close()
        except Exception as e:  # noqa: BLE001 - reported below
            bad.append((s, e))

    threads = [threading.Thread(target=work, args=(s,)) for s in (30, 45, 60)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_failed_call_leaves_the_context_usable():
    with L.Context(0) as ctx:
        csr, mu = _job(ctx, 60)
        ctx.set_option("alloc_cap_mb", 1)
        with pytest.raises(L.Leo2dError, match="alloc_cap_mb"):
            _job(ctx, 200)
        ctx.set_option("alloc_cap_mb", 0)
        csr.close()
        csr, again = _job(ctx, 60)
        np.testing.assert_allclose(again, mu, rtol=1e-6, atol=1e-6 * np.abs(mu).max())
        csr.close()
