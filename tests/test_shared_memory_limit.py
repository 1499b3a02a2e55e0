"""A kernel's limit on dynamic shared memory belongs to the device, so that contexts in
several threads share it: it is raised to the device's maximum in one place
(allow_smem) and never set to the size of one launch.
"""
import os
import threading
import time

import numpy as np
import pytest

import leo2d_gb300 as L

CSRC = os.path.join(os.path.dirname(os.path.abspath(L.__file__)), "csrc")


def test_the_limit_is_set_in_one_place():
    where = []
    for f in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, f)) as h:
            text = h.read()
        where += [f] * text.count("cudaFuncAttributeMaxDynamicSharedMemorySize")
    assert where == ["common.cuh"]


def _band(n, per_row, reach, seed):
    """Symmetric, distinct columns in a row, spectral radius below 1."""
    rng = np.random.default_rng(seed)
    i = rng.integers(0, n, n * per_row // 2)
    j = i + rng.integers(1, reach, len(i))
    key = np.unique(i[j < n] * n + j[j < n])
    i, j = key // n, key % n
    v = rng.uniform(-1, 1, len(i))
    r, c, v = np.concatenate([i, j]), np.concatenate([j, i]), np.concatenate([v, v])
    o = np.lexsort((c, r))
    r, c, v = r[o], c[o], v[o]
    return np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]), c, v / (1.01 * np.bincount(r, np.abs(v), n).max())


def _flake(ctx, sheets):
    return ctx.build_csr(ctx.prepare(L.make_geom(
        model=L.MODEL_SIMPLE, num_sheets=sheets, size=20, heights=(0.0, 3.35, 6.7)[:sheets],
        angles_deg=(0.0, 1.3, 2.6)[:sheets], energy_rescale=12.0)))


def _runs(ctx, kind):
    """Jobs of one kind with different shared memory: (prepare, run) pairs."""
    if kind == "blocks":  # block builds: tables for the largest block of a bilayer, of a trilayer
        ctx.set_option("step_kernel", 5)
        ctx.set_option("reorder", 1)
        return [lambda s=s: _flake(ctx, s).kpm_dos(L.kpm_cfg(16, R=16, block=32, seed=s)) for s in (2, 3)]
    if kind == "tiles":
        ctx.set_option("step_kernel", 0)
        mats = [ctx.upload_csr(*_band(2000, k, 90, k)) for k in (4, 60)]
        return [lambda m=m: m.kpm_dos(L.kpm_cfg(16, R=4, seed=2)) for m in mats]
    precision = L.FP64 if kind == "rows64" else L.FP32
    mats = [ctx.upload_csr(*_band(n, k, 60, n)) for n, k in ((900, 4), (900, 44), (9000, 4), (9000, 44))]
    return [lambda m=m: m.kpm_dos(L.kpm_cfg(64, R=4, seed=2, precision=precision)) for m in mats]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["rows32", "rows64", "blocks", "tiles"])
def test_threads_with_different_sizes(kind):
    """Every thread's launches find the limit they need, whatever size another thread's
    matrix takes (each thread starts at another of the jobs)."""
    with L.Context(0) as ctx:
        ref = [r() for r in _runs(ctx, kind)]
    bad, stop = [], time.monotonic() + 3.0

    def work(t):
        try:
            with L.Context(0) as ctx:
                runs = _runs(ctx, kind)
                k = t
                while time.monotonic() < stop and not bad:
                    got = runs[k % len(runs)]()
                    np.testing.assert_array_equal(got, ref[k % len(runs)])
                    k += 1
        except Exception as e:  # noqa: BLE001 - reported below
            bad.append((t, e))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
