"""Both tile widths of the BF16 tensor-core GEMM (128 x 64 below one wide tile per
SM, 128 x 256 from there) against FP64 products.

FP32 accumulation of K <= 512 products of magnitude <= 1: the error stays below
K 2^-23 in the worst order (6e-5), plus half an FP32 ulp of the result.
"""
import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


def _bf16(x):
    return (x.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)


def _back(b):
    return (b.astype(np.uint32) << 16).view(np.float32).astype(np.float64)


@pytest.mark.parametrize("M,N,K", [
    (1, 1, 8), (127, 63, 64), (129, 65, 72), (128, 256, 512), (8192, 256, 256), (1000, 300, 128),
    (19456, 256, 64), (19457, 257, 64), (40000, 70, 136)])
def test_tile_widths(M, N, K):
    rng = np.random.default_rng(M + N + K)
    a, b = _bf16(rng.uniform(-1, 1, (M, K))), _bf16(rng.uniform(-1, 1, (N, K)))
    with L.Context(0) as ctx:
        d = ctx.tc_gemm(a, b)
    ref = _back(a) @ _back(b).T
    assert np.max(np.abs(d - ref)) <= K * 2.0**-23 + 2.0**-24 * np.max(np.abs(ref))


@pytest.mark.parametrize("n", [64, 320, 9600, 20480])
def test_gradient_of_odd_batches(n):
    """Blocks, splits and tile widths of the gradient at batches off the powers of
    two, by linearity: the gradient over a batch is the mean of those over its
    quarters (BF16 roundings of dZ scale with the batch by powers of two only when
    the counts do, so 2^-8 of the norm is allowed)."""
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 16)).astype(np.float32)
    t = rng.normal(0, 0.3, (n, 256)).astype(np.float32)
    with L.Context(0) as ctx:
        net = L.Mlp(ctx, seed=3)
        loss, g = net.grad(x, t)
        parts = [net.grad(x[i:i + 64], t[i:i + 64]) for i in range(0, n, 64)] if n <= 320 else \
            [net.grad(x[i:i + n // 5], t[i:i + n // 5]) for i in range(0, n, n // 5)]
        net.close()
    assert abs(loss - np.mean([p[0] for p in parts])) <= 1e-9 * loss
    ref = np.mean([p[1].astype(np.float64) for p in parts], axis=0)
    assert np.linalg.norm(g - ref) <= 2.0**-8 * np.linalg.norm(ref)


# output tiles 1, 2 x 1 and 3 x 2 of the FP32 product; K = 32 n: one range, several,
# more than a wave of them; B sides of part of a tile
@pytest.mark.parametrize("size,M,chunk", [(3, 8, 4), (12, 132, 68), (40, 20, 0), (70, 260, 256), (70, 300, 0)])
def test_k_ranges_of_the_moment_product(size, M, chunk):
    """Moments of the Kubo trace against the FP64 oracle, to the trace's FP32 bar."""
    from oracle import oracle
    R, seed = 2, 8
    with L.Context(0) as ctx:
        g = L.make_geom(model=L.MODEL_SIMPLE, size=size, angles_deg=(0.0, 2.0), energy_rescale=10.5)
        csr = ctx.build_csr(ctx.prepare(g), with_dx=True)
        rp, col, val, dx, _ = csr.download(dx=True)
        cfg = L.kpm_cfg(M, R=R, kind=L.VEC_PHASE, seed=seed)
        ctx.set_option("kubo_chunk", chunk)
        mu = csr.kpm_cond(cfg)
        np.testing.assert_array_equal(mu, csr.kpm_cond(cfg))
        re, im = oracle.phase_vectors(seed, 0, R, csr.n)
    ref = (oracle.kpm_cond_trace(rp, col, val, dx, re, M) + oracle.kpm_cond_trace(rp, col, val, dx, im, M)) / R
    assert np.max(np.abs(mu - ref)) <= 1e-4 * np.max(np.abs(ref))
