"""Allocation-free traces on two streams of a device share one scratch array: the second
call's work waits for the first one's, whichever stream and thread it comes from."""
import ctypes
import threading

import numpy as np
import pytest

import leo2d_gb300 as L

pytestmark = pytest.mark.gpu


def test_calls_on_two_streams():
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda:0")
    with L.Context(0) as ctx:
        csr = ctx.build_csr(ctx.prepare(L.make_geom(model=L.MODEL_SIMPLE, size=60, angles_deg=(0.0, 2.0),
                                                    energy_rescale=10.5)))
        rp, col, val = csr.download()[:3]
        d = [torch.from_numpy(a).to(dev) for a in (rp, col, val.astype(np.float32))]
        P, R = 64, 20

        def call(seed, out, stream):
            st = ctx.lib.leo2d_kpm_dos_noalloc(*(ctypes.c_void_p(a.data_ptr()) for a in d), csr.n, P, R, seed, 0,
                                               ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(stream.cuda_stream))
            assert st == 0

        ref = []
        for seed in range(6):
            out = torch.empty((R, P), dtype=torch.float64, device=dev)
            call(seed, out, torch.cuda.current_stream(dev))
            torch.cuda.synchronize()
            ref.append(out.cpu().numpy())
        streams = [torch.cuda.Stream(dev) for _ in range(3)]
        outs = [torch.empty((R, P), dtype=torch.float64, device=dev) for _ in range(24)]
        torch.cuda.synchronize()
        for k, out in enumerate(outs[:12]):  # one thread, several streams
            call(k % 6, out, streams[k % 3])

        def work(t):
            for k in range(12 + t, 24, 3):
                call(k % 6, outs[k], streams[t])

        threads = [threading.Thread(target=work, args=(t,)) for t in range(3)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        for k, out in enumerate(outs):
            np.testing.assert_array_equal(out.cpu().numpy(), ref[k % 6])
        # captured: no wait for work outside the graph
        graph, out = torch.cuda.CUDAGraph(), torch.empty((R, P), dtype=torch.float64, device=dev)
        with torch.cuda.graph(graph):
            call(2, out, torch.cuda.current_stream(dev))
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), ref[2])
