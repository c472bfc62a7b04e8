"""Asynchronous calls recorded by a capturing stream, after the thread's first call was a
synchronous or an asynchronous one, replayed on new data."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("first", ["sync", "async"])
@pytest.mark.parametrize("mode", ["thread_local", "global"])
def test_capture_after(gpu, prec, first, mode):
    from ks_gb300 import gsks
    torch, n, k = gpu, 500, 7
    ker = gsks.make_kernel(0, scal=-0.5)
    fails = []

    def work():           # a thread of its own has a context of its own
        try:
            X = torch.rand(n, k, dtype=torch.float64, device="cuda")
            X2, w = (X * X).sum(1), torch.randn(n, dtype=torch.float64, device="cuda")
            i = torch.arange(n, dtype=torch.int32, device="cuda")
            u, ref = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2))

            def enqueue(out):
                gsks.dgsks_device(ker, n, n, k, out, i, X, X2, i, X, X2, i, w, i, precision=prec,
                                  stream=torch.cuda.current_stream(), nxa=n, nxb=n)

            torch.cuda.synchronize()
            gsks.set_precision(prec)
            if first == "sync":
                assert gsks.dgsks_status(ker, ref, i, X, X2, i, X, X2, i, w, i) == 0
            else:
                enqueue(ref)
            torch.cuda.synchronize()
            g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            with torch.cuda.graph(g, stream=s, capture_error_mode=mode):
                enqueue(u)
            for _ in range(2):
                u.zero_()
                g.replay()
                torch.cuda.synchronize()
                assert torch.equal(u, ref)
                w.mul_(-3.0)
                X.add_(0.25)
                X2.copy_((X * X).sum(1))
                ref.zero_()
                torch.cuda.synchronize()
                enqueue(ref)
                torch.cuda.synchronize()
        except Exception as e:          # reported by the test's own thread
            fails.append(repr(e))

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not fails
