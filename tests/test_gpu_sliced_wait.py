"""The bounded waits of the FP64 form's tensor-core kernel run out, and the library says so.

As for the split form: the producers issue nothing and the limit is 1e5 clock cycles, so
that the other roles wait for data that never comes, give up together, free their
tensor memory and return.  Synchronous calls return GSKS_ERR_TIMEOUT and leave a host u
alone, asynchronous ones set bit 1 of the error flags, and the next call is right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 3])
@pytest.mark.parametrize("k", [16, 100])
@pytest.mark.parametrize("ktype,params", [(1, dict(scal=1 / 16, cons=1.0, powe=3.0)), (0, dict(scal=-2.0))])
def test_reported_and_recovers(gpu, oracle_mod, ktype, params, k, nrhs):
    from ks_gb300 import gsks
    torch, O = gpu, oracle_mod
    rng = np.random.default_rng(k)
    N, m, n = 1000, 300, 400
    X = rng.random((N, k))
    X2 = O.norms(X)
    w = rng.standard_normal((N, nrhs))
    am, bm, um, wm = (rng.permutation(N)[:q].astype(np.int32) for q in (m, n, m, n))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    d = [t(q) for q in (um, X, X2, am, bm, w, wm)]
    ker = lambda: gsks.make_kernel(ktype, **params)

    def device(u):
        gsks.dgsks_device_rhs(ker(), m, n, k, nrhs, u, d[0], d[1], d[2], d[3], d[1], d[2], d[4], d[5], d[6],
                              precision=gsks.GSKS_FP64, stream=torch.cuda.current_stream(), nxa=N, nxb=N)
        torch.cuda.synchronize()

    gsks.set_precision(gsks.GSKS_FP64)
    assert gsks.device_errors() == 0
    gsks.split_test_wait(100_000, stall=True)
    try:
        u = np.full((N, nrhs), 7.0)
        assert gsks.dgsks_rhs(ker(), nrhs, u, um, X, X2, am, X, X2, bm, w, wm) == gsks.GSKS_ERR_TIMEOUT
        assert np.all(u == 7.0)
        device(torch.zeros(N * nrhs, dtype=torch.float64, device="cuda"))
        assert gsks.device_errors() & 2
        assert gsks.device_errors() == 0
        if nrhs == 1:
            off = np.array([0, 150, m], np.int32), np.array([0, 250, n], np.int32)
            v = np.full(N, 7.0)
            with pytest.raises(gsks.GsksError) as ex:
                gsks.dgsks_list(ker(), v, off[0], am, off[1], bm, X, X2, X, X2, np.ascontiguousarray(w[:, 0]), u_idx=um,
                                w_idx=wm)
            assert ex.value.code == gsks.GSKS_ERR_TIMEOUT
            assert np.all(v == 7.0)
    finally:
        gsks.split_test_wait(0, stall=False)

    ud = torch.zeros(N * nrhs, dtype=torch.float64, device="cuda")
    device(ud)
    assert gsks.device_errors() == 0
    got = ud.cpu().numpy().reshape(N, nrhs)
    for r in range(nrhs):
        s, a = O.rows(O.make_kernel(ktype, **params), np.arange(m, dtype=np.int32), X, X2, am, X, X2, bm,
                      np.ascontiguousarray(w[:, r]), wm)
        assert np.all(np.abs(got[um, r] - s) <= 1e-12 * a)
