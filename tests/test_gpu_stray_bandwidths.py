"""hi and hj belong to the variable-bandwidth kernel (ks.h): whatever a descriptor of
another type holds there changes no bit of the result.  The stray arrays here are device
memory of the pool's size whose values a scan for bandwidths would refuse."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = [(0, dict(scal=-0.7)), (1, dict(scal=0.2, cons=0.5, powe=3.0)), (2, {}), (4, dict(scal=0.2, cons=0.1)), (5, {}),
         (6, dict(cons=0.25)), (7, {})]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("ktype,params", KINDS)
def test_results_do_not_depend_on_them(gpu, ktype, params, prec):
    from ks_gb300 import gsks
    torch = gpu
    rng = np.random.default_rng(ktype)
    N, k, m, n = 600, 12, 300, 280
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    X = rng.random((N, k))
    Xd, X2, w, stray = t(X), t((X * X).sum(1)), t(rng.standard_normal(N)), t(np.full(N, 1e300))
    am, bm = t(rng.permutation(N)[:m].astype(np.int32)), t(rng.permutation(N)[:n].astype(np.int32))
    off_a, off_b = t(np.array([0, 100, m], np.int32)), t(np.array([0, 150, n], np.int32))
    out = []
    for h in (None, stray):
        ker = gsks.make_kernel(ktype, **params, hi=h, hj=h)
        one = torch.zeros(m, dtype=torch.float64, device="cuda")
        gsks.dgsks_device(ker, m, n, k, one, None, Xd, X2, am, Xd, X2, bm, w, bm, precision=prec, nxa=N, nxb=N)
        lst = torch.zeros(N, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        gsks.set_precision(prec)
        try:
            gsks.dgsks_list(ker, lst, off_a, am, off_b, bm, Xd, X2, Xd, X2, w)
        finally:
            gsks.set_precision(gsks.GSKS_FP64)
        out.append((one.cpu().numpy(), lst.cpu().numpy()))
    for a, b in zip(*out):
        assert np.abs(a).max() > 0
        assert np.array_equal(a, b)
