"""FP64 form, single calls: sizes at the edges of its tiles (128 targets, 32 sources, pairs of
source tiles, k-steps of 16, runs of 64), every kernel against the oracle.  Bound: as the
other FP64 tests, 1e-12 of the row's sum of magnitudes; for Laplace the distance's rounding,
(k + 4) 2^-53 of norms about four times the distance, times the power k / 2, on both sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = [(0, dict(scal=-0.7)), (1, dict(scal=0.2, cons=0.5, powe=3.0)), (2, {}), (3, {}), (4, dict(scal=0.2, cons=0.1)),
         (5, {}), (6, dict(cons=0.25)), (7, {})]


@pytest.mark.parametrize("m,n,k", [(127, 31, 15), (128, 32, 16), (129, 33, 17), (1, 63, 31), (255, 64, 33), (257, 65, 63),
                                   (130, 95, 64), (3, 97, 65), (129, 129, 128), (128, 31, 129)])
@pytest.mark.parametrize("ktype,params", KINDS)
def test_sizes(gpu, oracle_mod, ktype, params, m, n, k):
    from ks_gb300 import gsks
    torch, O = gpu, oracle_mod
    rng = np.random.default_rng(m * n + k)
    N = 600                    # targets from the first half, sources from the second: none coincide
    X = rng.random((N, k)) * (1.0 / k ** 0.5)
    X2, w, h = O.norms(X), rng.standard_normal(N), rng.uniform(0.5, 2.0, N)
    am, bm, um, wm = (rng.permutation(300)[:q].astype(np.int32) for q in (m, n, m, n))
    bm += 300
    if ktype == 2 and k > 64:
        X *= k ** 0.5          # (the power of smaller distances leaves FP64's range)
        X2 = O.norms(X)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    d = [t(q) for q in (um, X, X2, am, bm, w, wm, h)]
    kp = dict(params, **(dict(hi=d[7], hj=d[7]) if ktype == 3 else {}))
    ko = dict(params, **(dict(hi=h, hj=h) if ktype == 3 else {}))
    u = torch.zeros(N, dtype=torch.float64, device="cuda")
    gsks.dgsks_device(gsks.make_kernel(ktype, **kp), m, n, k, u, d[0], d[1], d[2], d[3], d[1], d[2], d[4], d[5], d[6],
                      stream=torch.cuda.current_stream(), nxa=N, nxb=N)
    torch.cuda.synchronize()
    s, a = O.rows(O.make_kernel(ktype, **ko), np.arange(m, dtype=np.int32), X, X2, am, X, X2, bm, w, wm)
    assert np.all(np.abs(u.cpu().numpy()[um] - s) <= max(1e-12, k / 2 * (k + 4) * 2.0 ** -50 if ktype == 2 else 0.0) * a)
