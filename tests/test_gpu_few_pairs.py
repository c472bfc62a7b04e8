"""Calls on either side of the sizes up to which the FP64 form takes them on the DFMA
kernels (tanh and general powers: 2^19 pairs, 16 or 8 coordinates): against the oracle, with maps,
several right-hand sides and an entry past the pool.  Bound: as the other FP64 tests,
1e-12 of the row's magnitudes.  (A negative base has no power of 2.5: NaN on both sides.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = [(4, 16, dict(cons=0.1)), (1, 8, dict(cons=9.0, powe=2.5)), (1, 8, dict(cons=1.0, powe=5.0)),
         (1, 8, dict(cons=1.0, powe=3.0)), (5, 4, {})]


@pytest.mark.parametrize("m,n", [(1, 1), (65, 63), (2048, 256), (2049, 256), (256, 2049), (75, 3000)])
@pytest.mark.parametrize("ktype,edge,params", KINDS)
@pytest.mark.parametrize("nrhs", [1, 3, 5])
def test_either_side(gpu, oracle_mod, m, n, ktype, edge, params, nrhs):
    from ks_gb300 import gsks
    torch, O = gpu, oracle_mod
    for k in (1, 3, edge, edge + 1):
        rng = np.random.default_rng(m + k)
        N = 3200
        X = rng.standard_normal((N, k)) * (0.5 / k ** 0.5 if ktype >= 5 else 1.0)
        w = rng.standard_normal((N, nrhs))
        am, bm, um, wm = (rng.permutation(N)[:q].astype(np.int32) for q in (m, n, m, n))
        good = am.copy()
        am[0], good[0] = N + 7, 0                    # past the pool: point 0, flagged
        X2 = O.norms(X)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        d = [t(q) for q in (um, X, am, bm, w, wm, X2)]
        u = torch.zeros(N, nrhs, dtype=torch.float64, device="cuda")
        par = dict(params, **(dict(scal=1.0 / k) if ktype in (1, 4) else {}))
        gsks.dgsks_device_rhs(gsks.make_kernel(ktype, **par), m, n, k, nrhs, u, d[0], d[1], d[6], d[2], d[1], d[6], d[3], d[4],
                              d[5], stream=torch.cuda.current_stream(), nxa=N, nxb=N)
        torch.cuda.synchronize()
        assert gsks.device_errors() == 1
        got = u.cpu().numpy()
        rows = np.unique(np.linspace(0, m - 1, 40).astype(np.int32))
        for r in range(nrhs):
            s, a = O.rows(O.make_kernel(ktype, **par), rows, X, X2, good, X, X2, bm, np.ascontiguousarray(w[:, r]), wm)
            v = got[um[rows], r]
            assert np.array_equal(np.isnan(v), np.isnan(s))
            assert np.all(np.isnan(s) | (np.abs(v - s) <= 1e-12 * a))
