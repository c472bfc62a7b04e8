"""Map entries past the pool on the device paths of every kernel, single and batched: the
entry counts as point 0 in everything (coordinates, norms, bandwidths) and is flagged.
The arrays are longer than the pool, so that a read at the bad index would find other
values (and nothing out of bounds)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

POOL, LONG = 300, 1000
KINDS = [(0, dict(scal=-0.7)), (1, dict(scal=0.2, cons=0.5, powe=3.0)), (2, {}), (3, {}), (4, dict(scal=0.2, cons=0.1)),
         (5, {}), (6, dict(cons=0.25)), (7, {})]


def _data(torch, k, spread):
    rng = np.random.default_rng(k)
    X = rng.random((LONG, k)) * spread + (0.5 if spread < 1e-3 else 0.0)
    h = rng.uniform(0.5, 2.0, LONG)
    X[POOL:] += 7.0                       # what a read past the pool would give
    h[POOL:] = 1e8
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    am = rng.permutation(POOL)[:150].astype(np.int32)
    bm = rng.permutation(POOL)[:140].astype(np.int32)
    am[7], bm[11] = 0, 0                  # point 0 itself, on both sides
    bad_a, bad_b = am.copy(), bm.copy()
    good_a, good_b = am.copy(), bm.copy()
    for q, p in ((3, POOL), (64, POOL + 1), (149, LONG - 1)):
        bad_a[q], good_a[q] = p, 0
    for q, p in ((0, POOL), (32, LONG - 2), (139, POOL + 5)):
        bad_b[q], good_b[q] = p, 0
    w = rng.standard_normal(POOL)
    return dict(X=t(X), X2=t((X * X).sum(1)), h=t(h), w=t(w), bad=(t(bad_a), t(bad_b)), good=(t(good_a), t(good_b)))


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("spread", [1.0, 1e-8])
@pytest.mark.parametrize("k", [3, 40, 100])
@pytest.mark.parametrize("ktype,params", KINDS)
def test_single_call(gpu, ktype, params, k, spread, prec):
    from ks_gb300 import gsks
    g = _data(gpu, k, spread)
    kp = dict(params, **(dict(hi=g["h"], hj=g["h"]) if ktype == 3 else {}))
    out = {}
    for name in ("good", "bad"):
        am, bm = g[name]
        u = gpu.zeros(150, dtype=gpu.float64, device="cuda")
        gsks.dgsks_device(gsks.make_kernel(ktype, **kp), 150, 140, k, u, None, g["X"], g["X2"], am, g["X"], g["X2"], bm, g["w"],
                          None, precision=prec, nxa=POOL, nxb=POOL)
        gpu.cuda.synchronize()
        assert gsks.device_errors() == (1 if name == "bad" else 0)
        out[name] = u.cpu().numpy()
    assert np.array_equal(out["bad"], out["good"], equal_nan=True)


@pytest.mark.parametrize("spread", [1.0, 1e-8])
@pytest.mark.parametrize("k", [3, 40])
@pytest.mark.parametrize("ktype,params", KINDS)
def test_planned_list(gpu, ktype, params, k, spread):
    """Device lists that were good when the plan was made and have bad entries when it runs."""
    from ks_gb300 import gsks
    g = _data(gpu, k, spread)
    kp = dict(params, **(dict(hi=g["h"], hj=g["h"]) if ktype == 3 else {}))
    off_a, off_b = (gpu.tensor([0, n], dtype=gpu.int32, device="cuda") for n in (150, 140))
    am, bm = g["good"][0].clone(), g["good"][1].clone()
    ui = gpu.arange(150, dtype=gpu.int32, device="cuda")
    wi = gpu.arange(140, dtype=gpu.int32, device="cuda")
    plan = gsks.ListPlan(gsks.make_kernel(ktype, **kp), off_a, am, off_b, bm, k, 150, POOL, POOL, POOL, u_idx=ui, w_idx=wi,
                         same_pool=True)
    out = []
    for name in ("good", "bad"):
        am.copy_(g[name][0])
        bm.copy_(g[name][1])
        u = gpu.zeros(150, dtype=gpu.float64, device="cuda")
        gpu.cuda.synchronize()
        plan.execute(u, g["X"], g["X2"], g["X"], g["X2"], g["w"])
        gpu.cuda.synchronize()
        assert plan.errors() == (1 if name == "bad" else 0)
        out.append(u.cpu().numpy())
    plan.close()
    assert np.array_equal(out[0], out[1], equal_nan=True)
