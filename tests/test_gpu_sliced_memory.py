"""FP64 calls whose digits (12 bytes a coordinate) do not fit the device run on the kernels
that need none, and the batched and several-right-hand-sides paths of those kernels (which
also take k > 1024) are right.

The large calls name a small pool's points many times over: 12 k bytes for each of their
positions is more than the device has, everything else is a few hundred MB."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = [(0, dict(scal=-0.002)), (1, dict(scal=1e-3, cons=0.5, powe=2.0)), (4, dict(scal=1e-3, cons=0.1)),
         (6, dict(cons=0.25))]


def _too_many(torch, k):
    return int(torch.cuda.get_device_properties(0).total_memory // (12 * k)) + 4096


def _pool(torch, k, rng, n=500):
    X = rng.standard_normal((n, k)) * 0.5
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t(X), t((X * X).sum(1)), t(rng.standard_normal(4 * n))


@pytest.mark.parametrize("sync", [False, True])
@pytest.mark.parametrize("nrhs", [1, 2])
def test_single_call(gpu, sync, nrhs):
    from ks_gb300 import gsks
    torch, k, n = gpu, 1024, 3
    rng = np.random.default_rng(nrhs)
    X, X2, w = _pool(torch, k, rng)
    m = _too_many(torch, k)
    am = torch.randint(500, (m,), dtype=torch.int32, device="cuda")
    bm = torch.arange(n, dtype=torch.int32, device="cuda")
    ker = gsks.make_kernel(gsks.KS_GAUSSIAN, scal=-0.002)
    row, every = torch.arange(500, dtype=torch.int32, device="cuda"), torch.arange(m, dtype=torch.int32, device="cuda")
    ref = torch.zeros(500, nrhs, dtype=torch.float64, device="cuda")
    u = torch.zeros(m, nrhs, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    gsks.set_precision(gsks.GSKS_FP64)
    for out, a, um in ((u, am, every), (ref, row, row)):
        if sync:
            assert gsks.dgsks_rhs(ker, nrhs, out, um, X, X2, a, X, X2, bm, w, bm, k=k) == 0
        else:
            gsks.dgsks_device_rhs(ker, len(a), n, k, nrhs, out, um, X, X2, a, X, X2, bm, w, bm,
                                  stream=torch.cuda.current_stream(), nxa=500, nxb=500)
    torch.cuda.synchronize()
    assert gsks.device_errors() == 0
    # both forms: a distance within a few units of 2^-53 of its norms' sum (512 here), times scal
    assert torch.all((u - ref[am.long()]).abs() <= 2.0 ** -53 * 64 * 3 * w[:n * nrhs].abs().max())


def test_captured_call(gpu):
    from ks_gb300 import gsks
    torch, k, n = gpu, 1024, 3
    X, X2, w = _pool(torch, k, np.random.default_rng(5))
    m = _too_many(torch, k)
    am = torch.randint(500, (m,), dtype=torch.int32, device="cuda")
    bm = torch.arange(n, dtype=torch.int32, device="cuda")
    ker = gsks.make_kernel(gsks.KS_GAUSSIAN, scal=-0.002)
    ref, u = (torch.zeros(q, dtype=torch.float64, device="cuda") for q in (500, m))
    row, every = torch.arange(500, dtype=torch.int32, device="cuda"), torch.arange(m, dtype=torch.int32, device="cuda")

    def enqueue(out, um, a):
        gsks.dgsks_device(ker, len(a), n, k, out, um, X, X2, a, X, X2, bm, w, bm, stream=torch.cuda.current_stream(),
                          nxa=500, nxb=500)

    enqueue(ref, row, row)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        enqueue(u, every, am)
    g.replay()
    torch.cuda.synchronize()
    assert gsks.device_errors() == 0
    assert torch.all((u - ref[am.long()]).abs() <= 2.0 ** -53 * 64 * 3 * w[:n].abs().max())


@pytest.mark.parametrize("planned", [False, True])
def test_list(gpu, planned):
    from ks_gb300 import gsks
    torch, k = gpu, 1024
    rng = np.random.default_rng(7)
    X, X2, w = _pool(torch, k, rng)
    m = _too_many(torch, k)
    ai = torch.randint(500, (m,), dtype=torch.int32, device="cuda")
    ao = torch.tensor([0, m // 3, m], dtype=torch.int32, device="cuda")
    bo = torch.tensor([0, 2, 3], dtype=torch.int32, device="cuda")
    bi = torch.tensor([5, 6, 7], dtype=torch.int32, device="cuda")
    kers = [gsks.make_kernel(KINDS[0][0], **KINDS[0][1]), gsks.make_kernel(KINDS[1][0], **KINDS[1][1])]
    u = torch.zeros(500, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    gsks.set_precision(gsks.GSKS_FP64)
    if planned:
        plan = gsks.ListPlan(kers[0], ao, ai, bo, bi, k, 500, 500, 500, len(w), kers=kers, same_pool=True)
        plan.execute(u, X, X2, X, X2, w)
        torch.cuda.synchronize()
        assert plan.errors() == 0
        plan.close()
    else:
        gsks.dgsks_list(kers[0], u, ao, ai, bo, bi, X, X2, X, X2, w, kers=kers)
    d2 = torch.cdist(X, X[5:8], compute_mode="donot_use_mm_for_euclid_dist") ** 2
    K0 = torch.exp(-0.002 * d2[:, :2]) @ w[5:7]
    K1 = (1e-3 * (X @ X[7]) + 0.5) ** 2 * w[7]
    n0 = torch.bincount(ai[:m // 3].long(), minlength=500)
    n1 = torch.bincount(ai[m // 3:].long(), minlength=500)
    ref = n0 * K0 + n1 * K1
    # (adding m / 500 equal terms one by one: half an ulp of the sum each)
    assert torch.all((u - ref).abs() <= (2.0 ** -53 * (n0 + n1) + 1e-12) * (n0 * 2 + n1) * w[5:8].abs().max())


@pytest.mark.parametrize("nrhs", [2, 3, 4])
@pytest.mark.parametrize("ktype,params", KINDS)
def test_rhs_beyond_1024(gpu, oracle_mod, ktype, params, nrhs):
    from ks_gb300 import gsks
    torch, O, k = gpu, oracle_mod, 1025
    rng = np.random.default_rng(nrhs)
    N, m, n = 300, 130, 140
    X = rng.standard_normal((N, k)) * 0.5
    X2 = O.norms(X)
    w = rng.standard_normal((N, nrhs))
    am, bm, um, wm = (rng.permutation(N)[:q].astype(np.int32) for q in (m, n, m, n))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    d = [t(q) for q in (um, X, X2, am, bm, w, wm)]
    u = torch.zeros(N * nrhs, dtype=torch.float64, device="cuda")
    gsks.dgsks_device_rhs(gsks.make_kernel(ktype, **params), m, n, k, nrhs, u, d[0], d[1], d[2], d[3], d[1], d[2], d[4],
                          d[5], d[6], stream=torch.cuda.current_stream(), nxa=N, nxb=N)
    torch.cuda.synchronize()
    got = u.cpu().numpy().reshape(N, nrhs)
    for r in range(nrhs):
        s, a = O.rows(O.make_kernel(ktype, **params), np.arange(m, dtype=np.int32), X, X2, am, X, X2, bm,
                      np.ascontiguousarray(w[:, r]), wm)
        assert np.all(np.abs(got[um, r] - s) <= 1e-12 * a)


@pytest.mark.parametrize("planned", [False, True])
def test_list_beyond_1024(gpu, oracle_mod, planned):
    from ks_gb300 import gsks
    torch, O, k = gpu, oracle_mod, 1025
    rng = np.random.default_rng(3)
    N = 400
    X = rng.standard_normal((N, k)) * 0.5
    X2 = O.norms(X)
    w = rng.standard_normal(N)
    sizes = [(1, 1), (63, 65), (130, 140), (200, 300)]
    am, bm = ([rng.permutation(N)[:q[s]].astype(np.int32) for q in sizes] for s in (0, 1))
    off = lambda a: np.concatenate([[0], np.cumsum([len(v) for v in a])]).astype(np.int32)
    ui = np.arange(sum(q[0] for q in sizes), dtype=np.int32)
    kers = [gsks.make_kernel(t, **p) for t, p in KINDS]
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    u = torch.zeros(len(ui), dtype=torch.float64, device="cuda")
    Xd, X2d, wd, lists = t(X), t(X2), t(w), [t(off(am)), t(np.concatenate(am)), t(off(bm)), t(np.concatenate(bm))]
    uid = t(ui)
    torch.cuda.synchronize()
    gsks.set_precision(gsks.GSKS_FP64)
    if planned:
        plan = gsks.ListPlan(kers[0], *lists, k, len(ui), N, N, N, kers=kers, u_idx=uid, same_pool=True)
        plan.execute(u, Xd, X2d, Xd, X2d, wd)
        torch.cuda.synchronize()
        assert plan.errors() == 0
        plan.close()
    else:
        gsks.dgsks_list(kers[0], u, *lists, Xd, X2d, Xd, X2d, wd, kers=kers, u_idx=uid)
    got, at = u.cpu().numpy(), 0
    for (ktype, params), a, b in zip(KINDS, am, bm):
        s, c = O.rows(O.make_kernel(ktype, **params), np.arange(len(a), dtype=np.int32), X, X2, a, X, X2, b, w, b)
        assert np.all(np.abs(got[at:at + len(a)] - s) <= 1e-12 * c)
        at += len(a)
