"""The FP64 form on the tensor cores: digits of the coordinates multiplied exactly,
kernel values in FP64 or 64-bit integers.  Compared with the CPU oracle at the edges
of the tiles (128 targets, 64 sources), of the k layouts (16-wide steps, resident up
to 64, streamed up to 1024, DFMA beyond) and of the operand format (points with
exponents the digits cannot hold, coincident points, one row far smaller than the
others), and with the DFMA kernels (gsks_dgsks_device_noalloc).

Tolerance: both sides round in FP64.  An inner product of k terms carries at most
about (k + 4) 2^-53 of the sum of the two norms, the kernel function turns an error of
its argument into at most `slope` times that relative to its value, and the function
and the row's sum add a few 2^-53 more; twice that bounds the difference of two such
evaluations, relative to sum_j |K_ij w_j|."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _case(seed, N, k, m, n, scale=1.0, dup=0):
    rng = np.random.default_rng(seed)
    X = rng.random((N, k)) * scale
    if dup:
        X[N - dup:] = X[:dup]
    return dict(X=X, w=rng.standard_normal((N, 4)), amap=rng.permutation(N)[:m].astype(np.int32),
                bmap=rng.permutation(N)[:n].astype(np.int32), umap=rng.permutation(N)[:m].astype(np.int32),
                wmap=rng.permutation(N)[:n].astype(np.int32), h=1.0 / (scale * rng.uniform(0.5, 3.0, N)))


def _run(torch, gsks, ktype, params, g, nrhs=1, noalloc=False):
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    X, m, n = t(g["X"]), g["amap"].size, g["bmap"].size
    N, k = g["X"].shape
    kp = dict(params)
    h = t(g["h"])
    if ktype == 3:
        kp.update(hi=h, hj=h)
    ker = gsks.make_kernel(ktype, **kp)
    X2, w = t(g["X2"]), t(g["w"][:, :nrhs])
    maps = [t(g[q]) for q in ("umap", "amap", "bmap", "wmap")]
    u = torch.zeros(N * nrhs, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    if noalloc:
        p = lambda x: C.c_void_p(x.data_ptr())
        rc = gsks.load().gsks_dgsks_device_noalloc(C.byref(ker), m, n, k, p(u), p(maps[0]), p(X), p(X2), p(maps[1]),
                                                   p(X), p(X2), p(maps[2]), p(w), p(maps[3]), C.c_void_p(0))
        assert rc == 0
    else:
        gsks.dgsks_device_rhs(ker, m, n, k, nrhs, u, maps[0], X, X2, maps[1], X, X2, maps[2], w, maps[3], nxa=N, nxb=N)
    torch.cuda.synchronize()
    assert gsks.device_errors() == 0
    return u.cpu().numpy().reshape(N, nrhs)


def _slope(ktype, params, g, k):
    """|d log K / d argument| x the rounding of the argument per 2^-53, for the points of g."""
    s = 2.0 * float(g["X2"].max())
    if ktype == 0:
        return abs(params["scal"]) * s
    if ktype == 3:
        return 0.5 * float(g["h"].max()) ** 2 * s
    if ktype == 2:                       # d2 of the nearest distinct points of the call
        X = g["X"]
        A, B = X[g["amap"]], X[g["bmap"]]
        d2 = min(float(np.min(d, initial=1e300, where=d > 0)) for d in (((B - a) ** 2).sum(1) for a in A))
        return 0.5 * k * s / d2
    return 4.0 * max(1.0, s) * max(1.0, abs(params.get("scal", 1.0)))


def _check(O, u, ktype, params, g, nrhs=1):
    N, k = g["X"].shape
    kp = dict(params)
    if ktype == 3:
        kp.update(hi=g["h"], hj=g["h"])
    m = g["amap"].size
    tol = 2.0 * EPS * ((k + 4) * _slope(ktype, params, g, k) + 64 + 2 * k)
    for r in range(nrhs):
        s, a = O.rows(O.make_kernel(ktype, **kp), np.arange(m, dtype=np.int32), g["X"], g["X2"], g["amap"], g["X"],
                      g["X2"], g["bmap"], np.ascontiguousarray(g["w"][:, r]), g["wmap"])
        err = np.abs(u[g["umap"], r] - s)
        assert np.all(err <= tol * a), (r, float((err / a).max()), tol)


KINDS = [(0, dict(scal=-1.5)), (1, dict(scal=0.3, cons=0.5, powe=3.0)), (2, {}), (3, {}), (4, dict(scal=0.2, cons=0.1)),
         (5, {}), (6, dict(cons=0.25)), (7, {})]


def _params(ktype, params, k):
    """scaled so that the kernel's argument stays of order one for any k"""
    p = dict(params)
    if ktype == 0:
        p["scal"] = -1.5 * 6.0 / k
    if ktype in (1, 4):
        p["scal"] = 1.0 / k
    return p


@pytest.mark.parametrize("k", [3, 15, 16, 17, 64, 65, 200, 1024, 1025])
@pytest.mark.parametrize("ktype,params", KINDS)
def test_kernels_over_k(gpu, oracle_mod, ktype, params, k):
    from ks_gb300 import gsks
    if ktype == 2 and k > 300:
        pytest.skip("the Laplace constant leaves the FP64 range")
    g = _case(k, 400, k, 130, 197, scale=(6.0 / k) ** 0.5)
    g["X2"] = oracle_mod.norms(g["X"])
    p = _params(ktype, params, 6) if ktype in (0, 1, 4) else dict(params)
    _check(oracle_mod, _run(gpu, gsks, ktype, p, g), ktype, p, g)


@pytest.mark.parametrize("m,n", [(1, 1), (127, 63), (128, 64), (129, 65), (1, 5000), (3000, 1), (2500, 2700)])
@pytest.mark.parametrize("ktype,params", KINDS[:4])
def test_tile_edges(gpu, oracle_mod, ktype, params, m, n):
    from ks_gb300 import gsks
    g = _case(m + n, 6000, 9, m, n)
    g["X2"] = oracle_mod.norms(g["X"])
    p = _params(ktype, params, 9)
    _check(oracle_mod, _run(gpu, gsks, ktype, p, g), ktype, p, g)


@pytest.mark.parametrize("nrhs", [2, 3, 4])
@pytest.mark.parametrize("k", [12, 100])
def test_right_hand_sides(gpu, oracle_mod, nrhs, k):
    from ks_gb300 import gsks
    g = _case(nrhs, 700, k, 300, 333)
    g["X2"] = oracle_mod.norms(g["X"])
    for ktype, params in KINDS[:4]:
        p = _params(ktype, params, k)
        _check(oracle_mod, _run(gpu, gsks, ktype, p, g, nrhs), ktype, p, g, nrhs)


@pytest.mark.parametrize("ktype,params", [(0, dict(scal=-800.0)), (0, dict(scal=-1e-3)), (0, dict(scal=0.05)), (3, {})])
def test_gaussian_ranges(gpu, oracle_mod, ktype, params):
    """Narrow (values down to and below the normal range), wide and growing exponentials;
    coincident points under a narrow kernel keep the value 1 to the last bit."""
    from ks_gb300 import gsks
    g = _case(3, 900, 8, 500, 600, dup=300)
    if ktype == 3:
        g["h"] = g["h"] * 60.0
    g["X2"] = oracle_mod.norms(g["X"])
    _check(oracle_mod, _run(gpu, gsks, ktype, params, g), ktype, params, g)


@pytest.mark.parametrize("ktype,params", [(0, dict(scal=-2.0)), (1, dict(scal=1.0, cons=0.0, powe=2.0)), (6, dict(cons=0.0))])
def test_points_of_very_different_size(gpu, oracle_mod, ktype, params):
    """Rows from 2^-40 to 2^20 of each other's size, zero rows, and coordinates whose
    exponents the digits do not hold (2^-600): the DFMA kernels are the reference."""
    from ks_gb300 import gsks
    g = _case(11, 500, 20, 260, 270)
    g["X"] *= 2.0 ** np.linspace(-40, 4 if ktype == 0 else 20, 500)[:, None]
    g["X"][::50] = 0.0
    g["X"][7] *= 2.0 ** -560
    g["X2"] = oracle_mod.norms(g["X"])
    gsks.load().gsks_dgsks_device_noalloc.restype = C.c_int
    u, ref = _run(gpu, gsks, ktype, params, g), _run(gpu, gsks, ktype, params, g, noalloc=True)
    kp = dict(params)
    s, a = oracle_mod.rows(oracle_mod.make_kernel(ktype, **kp), np.arange(260, dtype=np.int32), g["X"], g["X2"], g["amap"],
                           g["X"], g["X2"], g["bmap"], np.ascontiguousarray(g["w"][:, 0]), g["wmap"])
    tol = 2.0 * EPS * ((20 + 4) * max(4.0, abs(params.get("scal", 1.0)) * 2.0 * float(g["X2"].max()) if ktype == 0 else 4.0) + 128)
    err = np.abs(u[g["umap"], 0] - ref[g["umap"], 0])
    assert np.all(err <= tol * a), float((err / np.maximum(a, 1e-300)).max())


def test_infinite_and_nan_coordinates(gpu):
    """A point with an infinite or NaN coordinate gives what the DFMA kernels give."""
    from ks_gb300 import gsks
    g = _case(5, 300, 10, 140, 150)
    g["X"][g["amap"][3], 2] = np.inf
    g["X"][g["bmap"][9], 4] = np.nan
    g["X2"] = (g["X"] ** 2).sum(1)
    gsks.load().gsks_dgsks_device_noalloc.restype = C.c_int
    for ktype, params in [(0, dict(scal=-1.0)), (1, dict(scal=0.1, cons=1.0, powe=2.0)), (5, {}), (6, dict(cons=1.0))]:
        u, ref = _run(gpu, gsks, ktype, params, g), _run(gpu, gsks, ktype, params, g, noalloc=True)
        np.testing.assert_allclose(u, ref, rtol=1e-10, atol=1e-12)


@pytest.mark.parametrize("k", [3, 16, 33, 64, 65, 200])
def test_lists_of_all_kernels(gpu, oracle_mod, k):
    """A batch of tasks of every kernel type, of sizes around the tiles and the source
    chunk (1024), empty ones among them; shared u entries add up."""
    from ks_gb300 import gsks
    O = oracle_mod
    rng = np.random.default_rng(k)
    N = 3000
    X = rng.random((N, k)) * (6.0 / k) ** 0.5
    g = dict(X=X, X2=O.norms(X), w=rng.standard_normal((N, 1)), h=rng.uniform(0.5, 2.0, N))
    sizes = [(1, 1), (127, 31), (128, 32), (129, 33), (0, 40), (40, 0), (300, 1100), (64, 1024), (200, 1025), (5, 2500)]
    tasks = []
    for t in range(2 * len(sizes)):
        ktype, params = KINDS[t % len(KINDS)]
        if ktype == 2 and k < 3:
            continue
        m, n = sizes[t % len(sizes)]
        p = _params(ktype, params, 6) if ktype in (0, 1, 4) else dict(params)
        tasks.append((ktype, p, rng.choice(N, m, replace=False).astype(np.int32), rng.choice(N, n, replace=False).astype(np.int32)))
    a_off = np.cumsum([0] + [len(t[2]) for t in tasks]).astype(np.int32)
    b_off = np.cumsum([0] + [len(t[3]) for t in tasks]).astype(np.int32)
    a_idx = np.concatenate([t[2] for t in tasks]).astype(np.int32)
    b_idx = np.concatenate([t[3] for t in tasks]).astype(np.int32)
    kers = [gsks.make_kernel(t[0], **t[1], **(dict(hi=g["h"], hj=g["h"]) if t[0] == 3 else {})) for t in tasks]
    u = np.zeros(N)
    gsks.set_precision(gsks.GSKS_FP64)
    gsks.dgsks_list(kers[0], u, a_off, a_idx, b_off, b_idx, X, g["X2"], X, g["X2"], np.ascontiguousarray(g["w"][:, 0]),
                    kers=kers)
    ref, bound = np.zeros(N), np.zeros(N)
    for ktype, p, a, b in tasks:
        if not len(a) or not len(b):
            continue
        kp = dict(p, **(dict(hi=g["h"], hj=g["h"]) if ktype == 3 else {}))
        s, c = O.rows(O.make_kernel(ktype, **kp), np.arange(len(a), dtype=np.int32), X, g["X2"], a, X, g["X2"], b,
                      np.ascontiguousarray(g["w"][:, 0]), b)
        ref[a] += s
        gg = dict(g, amap=a, bmap=b)
        bound[a] += 2.0 * EPS * ((k + 4) * _slope(ktype, p, gg, k) + 64 + 2 * k) * c
    assert np.all(np.abs(u - ref) <= bound + 32 * EPS * np.abs(ref))
