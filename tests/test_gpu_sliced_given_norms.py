"""Norms that are not the points' own are used as given, in every pair: nearly coincident
points and pairs of small norms too, whose distances are formed from the pools otherwise.

|x|^2 + |y|^2 - 2 x.y with the given norms, in exact sums; the bound is what FP64 leaves of
such a distance: (k + 8) 2^-53 of the norms' sum, times the kernel's slope, and 2^-49 of the
value (a power of up to 19, or an exponent below 16, of a few units' error)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHANGES = {"times4": lambda n: 4.0 * n, "plus": lambda n: n + 0.5, "plus_little": lambda n: n + 1e-9, "own": lambda n: n}


def _kernel(gsks, kind, k, h):
    if kind == "varbw":
        return gsks.make_kernel(3, hi=h, hj=h)
    return {"gaussian": lambda: gsks.make_kernel(0, scal=-0.3 / k), "narrow": lambda: gsks.make_kernel(0, scal=-20.0 / k),
            "laplace": lambda: gsks.make_kernel(2), "multiquadratic": lambda: gsks.make_kernel(6, cons=0.25),
            "epanechnikov": lambda: gsks.make_kernel(7)}[kind]()


@pytest.mark.parametrize("listed", [False, True])
@pytest.mark.parametrize("change", list(CHANGES))
@pytest.mark.parametrize("kind", ["gaussian", "narrow", "varbw", "laplace", "multiquadratic", "epanechnikov"])
@pytest.mark.parametrize("k", [3, 8, 40, 100])
def test_given_norms(gpu, k, kind, change, listed):
    from ks_gb300 import gsks
    torch, n = gpu, 150
    if kind == "laplace" and k > 40:
        k = 39
    rng = np.random.default_rng(k)
    x = rng.standard_normal((n, k)) * 0.3
    x[:20] *= 1e-3                               # small norms
    x[40:50] = x[50:60] * (1 + 1e-13)            # nearly coincident
    L = np.longdouble
    d2own = ((x[:, None, :].astype(L) - x[None].astype(L)) ** 2).sum(2)
    own = (x.astype(L) ** 2).sum(1)
    x2 = CHANGES[change](own.astype(float))
    d2 = d2own + (x2.astype(L) - own)[:, None] + (x2.astype(L) - own)[None, :]
    if change == "own":
        d2 = d2own
    h = rng.uniform(0.5, 2.0, n)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    X, X2, hd = t(x), t(x2), t(h)
    ker = _kernel(gsks, kind, k, hd)
    u = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    i32 = lambda a: t(np.asarray(a, dtype=np.int32))
    ones = torch.ones(n, dtype=torch.float64, device="cuda")
    every = i32(np.arange(n))
    torch.cuda.synchronize()
    gsks.set_precision(gsks.GSKS_FP64)
    if listed:           # a task per source
        gsks.dgsks_list(ker, u, i32(np.arange(n + 1) * n), i32(np.tile(np.arange(n), n)), i32(np.arange(n + 1)), every, X,
                        X2, X, X2, ones, u_idx=i32(np.arange(n * n)))
        got = u.cpu().numpy().reshape(n, n).T
    else:                # all sources, one weight at a time
        got = np.empty((n, n))
        for j in list(range(0, n, 6)) + [45, 55]:
            w = torch.zeros(n, dtype=torch.float64, device="cuda")
            w[j] = 1.0
            v = torch.zeros(n, dtype=torch.float64, device="cuda")
            gsks.dgsks_device(ker, n, n, k, v, every, X, X2, every, X, X2, every, w, every,
                              stream=torch.cuda.current_stream(), nxa=n, nxb=n)
            torch.cuda.synchronize()
            got[:, j] = v.cpu().numpy()
    cols = np.arange(n) if listed else np.array(list(range(0, n, 6)) + [45, 55])
    got, d2 = got[:, cols], d2[:, cols]
    s2 = np.abs(x2)[:, None] + np.abs(x2)[None, cols]
    dd = (k + 8) * 2.0 ** -53 * (s2 + np.abs(own.astype(float))[:, None] + np.abs(own.astype(float))[None, cols])
    f = (d2 * 1).astype(float)
    if kind in ("gaussian", "narrow"):
        c = 0.3 / k if kind == "gaussian" else 20.0 / k
        val, slope = np.exp(L(-c) * d2), c * np.exp(-c * f)
    elif kind == "varbw":
        c = 0.5 * h[:, None] * h[None, cols]
        val, slope = np.exp(-c.astype(L) * d2), c * np.exp(-c * f)
    elif kind == "multiquadratic":
        val, slope = d2 + L(0.25), np.ones_like(f)
    elif kind == "epanechnikov":
        val, slope = np.where(d2 < 1, L(0.75) * (1 - d2), L(0.0)), np.full_like(f, 0.75)
    else:
        keep = f > 1e4 * dd + 1e-14                # away from coincidence, which is cut off at the rounding
        with np.errstate(all="ignore"):
            val = np.where(keep, L(ker.scal) * np.exp(L(ker.powe) * np.log(np.abs(d2))), 0)
            slope = np.where(keep, np.abs(ker.powe) * val.astype(float) / f, 0.0)
        got = np.where(keep, got, 0.0)
    err = np.abs((got.astype(L) - val).astype(float))
    assert np.all(err <= 1.01 * slope * dd + 2.0 ** -49 * np.abs(val.astype(float)))
