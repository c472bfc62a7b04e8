"""The integer exponential and power of the FP64 form are not biased: signed errors of 4096
pairs' values, in units of 2^-53 of the value.

Points on a grid of 2^-20, so that norms and distances are exact and what is measured is
the function.  Just below 1 (wide Gaussians) a value's own rounding is rms 0.29 and the
evaluation's mean below 0.1: bounds 0.45 and 0.15.  A power P / 2 of the distance has its
exponent's error, P 2^-58 rms, besides: bounds 0.8 + 0.08 P, and for the mean five standard
errors of 4096 samples and P / 100 more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["gaussian", "varbw", "laplace"])
@pytest.mark.parametrize("listed", [False, True])
@pytest.mark.parametrize("k", [3, 8, 40, 100])
def test_mean_error(gpu, k, listed, kind):
    from ks_gb300 import gsks
    torch, m = gpu, 4096
    rng = np.random.default_rng(k)
    x = np.floor((0.5 + 0.5 * rng.random((m + 1, k))) * 2.0 ** 20) * 2.0 ** -20
    scal = -(2.0 ** -14) / k
    X = torch.from_numpy(x).cuda()
    X2 = torch.from_numpy((x * x).sum(1)).cuda()
    h = torch.full((m + 1,), float(np.sqrt(-2.0 * scal)), dtype=torch.float64, device="cuda")
    ker = {"gaussian": lambda: gsks.make_kernel(0, scal=scal), "varbw": lambda: gsks.make_kernel(3, hi=h, hj=h),
           "laplace": lambda: gsks.make_kernel(2)}[kind]()
    i32 = lambda a: torch.from_numpy(np.asarray(a, dtype=np.int32)).cuda()
    am, bm, one = i32(np.arange(m)), i32([m]), torch.ones(m + 1, dtype=torch.float64, device="cuda")
    u = torch.zeros(m, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    if listed:
        gsks.set_precision(gsks.GSKS_FP64)
        gsks.dgsks_list(ker, u, i32([0, m]), am, i32([0, 1]), bm, X, X2, X, X2, one)
    else:
        gsks.dgsks_device(ker, m, 1, k, u, None, X, X2, am, X, X2, bm, one, None, nxa=m + 1, nxb=m + 1)
    torch.cuda.synchronize()
    L = np.longdouble
    d2 = ((x[:m] - x[m]).astype(L) ** 2).sum(1)
    hl = L(float(h[0].cpu()))
    if kind == "laplace":
        # (the descriptor's powe and scal are set by the call; the power is exact)
        exact, P = L(ker.scal) * np.exp(L(ker.powe) * np.log(d2)), k - 2.0
    else:
        exact, P = np.exp((L(scal) if kind == "gaussian" else -hl * hl / 2) * d2), 0.0
    err = ((u.cpu().numpy().astype(L) / exact - 1) * L(2.0) ** 53).astype(float)
    rms = np.sqrt((err * err).mean())
    if P:
        # scal multiplies the row's sum: one more rounding, up to 1 unit
        assert rms <= 1.0 + 0.08 * P and abs(err.mean()) <= 0.15 + 5 * rms / 64 + P / 100
    else:
        assert rms <= 0.45 and abs(err.mean()) <= 0.15
