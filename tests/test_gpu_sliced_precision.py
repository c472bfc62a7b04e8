"""Bits that the FP64 form's inner products hold, against exact rational sums.

A row of one coordinate 1 and k - 1 of s = 2 (255 2^-17 + 255 2^-26 + .. + 255 2^-53) with
itself: the digits of s are 0, 255, 255, 255, 255, 255 at the row's exponent 1, so that
every product of the levels beyond the leading ones is at its largest and of one sign.
Bound on |x.y - exact|: the levels left out (7 and beyond) are 4 255^2 2^-77 < 2^-59 a
coordinate and less than as much again; a run of 64 coordinates is rounded once in FP32
(levels 4 to 6 joined: at most 2^27 units of 2^-53, half an ulp of which is 2^-50) and
once to W's unit (2^-50 at most); the conversion and the kernel add a few 2^-53 of the
sum.  Without level 6 the error would be (k - 1) 5 255^2 2^-68 = (k - 1) 2^-49.7."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("listed", [False, True])
@pytest.mark.parametrize("k", [5, 16, 17, 48, 64, 65, 256, 1000, 1024])
def test_every_level_that_reaches_the_rounding(gpu, k, listed):
    from ks_gb300 import gsks
    torch = gpu
    s = 2.0 * sum(255.0 * 2.0 ** (-17 - 9 * q) for q in range(5))
    x = np.full((1, k), s)
    x[0, 0] = 1.0
    X = torch.from_numpy(x).cuda()
    one = torch.ones(1, dtype=torch.float64, device="cuda")
    z = torch.zeros(1, dtype=torch.int32, device="cuda")
    off = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    u = torch.zeros(1, dtype=torch.float64, device="cuda")
    ker = gsks.make_kernel(gsks.KS_POLYNOMIAL, scal=1.0, cons=0.0, powe=1.0)
    torch.cuda.synchronize()
    if listed:
        gsks.set_precision(gsks.GSKS_FP64)
        gsks.dgsks_list(ker, u, off, z, off, z, X, None, X, None, one)
    else:
        gsks.dgsks_device(ker, 1, 1, k, u, None, X, None, None, X, None, None, one, None, nxa=1, nxb=1)
    torch.cuda.synchronize()
    exact = 1 + (k - 1) * Fraction(s) ** 2
    runs = (k + 63) // 64
    tol = runs * 2.0 ** -49 + 2 * k * 2.0 ** -59 + 8 * 2.0 ** -53 * float(exact)
    err = abs(Fraction(float(u.cpu()[0])) - exact)
    assert err <= tol, (float(err), tol)
