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


def test_guard_bits_without_a_frame(gpu):
    """A kernel that has a fixed-point form, on points that leave it off (one near the
    origin): x.y keeps the guard bits of a plain inner product.  Rows x = (3/4, s, .., s)
    and y = (5/8, t, .., t) on the digits' grid, k = 1024: every run of 64 coordinates has
    the same sum, so that its rounding to W's unit (2^-52; 2^-50 with the frame's guard
    bits) adds up 16 times.  Bound on the exponent: 16 roundings of at most one unit, twice
    for 2 x.y, the level left out (2^-50), the norms' and the value's own rounding."""
    import math
    from ks_gb300 import gsks
    torch = gpu
    k, rows = 1024, 400
    rng = np.random.default_rng(1)
    s = rng.integers(2 ** 47, 2 ** 48, rows)             # units of 2^-53: 2^-6 .. 2^-5
    t = int(rng.integers(2 ** 47, 2 ** 48))
    x = np.empty((rows + 2, k))
    x[:rows] = (s.astype(float) * 2.0 ** -53)[:, None]
    x[:rows, 0] = 0.75
    x[rows] = t * 2.0 ** -53
    x[rows, 0] = 0.625
    x[rows + 1] = 2.0 ** -40                             # the point near the origin
    n2 = lambda c0, c: Fraction(c0) ** 2 + (k - 1) * Fraction(int(c), 2 ** 53) ** 2
    x2 = np.array([float(n2(0.75, c)) for c in s] + [float(n2(0.625, t)), k * 2.0 ** -80])
    X, X2 = torch.from_numpy(x).cuda(), torch.from_numpy(x2).cuda()
    w = torch.tensor([1.0, 0.0], dtype=torch.float64, device="cuda")
    bm = torch.tensor([rows, rows + 1], dtype=torch.int32, device="cuda")
    u = torch.zeros(rows, dtype=torch.float64, device="cuda")
    wm = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    gsks.dgsks_device(gsks.make_kernel(0, scal=-1.0), rows, 2, k, u, None, X, X2, None, X, X2, bm, w, wm, nxa=rows + 2,
                      nxb=rows + 2)
    torch.cuda.synchronize()
    d2 = [Fraction(1, 64) + (k - 1) * Fraction(int(c) - t, 2 ** 53) ** 2 for c in s]
    err = max(abs(float(u.cpu()[i]) / math.exp(-float(d2[i])) - 1.0) for i in range(rows))
    assert err <= 2.0 ** -47 + 2.0 ** -50 + 8 * 2.0 ** -53, err / 2.0 ** -53
