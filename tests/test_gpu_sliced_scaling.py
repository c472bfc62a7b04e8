"""Inner products of points whose coordinates differ widely in size, against exact sums.

The FP64 form holds a point's coordinates relative to the largest one; the kernels without
norms (polynomial, tanh) need x.y to a few units of 2^-53 sum |x_p y_p| all the same.

Bound on |x.y - exact| in units of 2^-53 sum |x_p y_p|: a pair formed directly is a chain of k
fused multiply-adds, rms below k^1/2 / 2: 4 k^1/2.  A pair from digits has W at least 2^-4 of
the longer point's length N (or points with half of their coordinates in common), and W's
error is 2^-54.3 N rms: 2^-50.3 of the sum, 6.5 units; six times that is 39, 64 with the
roundings to W's unit.  Kernel values: that times |f'|, and a few units of the value."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS, COLS = 70, 24


def _points(kind, k, rng, n):
    x = rng.standard_normal((n, k))
    if kind == "columns":                       # every feature in a unit of its own
        x *= 10.0 ** rng.uniform(-6, 6, k)
    elif kind == "one_large":                   # one large feature, zero in half of the points
        x[:, 0] *= 1e12 * (rng.random(n) < 0.5)
    elif kind == "heavy":
        x *= np.exp(4.0 * rng.standard_normal((n, k)))
    elif kind == "sparse":
        x *= rng.random((n, k)) < 0.15
    elif kind == "disjoint":                    # large coordinates that meet zeros and small ones
        half = np.arange(n) % 2 == 0
        x[np.ix_(half, np.arange(k) < (k + 1) // 2)] *= 1e15
        x[np.ix_(~half, np.arange(k) >= (k + 1) // 2)] *= 1e15
        x[::5] *= rng.random((len(x[::5]), k)) < 0.5
    elif kind == "counts":
        x = np.floor(np.abs(rng.standard_cauchy((n, k))) * (rng.random((n, k)) < 0.3))
    return x


def _exact(x, y):
    f = [[Fraction(v) for v in r] for r in x.tolist()], [[Fraction(v) for v in r] for r in y.tolist()]
    dot = [[sum((a * b for a, b in zip(r, s) if a and b), Fraction(0)) for s in f[1]] for r in f[0]]
    ab = np.abs(x) @ np.abs(y).T
    return dot, ab


def _pairs(gsks, torch, ker, x, y, how):
    """K(x_i, y_j), one source a call (or task)."""
    m, n, k = len(x), len(y), x.shape[1]
    X, Y = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    if how == "list":
        i32 = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()
        u = torch.zeros(m * n, dtype=torch.float64, device="cuda")
        gsks.set_precision(gsks.GSKS_FP64)
        torch.cuda.synchronize()
        gsks.dgsks_list(ker, u, i32(np.arange(n + 1) * m), i32(np.tile(np.arange(m), n)), i32(np.arange(n + 1)),
                        i32(np.arange(n)), X, None, Y, None, torch.ones(n, dtype=torch.float64, device="cuda"),
                        u_idx=i32(np.arange(m * n)))
        return u.cpu().numpy().reshape(n, m).T
    nrhs = 3 if how == "rhs" else 1
    out = np.empty((m, n))
    w = torch.tensor([1.0, 2.0, 4.0][:nrhs], dtype=torch.float64, device="cuda")
    for j in range(n):
        u = torch.zeros(m * nrhs, dtype=torch.float64, device="cuda")
        gsks.dgsks_device_rhs(ker, m, 1, k, nrhs, u, None, X, None, None, Y[j:], None, None, w, None,
                              stream=torch.cuda.current_stream(), nxa=m, nxb=1)
        torch.cuda.synchronize()
        v = u.cpu().numpy().reshape(m, nrhs)
        for r in range(nrhs):
            assert np.array_equal(v[:, r], v[:, 0] * 2.0 ** r)
        out[:, j] = v[:, 0]
    return out


TABLE = [((1e6, 1 / 3), (0, 1)), ((1e12, 1 / 3), (0, 1)), ((1e20, 1 / 3), (0, 1)), ((1e20, 1), (1e-20, 1)),
         ((1e6, 0.3), (0, 0.7)), ((1e15, 0.3), (0, 0.7)), ((1, 1e-10, 1, 1, 1), (0, 1, 0, 0, 0)),
         ((1, 2.0 ** -5, 2.0 ** -5, 1e-9), (1e-9, 2.0 ** -5, -2.0 ** -5, 1)), ((1e-140, 1e-150, 3), (1e145, 1e-100, 0))]


@pytest.mark.parametrize("how", ["single", "rhs", "list"])
def test_rows_of_a_few_coordinates(gpu, how):
    from ks_gb300 import gsks
    ker = gsks.make_kernel(gsks.KS_POLYNOMIAL, scal=1.0, cons=0.0, powe=1.0)
    for x, y in TABLE:
        x, y = np.array([x, y], float), np.array([y, x], float)
        got = _pairs(gsks, gpu, ker, x, y, how)
        dot, ab = _exact(x, y)
        for i in range(2):
            for j in range(2):
                assert abs(Fraction(got[i, j]) - dot[i][j]) <= (64 + 4 * 5 ** 0.5) * 2.0 ** -53 * ab[i, j], (x, y, i, j)


@pytest.mark.parametrize("kind", ["columns", "one_large", "heavy", "sparse", "disjoint", "counts", "normal"])
@pytest.mark.parametrize("k,how", [(2, "single"), (3, "list"), (7, "single"), (16, "rhs"), (33, "list"), (64, "single"),
                                   (65, "single"), (200, "list"), (257, "rhs"), (600, "single")])
def test_inner_products(gpu, kind, k, how):
    from ks_gb300 import gsks
    rng = np.random.default_rng(k)
    x, y = _points(kind, k, rng, ROWS), _points(kind, k, rng, COLS)
    ker = gsks.make_kernel(gsks.KS_POLYNOMIAL, scal=1.0, cons=0.0, powe=1.0)
    got = _pairs(gsks, gpu, ker, x, y, how)
    dot, ab = _exact(x, y)
    worst = max(float(abs(Fraction(got[i, j]) - dot[i][j])) / (2.0 ** -53 * ab[i, j])
                for i in range(ROWS) for j in range(COLS) if ab[i, j] > 0)
    assert worst <= 64 + 4 * k ** 0.5
    assert all(got[i, j] == 0.0 for i in range(ROWS) for j in range(COLS) if ab[i, j] == 0)


@pytest.mark.parametrize("kind", ["columns", "one_large", "disjoint", "sparse"])
@pytest.mark.parametrize("k", [3, 20, 130])
@pytest.mark.parametrize("power", [0, 2, 3, 4])       # 0: tanh
def test_kernel_values(gpu, kind, k, power):
    from ks_gb300 import gsks
    rng = np.random.default_rng(100 + k)
    x, y = _points(kind, k, rng, 40), _points(kind, k, rng, 9)
    dot, ab = _exact(x, y)
    scal = 1.0 / float(np.median(ab[ab > 0]))
    cons = 0.125
    ker = (gsks.make_kernel(gsks.KS_POLYNOMIAL, scal=scal, cons=cons, powe=float(power)) if power
           else gsks.make_kernel(gsks.KS_TANH, scal=scal, cons=cons))
    got = _pairs(gsks, gpu, ker, x, y, "single")
    c = np.array([[float(Fraction(scal) * d + Fraction(cons)) for d in r] for r in dot])
    dc = 2.0 ** -53 * ((64 + 4 * k ** 0.5) * ab * scal + 2 * np.abs(c) + 2 * np.abs(c - cons))
    if power:
        val, slope = c ** power, power * np.abs(c) ** (power - 1)
    else:
        val, slope = np.tanh(c), np.cosh(np.minimum(np.abs(c), 300.0)) ** -2.0
    # (near 0 the slope changes over dc: to second order; 8 units of the value for the
    # power or tanh and for numpy's own)
    curve = power * (power - 1) * (np.abs(c) + dc) ** max(power - 2, 0) if power else 1.0
    assert np.all(np.abs(got - val) <= slope * dc + curve * dc * dc + 8 * 2.0 ** -53 * np.abs(val))


@pytest.mark.parametrize("how", ["single", "rhs", "list"])
@pytest.mark.parametrize("k", [3, 20, 70, 300])
def test_sums_beyond_the_range(gpu, k, how):
    """x.y beyond FP64's range: a chain of fused multiply-adds has the sign of its first
    overflow (and is a NaN only where a coordinate is), tanh of it 1 or -1."""
    from ks_gb300 import gsks
    rng = np.random.default_rng(k)
    x, y = rng.standard_normal((40, k)) * 1e160, rng.standard_normal((6, k)) * 1e160
    got = _pairs(gsks, gpu, gsks.make_kernel(gsks.KS_TANH, scal=1.0), x, y, how)
    for i in range(40):
        for j in range(6):
            s = Fraction(0)
            for a, b in zip(x[i], y[j]):
                s += Fraction(a) * Fraction(b)
                if abs(s) >= 2 ** 1024:
                    break
            assert got[i, j] == (1.0 if s > 0 else -1.0)
