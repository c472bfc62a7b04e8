"""Split-precision form: the survey of a call's points (bounding box, anchor
coordinates, weight sum: three kinds of blocks of one launch) at the edges of its
blocks: 32 coordinates, a sample of 2048 sources in 16 parts, 4096 weights.

Tolerance 1e-6, the gate of the split form (normwise and conditioned)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-6


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (2, 15, 31), (129, 2047, 32), (3, 2049, 33), (64, 4096, 5),
                                   (5, 4097, 65), (1, 8193, 300)])
@pytest.mark.parametrize("ktype,params", [(1, dict(scal=0.05, cons=1.0, powe=2.0)), (4, dict(scal=0.1, cons=0.1)),
                                          (0, dict(scal=-0.5))])
def test_split_survey_edges(gpu, oracle_mod, m, n, k, ktype, params):
    from test_gpu_split import _run
    rng = np.random.default_rng(m + n + k)
    N = m + n
    X = rng.random((N, k)) / np.sqrt(k) + (0.25 if ktype else 0.0)
    perm = rng.permutation(N).astype(np.int32)
    e = _run(gpu, oracle_mod, ktype, params, X, rng.standard_normal(N), perm[:m], perm[m:], perm[:m], perm[m:])
    assert e["normwise"] <= TOL and e["cond_max"] <= TOL, e


@pytest.mark.parametrize("k", [5, 64, 100])
@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e200])
def test_split_non_finite_coordinate(gpu, k, bad):
    """A coordinate that the operand slices cannot hold does not turn into a finite value."""
    from ks_gb300 import gsks
    rng = np.random.default_rng(k)
    X = rng.random((300, k))
    X[7, k // 2] = bad
    t = lambda a: gpu.from_numpy(np.ascontiguousarray(a)).cuda()
    i = t(np.arange(300, dtype=np.int32))
    x, u = t(X), gpu.zeros(300, dtype=gpu.float64, device="cuda")
    with np.errstate(over="ignore"):
        x2 = t((X * X).sum(1))
    gsks.dgsks_device(gsks.make_kernel(1, scal=0.05, cons=1.0, powe=2.0), 300, 300, k, u, i, x, x2, i, x, x2, i,
                      t(rng.random(300)), i, precision=1, stream=gpu.cuda.current_stream(), nxa=300, nxb=300)
    gpu.cuda.synchronize()
    assert not np.isfinite(u.cpu().numpy()[7])
