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
