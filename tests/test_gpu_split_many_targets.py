"""Split form, many more targets than sources: maps of the sources have an entry per source
and are read at no target's position (wmap in an allocation of its own here)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ktype,params", [(0, dict(scal=-0.7)), (1, dict(scal=0.3, cons=0.5, powe=3.0)), (7, {})])
@pytest.mark.parametrize("how", ["single", "rhs", "list"])
def test_many_targets(gpu, how, ktype, params):
    from ks_gb300 import gsks
    torch, k, m, n, N = gpu, 14, 3_000_000, 70, 5000
    rng = np.random.default_rng(0)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    X = t(rng.random((N, k)) * 0.5)
    X2 = (X * X).sum(1)
    nrhs = 2 if how == "rhs" else 1
    w = t(rng.standard_normal((n, nrhs)))
    am, bm = t(rng.integers(0, N, m).astype(np.int32)), t(rng.permutation(N)[:n].astype(np.int32))
    wm = torch.empty(n, dtype=torch.int32, device="cuda")
    wm.copy_(torch.arange(n, dtype=torch.int32).flip(0))
    row = torch.arange(m, dtype=torch.int32, device="cuda")
    u = torch.zeros(m, nrhs, dtype=torch.float64, device="cuda")
    ker = gsks.make_kernel(ktype, **params)
    torch.cuda.synchronize()
    if how == "list":
        gsks.set_precision(gsks.GSKS_SPLIT_BF16X3)
        off = lambda q: torch.tensor([0, q], dtype=torch.int32, device="cuda")
        try:
            gsks.dgsks_list(ker, u.view(-1), off(m), am, off(n), bm, X, X2, X, X2, w.view(-1), u_idx=row, w_idx=wm)
        finally:
            gsks.set_precision(gsks.GSKS_FP64)
    else:
        gsks.dgsks_device_rhs(ker, m, n, k, nrhs, u, row, X, X2, am, X, X2, bm, w, wm, precision=gsks.GSKS_SPLIT_BF16X3,
                              stream=torch.cuda.current_stream(), nxa=N, nxb=N)
        torch.cuda.synchronize()
        assert gsks.device_errors() == 0
    W = w[wm.long()]
    Y = X[bm.long()]
    dot, d2 = X @ Y.T, torch.cdist(X, Y, compute_mode="donot_use_mm_for_euclid_dist") ** 2
    K = {0: lambda: torch.exp(-0.7 * d2), 1: lambda: (0.3 * dot + 0.5) ** 3, 7: lambda: 0.75 * (1 - d2).clamp(min=0)}[ktype]()
    ref, mag = (K @ W)[am.long()], (K.abs() @ W.abs())[am.long()]
    assert torch.all((u - ref).abs() <= 1e-6 * mag + 1e-12)
