"""Batched FP64 calls of several kernel types: a launch per type, in two streams that start
after the preparation and join before the merge.  Each type's tasks on their own (one
launch, no second stream) give the same sums bit for bit: direct, planned and replayed, and
from several threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = [(0, dict(scal=-0.7)), (1, dict(scal=0.2, cons=0.5, powe=3.0)), (2, {}), (4, dict(scal=0.2, cons=0.1)), (5, {}),
         (6, dict(cons=0.25)), (7, {})]
POOL = 3000


def _lists(rng, kinds, ntask):
    tasks = []
    for t in range(ntask):
        m, n = (int(np.exp(rng.uniform(0, np.log(700)))) for _ in range(2))
        tasks.append((kinds[t % len(kinds)], rng.permutation(POOL)[:m], rng.permutation(POOL)[:n]))
    return tasks


def _args(torch, gsks, tasks, base):
    """Device lists; task t's row sums in u of their own (base[t] ..)."""
    i32 = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()
    off = lambda q: i32(np.concatenate([[0], np.cumsum([len(t[q]) for t in tasks])]))
    cat = lambda a: i32(np.concatenate(a))
    kers = [gsks.make_kernel(t[0][0], **t[0][1]) for t in tasks]
    u_idx = cat([b + np.arange(len(t[1])) for b, t in zip(base, tasks)])
    return kers, off(1), cat([t[1] for t in tasks]), off(2), cat([t[2] for t in tasks]), u_idx


def _setup(torch, gsks, k, seed, ntask=60):
    rng = np.random.default_rng(seed)
    X = torch.from_numpy(rng.random((POOL, k))).cuda()
    w = torch.from_numpy(rng.standard_normal(POOL)).cuda()
    tasks = _lists(rng, KINDS, ntask)
    base = np.concatenate([[0], np.cumsum([len(t[1]) for t in tasks])])
    nu = int(base[-1])
    torch.cuda.synchronize()

    def evaluate(idx):
        u = torch.zeros(nu, dtype=torch.float64, device="cuda")
        kers, ao, ai, bo, bi, ui = _args(torch, gsks, [tasks[t] for t in idx], [base[t] for t in idx])
        torch.cuda.synchronize()
        gsks.dgsks_list(kers[0], u, ao, ai, bo, bi, X, None, X, None, w, kers=kers, u_idx=ui)
        return u

    gsks.set_precision(gsks.GSKS_FP64)
    parts = torch.zeros(nu, dtype=torch.float64, device="cuda")
    for q in range(len(KINDS)):
        parts += evaluate(range(q, ntask, len(KINDS)))
    torch.cuda.synchronize()
    return X, w, tasks, base, nu, evaluate, parts


@pytest.mark.parametrize("k", [7, 40, 100])
def test_types_together(gpu, k):
    from ks_gb300 import gsks
    torch = gpu
    X, w, tasks, base, nu, evaluate, parts = _setup(torch, gsks, k, k)
    for _ in range(3):
        assert torch.equal(evaluate(range(len(tasks))), parts)
    kers, ao, ai, bo, bi, ui = _args(torch, gsks, tasks, base)
    plan = gsks.ListPlan(kers[0], ao, ai, bo, bi, k, nu, POOL, POOL, POOL, kers=kers, u_idx=ui, same_pool=True)
    s = torch.cuda.Stream()
    u = torch.zeros(nu, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(4):            # launched, captured, replayed
        with torch.cuda.stream(s):
            u.zero_()
            plan.execute(u, X, None, X, None, w, stream=s)
        s.synchronize()
        assert plan.errors() == 0 and torch.equal(u, parts)
    plan.close()


def test_threads(gpu):
    from ks_gb300 import gsks
    torch = gpu
    X, w, tasks, base, nu, _, parts = _setup(torch, gsks, 16, 5)
    bad = []

    def work():
        kers, ao, ai, bo, bi, ui = _args(torch, gsks, tasks, base)
        plan = gsks.ListPlan(kers[0], ao, ai, bo, bi, 16, nu, POOL, POOL, POOL, kers=kers, u_idx=ui, same_pool=True)
        s = torch.cuda.Stream()
        for _ in range(5):
            with torch.cuda.stream(s):
                u = torch.zeros(nu, dtype=torch.float64, device="cuda")
                plan.execute(u, X, None, X, None, w, stream=s)
            s.synchronize()
            bad.append(not torch.equal(u, parts))
        plan.close()

    ts = [threading.Thread(target=work) for _ in range(3)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert len(bad) == 15 and not any(bad)
