"""Timed workloads of the kernel summation library, through its Python entry points.

A case names an entry point, a precision, a kernel with its parameters, sizes and
the distribution of the points.  listed() holds the workloads that a program of this
library runs; draw() gives others of the same ranges.  prepare() makes the arrays (and
the plan of a planned list), run() is one evaluation u = sum_j K(x_i, y_j) w_j, exact()
the same sums from plain torch in FP64.

Entry points ("entry"):
    device   gsks.dgsks_device        device tensors, asynchronous
    rhs      gsks.dgsks_device_rhs    the same with several right-hand sides
    host     gsks.dgsks_status        host numpy arrays (the ks.h call), synchronous
    single   gsks.sgsks_status        FP32 device tensors, synchronous
    list     gsks.dgsks_list          a batch of tasks, planned by the call itself
    plan     gsks.ListPlan.execute    a batch of tasks planned once
"""
import math

import numpy as np
import torch

from ks_gb300 import gsks

KERNELS = {"gaussian": gsks.KS_GAUSSIAN, "polynomial": gsks.KS_POLYNOMIAL, "laplace": gsks.KS_LAPLACE,
           "varbw": gsks.KS_GAUSSIAN_VAR_BANDWIDTH, "tanh": gsks.KS_TANH, "quartic": gsks.KS_QUARTIC,
           "multiquadratic": gsks.KS_MULTIQUADRATIC, "epanechnikov": gsks.KS_EPANECHNIKOV}
# flops of one kernel value beyond the 2k of the inner product
KERNEL_FLOPS = {"gaussian": 37, "varbw": 35, "polynomial": 6, "laplace": 60, "tanh": 89, "quartic": 8,
                "multiquadratic": 6, "epanechnikov": 7, "mixed": 34}
DISTANCE = ("gaussian", "varbw", "laplace", "quartic", "multiquadratic", "epanechnikov")
PRECISION = {"fp64": gsks.GSKS_FP64, "split": gsks.GSKS_SPLIT_BF16X3}
LIST_SIZES = (32, 4096)      # log-uniform task sizes of the batched workload


def listed():
    return [
        # The smallest calls: one leaf block of a tree code against another.
        dict(name="fp64_gaussian_leaf", entry="device", precision="fp64", kernel="gaussian", h=0.5, m=100, n=120, k=3,
             pool=4096, points="uniform"),
        # The CPU-runnable configuration: 2048 points against themselves, k = 16, identity maps.
        dict(name="fp64_gaussian_2048", entry="device", precision="fp64", kernel="gaussian", h=1.0, m=2048, n=2048,
             k=16, pool=2048, points="uniform", identity=True),
        # The general-stride configuration at its stated size.
        dict(name="fp64_gaussian_general", entry="device", precision="fp64", kernel="gaussian", h=0.5, m=65536,
             n=65536, k=64, pool=262144, points="uniform"),
        # The same configuration's Laplace kernel on odd sizes.
        dict(name="fp64_laplace_ragged", entry="device", precision="fp64", kernel="laplace", m=20011, n=16411, k=64,
             pool=65537, points="uniform"),
        # The dense configuration (long rows, polynomial of power 4), a block of it.
        dict(name="fp64_polynomial_dense", entry="device", precision="fp64", kernel="polynomial", scal=1.0, cons=1.0,
             powe=4.0, m=8192, n=12000, k=1024, pool=16384, points="normal"),
        # Kernel regression with per-point bandwidths: numerator and denominator as two right-hand sides.
        dict(name="fp64_varbw_regression", entry="rhs", precision="fp64", kernel="varbw", hmin=0.01, hmax=0.5, nrhs=2,
             m=30000, n=32768, k=8, pool=32768, points="uniform"),
        # The batched configuration, planned once and evaluated many times (an iterative solver).
        dict(name="fp64_list_planned", entry="plan", precision="fp64", kernel="mixed", tasks=2000, k=16, pool=262144,
             points="uniform"),
        # The drop-in C call on host arrays, default precision.
        dict(name="fp64_host_gaussian", entry="host", precision="fp64", kernel="gaussian", h=0.4, m=8192, n=8191,
             k=32, pool=32768, points="uniform"),
        # The split-precision form on the general-stride configuration.
        dict(name="split_gaussian_general", entry="device", precision="split", kernel="gaussian", h=0.5, m=65536,
             n=65536, k=64, pool=262144, points="uniform"),
        dict(name="split_laplace_ragged", entry="device", precision="split", kernel="laplace", m=50021, n=40009, k=64,
             pool=131072, points="uniform"),
        # The batched configuration evaluated once: the call plans it itself.
        dict(name="split_list_oneshot", entry="list", precision="split", kernel="mixed", tasks=4000, k=16, pool=262144,
             points="uniform"),
        # Single-precision arrays, a small ordinary call.
        dict(name="single_split_polynomial", entry="single", precision="split", kernel="polynomial", scal=0.05,
             cons=1.0, powe=2.0, m=3001, n=2003, k=24, pool=8192, points="uniform"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["device", "device", "device", "rhs", "host", "single", "list", "plan"])
    precision = rng.choice(["fp64", "split"])
    if entry in ("list", "plan"):
        return dict(entry=entry, precision=precision, kernel="mixed", tasks=_log_uniform(rng, 20, 2000),
                    k=_log_uniform(rng, 8, 64), pool=_log_uniform(rng, 20000, 262144), points="uniform")
    kernel = rng.choice(["gaussian", "gaussian", "laplace", "polynomial", "polynomial", "varbw", "tanh", "quartic",
                         "multiquadratic", "epanechnikov"])
    k = _log_uniform(rng, 3, 1024)
    if kernel == "laplace":
        k = _log_uniform(rng, 5, 128)
    elif kernel == "varbw":
        k = _log_uniform(rng, 3, 64)
    m, n = _log_uniform(rng, 64, 65536), _log_uniform(rng, 64, 65536)
    # at most the largest listed case's work
    while m * n * (k + 40.0) > 65536.0 * 65536.0 * 104.0:
        m = max(64, m * 3 // 4)
        n = max(64, n * 3 // 4)
    case = dict(entry=entry, precision=precision, kernel=kernel, m=m, n=n, k=k,
                pool=_log_uniform(rng, max(m, n), 4 * max(m, n)), points="uniform")
    rms = math.sqrt(k / 6.0)                      # rms distance of uniform points
    if kernel == "gaussian":
        case["h"] = rng.uniform(0.15, 0.6) * rms
        if rng.random() < 0.3:                    # clusters far apart, kernel as wide as a cluster
            case["points"] = "mixture"
            case["h"] = rng.uniform(0.1, 0.4)
    elif kernel == "varbw":
        case["hmin"], case["hmax"] = 0.1 * rms, rms
    elif kernel == "polynomial":
        case["powe"] = float(rng.choice([2, 3, 4]))
        case["scal"], case["cons"] = 1.0 / k, 1.0
    elif kernel == "tanh":
        case["scal"], case["cons"] = 1.0 / k, rng.uniform(-0.5, 0.5)
    elif kernel == "multiquadratic":
        case["cons"] = 1.0
    elif kernel in ("quartic", "epanechnikov"):
        case["scale"] = rng.uniform(0.6, 1.4) / rms   # compact support: the points scaled to it
    if entry == "rhs":
        case["nrhs"] = rng.randint(2, 4)
    return case


def _points(case, g, count):
    k = case["k"]
    if case["points"] == "normal":
        X = torch.randn(count, k, generator=g, dtype=torch.float64, device="cuda") * (1.0 / math.sqrt(k))
    elif case["points"] == "mixture":             # 64 clusters of width 0.05 spread over [-10, 10]^k
        c = torch.rand(64, k, generator=g, dtype=torch.float64, device="cuda") * 20.0 - 10.0
        at = torch.randint(64, (count,), generator=g, device="cuda")
        X = c[at] + 0.05 * torch.randn(count, k, generator=g, dtype=torch.float64, device="cuda")
    else:
        X = torch.rand(count, k, generator=g, dtype=torch.float64, device="cuda")
    return X * case.get("scale", 1.0)


def _kernel(case, h=None):
    kind = case["kernel"]
    if kind == "gaussian":
        return gsks.make_kernel(KERNELS[kind], scal=-0.5 / case["h"] ** 2)
    if kind == "varbw":
        return gsks.make_kernel(KERNELS[kind], hi=h, hj=h)
    return gsks.make_kernel(KERNELS[kind], scal=case.get("scal", 0.0), cons=case.get("cons", 0.0),
                            powe=case.get("powe", 1.0))


def _inputs(case, seed):
    """The arrays of a single evaluation, on the device."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    N, m, n = case["pool"], case["m"], case["n"]
    d = {"X": _points(case, g, N)}
    cols = case.get("nrhs", 1)
    d["w"] = torch.randn(N * cols, generator=g, dtype=torch.float64, device="cuda")
    if case.get("identity"):
        for name, size in (("amap", m), ("bmap", n), ("umap", m), ("wmap", n)):
            d[name] = torch.arange(size, dtype=torch.int32, device="cuda")
    else:
        for name, size in (("amap", m), ("bmap", n), ("umap", m), ("wmap", n)):
            d[name] = torch.randperm(N, generator=g, device="cuda")[:size].to(torch.int32).contiguous()
    if case["kernel"] == "varbw":                 # factors 1 / h of log-uniform bandwidths
        lo, hi = math.log(case["hmin"]), math.log(case["hmax"])
        d["h"] = torch.exp(-(lo + (hi - lo) * torch.rand(N, generator=g, dtype=torch.float64, device="cuda")))
    if case["entry"] == "single":
        d["X"], d["w"] = d["X"].float(), d["w"].float()
    return d


def _list_inputs(case, seed):
    """Task lists: windows of a random permutation of the pool; every task's kernel is a Gaussian,
    a Laplace or a polynomial kernel."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = np.random.default_rng(seed)
    N, T = case["pool"], case["tasks"]
    d = {"X": _points(case, g, N), "w": torch.randn(N, generator=g, dtype=torch.float64, device="cuda")}
    perm = torch.randperm(N, generator=g, device="cuda").to(torch.int32)
    top = min(LIST_SIZES[1], N)
    for side in ("a", "b"):
        size = np.exp(r.uniform(math.log(LIST_SIZES[0]), math.log(top), T)).astype(np.int64)
        size = np.minimum(size, top)
        start = r.integers(0, N - size + 1)
        off = np.concatenate([[0], np.cumsum(size)]).astype(np.int32)
        at = np.repeat(start - off[:-1], size) + np.arange(off[-1])
        d[side + "_off"] = torch.from_numpy(off).cuda()
        d[side + "_idx"] = perm[torch.from_numpy(at).cuda()].contiguous()
    kinds = r.integers(0, 3, T)
    h = r.uniform(0.1, 2.0, T)
    power = r.integers(2, 4, T)
    d["tasks"] = [("gaussian", -0.5 / h[t] ** 2, 0.0, 1.0) if kinds[t] == 0 else
                  ("laplace", 0.0, 0.0, 1.0) if kinds[t] == 1 else
                  ("polynomial", 1.0 / case["k"], 1.0, float(power[t])) for t in range(T)]
    return d


def prepare(case, seed):
    if case["entry"] in ("list", "plan"):
        d = _list_inputs(case, seed)
        d["kers"] = [gsks.make_kernel(KERNELS[t], scal=s, cons=c, powe=p) for t, s, c, p in d["tasks"]]
        d["u"] = torch.zeros(case["pool"], dtype=torch.float64, device="cuda")
        if case["entry"] == "plan":
            N = case["pool"]
            d["plan"] = gsks.ListPlan(d["kers"][0], d["a_off"], d["a_idx"], d["b_off"], d["b_idx"], case["k"], N, N, N,
                                      N, kers=d["kers"], precision=PRECISION[case["precision"]], same_pool=True)
    else:
        d = _inputs(case, seed)
        X = d["X"].double()
        d["X2"] = (X * X).sum(1)
        cols = case.get("nrhs", 1)
        d["u"] = torch.zeros(case["pool"] * cols, dtype=d["w"].dtype, device="cuda")
        if case["entry"] == "host":
            d = {name: t.cpu().numpy() for name, t in d.items()}
        d["ker"] = _kernel(case, d.get("h"))
    d["case"] = dict(case)
    return d


def run(d):
    case = d["case"]
    entry, prec, k = case["entry"], PRECISION[case["precision"]], case["k"]
    u, X, w = d["u"], d["X"], d["w"]
    if entry == "host":
        u[:] = 0.0
        gsks.set_precision(prec)
        rc = gsks.dgsks_status(d["ker"], u, d["umap"], X, d["X2"], d["amap"], X, d["X2"], d["bmap"], w, d["wmap"])
        if rc:
            raise gsks.GsksError(rc, "dgsks")
        return u
    u.zero_()
    if entry == "device":
        N = case["pool"]
        gsks.dgsks_device(d["ker"], case["m"], case["n"], k, u, d["umap"], X, d["X2"], d["amap"], X, d["X2"],
                          d["bmap"], w, d["wmap"], precision=prec, stream=torch.cuda.current_stream(), nxa=N, nxb=N)
    elif entry == "rhs":
        N = case["pool"]
        gsks.dgsks_device_rhs(d["ker"], case["m"], case["n"], k, case["nrhs"], u, d["umap"], X, d["X2"], d["amap"], X,
                              d["X2"], d["bmap"], w, d["wmap"], precision=prec, stream=torch.cuda.current_stream(),
                              nxa=N, nxb=N)
    elif entry == "plan":
        d["plan"].execute(u, X, None, X, None, w, stream=torch.cuda.current_stream())
    else:
        # the synchronous calls run on the library's own stream: what the program enqueued before is waited for
        torch.cuda.current_stream().synchronize()
        gsks.set_precision(prec)
        if entry == "list":
            gsks.dgsks_list(d["kers"][0], u, d["a_off"], d["a_idx"], d["b_off"], d["b_idx"], X, None, X, None, w,
                            kers=d["kers"])
        else:
            rc = gsks.sgsks_status(d["ker"], u, d["umap"], X, None, d["amap"], X, None, d["bmap"], w, d["wmap"])
            if rc:
                raise gsks.GsksError(rc, "sgsks")
    return u


def work(case):
    """Each named row, weight, map entry and result once; 2k + f flops per pair."""
    k, word = case["k"], 4 if case["entry"] == "single" else 8
    f = KERNEL_FLOPS[case["kernel"]]
    if case["entry"] in ("list", "plan"):
        # the mean size of the log-uniform tasks, on each side
        lo, hi = LIST_SIZES[0], min(LIST_SIZES[1], case["pool"])
        mean = (hi - lo) / math.log(hi / lo)
        T = case["tasks"]
        pairs, rows = T * mean * mean, 2 * T * mean
        pool = case["pool"]
        return {"bytes": pool * (k + 3) * 8 + rows * 4, "flops": pairs * (2 * k + f)}
    m, n, cols = case["m"], case["n"], case.get("nrhs", 1)
    per_row = k * word + 8 + 2 * 4
    return {"bytes": (m + n) * per_row + (2 * m + n) * cols * word,
            "flops": float(m) * n * (2 * k + f + 2 * (cols - 1))}


def _values(kind, scal, cons, powe, XA, XB, same, hi=None, hj=None):
    """Kernel matrix of the rows XA against XB in FP64; same marks pairs of one and the same point."""
    if kind in DISTANCE:
        c = XB.mean(0)
        A, B = XA - c, XB - c
        d2 = (A * A).sum(1)[:, None] + (B * B).sum(1)[None, :]
        d2 = torch.addmm(d2, A, B.T, alpha=-2.0).clamp_(min=0.0)
        d2.masked_fill_(same, 0.0)
        if kind == "gaussian":
            return d2.mul_(scal).exp_()
        if kind == "varbw":
            return d2.mul_(-0.5).mul_(hi[:, None]).mul_(hj[None, :]).exp_()
        if kind == "laplace":
            k = XA.shape[1]
            front = math.gamma(0.5 * k + 1.0) / (k * (k - 2) * math.pi ** (0.5 * k))
            d2.masked_fill_(d2 < 1e-15, 1.79e308)
            return d2.pow_(0.5 * (2.0 - k)).mul_(front)
        if kind == "multiquadratic":
            return d2.add_(cons)
        t = (1.0 - d2).clamp_(min=0.0)
        return t.square_().mul_(15.0 / 16.0) if kind == "quartic" else t.mul_(0.75)
    v = (XA @ XB.T).mul_(scal).add_(cons)
    return v.tanh_() if kind == "tanh" else v.pow_(powe)


def exact(case, seed):
    if case["entry"] in ("list", "plan"):
        d = _list_inputs(case, seed)
        u = torch.zeros(case["pool"], dtype=torch.float64, device="cuda")
        a_off, b_off = d["a_off"].tolist(), d["b_off"].tolist()
        for t, (kind, scal, cons, powe) in enumerate(d["tasks"]):
            a = d["a_idx"][a_off[t]:a_off[t + 1]].long()
            b = d["b_idx"][b_off[t]:b_off[t + 1]].long()
            K = _values(kind, scal, cons, powe, d["X"][a], d["X"][b], a[:, None] == b[None, :])
            u.index_add_(0, a, K @ d["w"][b])
        return u
    d = _inputs(case, seed)
    X, cols = d["X"].double(), case.get("nrhs", 1)
    a, b = d["amap"].long(), d["bmap"].long()
    XB = X[b]
    W = d["w"].double().view(-1, cols)[d["wmap"].long()]
    u = torch.zeros(case["pool"], cols, dtype=torch.float64, device="cuda")
    scal = -0.5 / case["h"] ** 2 if case["kernel"] == "gaussian" else case.get("scal", 0.0)
    step = max(1, (1 << 28) // case["n"])
    for i in range(0, case["m"], step):
        ai = a[i:i + step]
        hi, hj = (d["h"][ai], d["h"][b]) if "h" in d else (None, None)
        K = _values(case["kernel"], scal, case.get("cons", 0.0), case.get("powe", 1.0), X[ai], XB,
                    ai[:, None] == b[None, :], hi, hj)
        u[d["umap"][i:i + step].long()] = K @ W
    u = u.view(-1)
    return u.cpu().numpy() if case["entry"] == "host" else u
