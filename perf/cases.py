"""The workloads by which this framework's speed is measured.

Every case is a piece of work that a program fitting streamline weights has the framework
do, through its public entry points: operator products A x and A' y in the FP64-accurate
and in the reduced-precision arithmetics, FISTA fits, regularisation paths and a training step
through the autograd function.  Tractograms
are smooth random walks inside an ellipsoidal mask, voxelised on a regular grid; response
functions are sticks, zeppelins and balls on a multi-shell acquisition; everything is made
on the GPU from the seed.
"""
import math

import numpy as np
import torch

NDIRS = 500          # orientations of the response-function tables
STEP = 0.5           # step of the synthetic streamlines, in voxels
GROUPS = 64          # bundles of the group-lasso paths


# ------------------------------------------------------------------------------ the cases
def listed():
    pair = dict(kind="pair", arith="ff", n_ic=1, n_ec=1, n_iso=2)
    fit = dict(n_ic=1, n_ec=1, n_iso=2)
    return [
        # a single bundle in a small region of interest: the smallest products, all latency
        dict(pair, name="pair_roi", fibers=300, voxels=1500, segs=25, n_s=66),
        # the demo-scale problem of the reference's tutorial: 32 x 32 x 16, one shell
        dict(pair, name="pair_demo", fibers=5000, voxels=12000, segs=80, n_s=66),
        # several responses per compartment, an odd acquisition and an eval mask (multi-compartment models)
        dict(pair, name="pair_multi_rf", fibers=20000, voxels=60000, segs=80, n_s=99, n_ic=3, n_ec=2, n_iso=3),
        # a sparse whole-brain tractogram on a three-shell acquisition
        dict(pair, name="pair_tract", fibers=100000, voxels=600000, segs=120, n_s=288),
        # the full-brain workload: one million streamlines on the three-shell acquisition
        dict(pair, name="pair_brain", fibers=1000000, voxels=600000, segs=120, n_s=288),
        # the same products in the BF16 arithmetic of the mixed-precision fits
        dict(pair, name="pair_brain_bf16", arith="bf16", fibers=1000000, voxels=600000, segs=120, n_s=288),
        # the FP16 arithmetic on a medium tractogram with an odd number of samples
        dict(pair, name="pair_tract_fp16", arith="fp16", fibers=150000, voxels=300000, segs=100, n_s=145),
        # a nonnegative least-squares fit as Evaluation.fit runs it: host signal in, host weights out
        dict(fit, kind="fista", name="fista_demo", reg="nnls", host=True, iters=100, fibers=5000, voxels=12000, segs=80,
             n_s=66),
        # a lasso fit of a larger tractogram with all vectors on the device
        dict(fit, kind="fista", name="fista_tract_lasso", reg="lasso", host=False, iters=12, fibers=150000,
             voxels=150000, segs=100, n_s=288),
        # a regularisation path: eight group-lasso problems on one operator
        dict(fit, kind="path", name="path_group_lasso", lambdas=8, iters=8, fibers=30000, voxels=100000, segs=100,
             n_s=288),
        # one training step: loss, gradient with respect to the weights and to all response functions
        dict(fit, kind="grad", name="grad_demo50k", fibers=50000, voxels=12000, segs=80, n_s=66),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "pair", "pair", "pair", "fista", "path", "grad"])
    case = dict(kind=kind, n_ic=1, n_ec=1, n_iso=2)
    if kind == "pair":
        case["arith"] = rng.choice(["ff", "ff", "ff", "bf16", "fp16", "f32"])
        case["fibers"] = _log(rng, 300, 800000)
        case["voxels"] = _log(rng, 1500, 600000)
        case["n_s"] = rng.randint(33, 288)
        if rng.random() < 0.25:
            case.update(n_ic=rng.randint(1, 3), n_ec=rng.randint(0, 2), n_iso=rng.randint(0, 3))
            case["fibers"] = _log(rng, 300, 100000)
    elif kind == "fista":
        case["fibers"] = _log(rng, 2000, 120000)
        case["voxels"] = _log(rng, 4000, 120000)
        case["n_s"] = rng.randint(33, 200)
        case.update(reg=rng.choice(["nnls", "lasso"]), host=rng.random() < 0.5, iters=rng.randint(8, 40))
    elif kind == "path":
        case["fibers"] = _log(rng, 3000, 30000)
        case["voxels"] = _log(rng, 8000, 100000)
        case["n_s"] = rng.randint(33, 288)
        case.update(lambdas=rng.randint(3, 8), iters=rng.randint(4, 8))
    else:
        case["fibers"] = _log(rng, 3000, 60000)
        case["voxels"] = _log(rng, 6000, 40000)
        case["n_s"] = rng.randint(33, 150)
    # streamlines cross a share of the mask's extent: short ones in small regions
    case["segs"] = rng.randint(20, max(21, min(120, int(3.0 * case["voxels"] ** (1 / 3)))))
    return case


# ------------------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _grid(voxels):
    """Grid dimensions and level of the ellipsoid r2 <= level that holds about `voxels` voxels, the mask of the fit."""
    scale = (voxels / 600000) ** (1 / 3)
    dim = [max(8, int(round(d * scale))) for d in (145, 174, 145)]
    level = (voxels / (math.pi / 6 * dim[0] * dim[1] * dim[2])) ** (2 / 3)
    return dim, level


def _walk(fibers, dim, level, mean_steps, gen):
    """Smooth random walks inside the ellipsoid: yields (count of walks still going, points,
    unit directions) step by step; walk k is the k-th longest."""
    dev = gen.device
    half = torch.tensor(dim, dtype=torch.float32, device=dev) / 2
    steps = torch.exp(math.log(mean_steps) - 0.125 + 0.5 * torch.randn(fibers, generator=gen, device=dev))
    steps = steps.clamp(2, 4 * mean_steps).to(torch.int64).sort(descending=True).values
    d = torch.nn.functional.normalize(torch.randn(fibers, 3, generator=gen, device=dev), dim=1)
    u = torch.nn.functional.normalize(torch.randn(fibers, 3, generator=gen, device=dev), dim=1)
    r = 0.95 * torch.rand(fibers, 1, generator=gen, device=dev) ** (1 / 3) * min(1.0, math.sqrt(level))
    p = half + half * r * u
    alive = (steps[None, :] > torch.arange(int(steps[0]), device=dev)[:, None]).sum(1) if fibers * int(steps[0]) < 1 << 24 \
        else fibers - torch.searchsorted(steps.flip(0), torch.arange(int(steps[0]), device=dev), right=True)
    for n in alive.tolist():
        p, d = p[:n], d[:n]
        yield n, p, d
        d = torch.nn.functional.normalize(d + 0.12 * torch.randn(n, 3, generator=gen, device=dev), dim=1)
        q = p + STEP * d
        w = (q - half) / half
        out = ((w * w).sum(1) > 0.97 * level) | (w.abs().amax(1) > 0.98)
        inward = torch.nn.functional.normalize((half - p) / half + 0.5 * torch.randn(n, 3, generator=gen, device=dev), dim=1)
        d = torch.where(out[:, None], inward, d)
        p = torch.minimum((p + STEP * d).clamp(min=0), 2 * half - 1e-3)


def _directions(dev):
    i = torch.arange(NDIRS, dtype=torch.float64, device=dev) + 0.5
    z = 1 - i / NDIRS
    phi = i * math.pi * (3 - math.sqrt(5))
    s = torch.sqrt(1 - z * z)
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z], 1)


def _direction_table(dirs):
    """Index of the direction nearest, up to sign, to each whole-degree (colatitude, longitude)."""
    deg = torch.arange(181, dtype=torch.float64, device=dirs.device) * (math.pi / 180)
    th, ph = deg[:, None], deg[None, :]
    v = torch.stack([torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th) + 0 * ph], -1)
    return (v.reshape(-1, 3) @ dirs.T).abs().argmax(1)


def _orientation(d, table):
    d = torch.where(d[:, 1:2] < 0, -d, d)
    th = (torch.acos(d[:, 2].clamp(-1, 1)) * (180 / math.pi)).round().to(torch.int64)
    ph = (torch.atan2(d[:, 1], d[:, 0]) * (180 / math.pi)).round().to(torch.int64).clamp(0, 180)
    return table[th * 181 + ph]


def _tables(case, dirs):
    """Stick, zeppelin and ball responses on b0 and three shells (FP32), normalised per compartment."""
    n_s, dev = case["n_s"], dirs.device
    n_b0 = max(1, n_s // 16)
    k = torch.arange(n_s - n_b0, device=dev)
    b = torch.cat([torch.zeros(n_b0, dtype=torch.float64, device=dev), 1000.0 * (1 + k % 3).to(torch.float64)])
    if n_s < 100:
        b = b.clamp(max=1000.0)
    i = torch.arange(n_s, dtype=torch.float64, device=dev) + 0.5
    z, phi = 1 - 2 * i / n_s, i * math.pi * (3 - math.sqrt(5))
    s = torch.sqrt(1 - z * z)
    cos2 = (dirs @ torch.stack([s * torch.cos(phi), s * torch.sin(phi), z], 0)) ** 2
    ic = [torch.exp(-b * 1.7e-3 * (1 - 0.15 * r) * cos2) for r in range(case["n_ic"])]
    ec = [torch.exp(-b * (q + (1.7e-3 - q) * cos2)) for q in (0.51e-3, 0.85e-3)[:case["n_ec"]]]
    iso = [torch.exp(-b * q) for q in (1.7e-3, 3.0e-3, 0.9e-3)[:case["n_iso"]]]
    ic = [m / m[0].norm() for m in ic]
    ec = [m / m[0].norm() for m in ec]
    iso = [m / m.norm() for m in iso]

    def stack(rows, shape):
        return torch.stack(rows).float().contiguous() if rows else torch.zeros(shape, dtype=torch.float32, device=dev)
    return stack(ic, (0, NDIRS, n_s)), stack(ec, (0, NDIRS, n_s)), stack(iso, (0, n_s))


def _problem(case, seed):
    """Dictionary arrays (voxel-sorted), response tables, weights x and signal y on the GPU."""
    gen = _generator(seed)
    dev = gen.device
    dim, level = _grid(case["voxels"])
    fibers = case["fibers"]
    dirs = _directions(dev)
    table = _direction_table(dirs)
    size = dim[0] * dim[1] * dim[2]
    name = torch.randperm(fibers, generator=gen, device=dev)     # walks come longest first
    keys = []
    for n, p, d in _walk(fibers, dim, level, 1.06 * case["segs"], gen):
        q = p.to(torch.int64)
        lin = q[:, 0] + dim[0] * (q[:, 1] + dim[1] * q[:, 2])
        keys.append((lin * fibers + name[:n]) * NDIRS + _orientation(d, table))
    key, count = torch.unique(torch.cat(keys), return_counts=True)
    del keys
    o = key % NDIRS
    key = key // NDIRS
    f = key % fibers
    lin = key // fibers
    del key
    at = torch.arange(size, device=dev)
    at = torch.stack([at % dim[0], at // dim[0] % dim[1], at // (dim[0] * dim[1])], 1)
    half = torch.tensor(dim, dtype=torch.float32, device=dev) / 2
    mask = ((((at + 0.5 - half) / half) ** 2).sum(1) <= level).to(torch.int64)
    del at
    inside = mask[lin] > 0
    v = (torch.cumsum(mask, 0) - 1)[lin[inside]]
    f, o, count = f[inside], o[inside], count[inside]
    n_vox = int(mask.sum())
    del lin, mask, inside
    raw = count * torch.randint(600, 1400, count.shape, generator=gen, device=dev)   # lengths, exact in any order
    norm = torch.zeros(fibers, dtype=torch.int64, device=dev).index_add_(0, f, raw)
    length = (raw.double() / norm[f].clamp(min=1).double()).float()
    del raw, norm, count
    wic, wec, wiso = _tables(case, dirs)
    peaks = 1 + torch.randperm(n_vox, generator=gen, device=dev) % 4 if case["n_ec"] else torch.zeros_like(v[:1]).expand(n_vox)
    ecv = torch.repeat_interleave(torch.arange(n_vox, device=dev), peaks)
    eco = torch.randint(0, NDIRS, ecv.shape, generator=gen, device=dev)
    n_iso = n_vox if case["n_iso"] else 0
    n_cols = fibers * case["n_ic"] + ecv.numel() * case["n_ec"] + n_iso * case["n_iso"]
    x = torch.rand(n_cols, generator=gen, device=dev, dtype=torch.float64)
    keep = torch.ones(fibers * case["n_ic"], dtype=torch.int32, device=dev)
    if case["n_ic"] > 1:
        keep = (torch.rand(fibers * case["n_ic"], generator=gen, device=dev) < 0.95).to(torch.int32)
    # a measured signal: a random mixture of two sticks and a ball per voxel, Rician noise of 2 %
    y = torch.empty(n_vox, case["n_s"], dtype=torch.float64, device=dev)
    ball = wiso[0].double() if case["n_iso"] else wic[0].double().mean(0)
    for a in range(0, n_vox, 1 << 16):
        m = min(n_vox - a, 1 << 16)
        w = torch.rand(m, 3, generator=gen, device=dev, dtype=torch.float64)
        r = wic[0].double()[torch.randint(0, NDIRS, (2, m), generator=gen, device=dev)]
        s = w[:, 0:1] * r[0] + w[:, 1:2] * r[1] + w[:, 2:3] * ball
        e = 0.02 * s.mean() * torch.randn(2, m, case["n_s"], generator=gen, device=dev, dtype=torch.float64)
        y[a:a + m] = torch.sqrt((s + e[0]) ** 2 + e[1] ** 2)
    if case["kind"] == "pair" and case["arith"] != "ff":
        x, y = x.float(), y.float()
    return dict(f=f, v=v, o=o, l=length, ecv=ecv, eco=eco, n_iso=n_iso, n_vox=n_vox, wic=wic, wec=wec, wiso=wiso, x=x,
                y=y.reshape(-1), keep=keep, fibers=fibers)


def _dictionary(p):
    """The problem as the DICTIONARY and KERNELS that LinearOperator takes."""
    IC = {"str": p["f"].to(torch.int32), "vox": p["v"].to(torch.int32), "dir": p["o"].to(torch.int16), "len": p["l"],
          "eval": p["keep"], "n": p["f"].numel(), "nSTR": p["fibers"], "nVOX": p["n_vox"]}
    EC = {"vox": p["ecv"].to(torch.int32), "dir": p["eco"].to(torch.int16), "n": p["ecv"].numel()}
    ISO = {"vox": torch.arange(p["n_iso"], dtype=torch.int32, device=p["f"].device), "n": p["n_iso"]}
    K = {"wmr": p["wic"].cpu().numpy(), "wmh": p["wec"].cpu().numpy(), "iso": p["wiso"].cpu().numpy()}
    return {"IC": IC, "EC": EC, "ISO": ISO}, K


def _layout(case, p):
    """The compartment layout part of a regularisation dict."""
    ic, ec = p["fibers"] * case["n_ic"], p["ecv"].numel() * case["n_ec"]
    return {"startIC": 0, "sizeIC": ic, "startEC": ic, "sizeEC": ec, "startISO": ic + ec,
            "sizeISO": p["n_iso"] * case["n_iso"], "regIC": None, "regEC": None, "regISO": None, "nnIC": True,
            "nnEC": True, "nnISO": True, "dictIC_params": None, "dictEC_params": None, "dictISO_params": None}


def _lasso(case):
    return 0.02 if case["reg"] == "lasso" else 0.0


def _bundles(case, seed):
    label = np.random.default_rng(seed).integers(0, GROUPS, case["fibers"])
    groups = [g for g in (np.flatnonzero(label == k) for k in range(GROUPS)) if g.size]
    weights = np.sqrt([float(g.size) for g in groups])
    lambdas = np.logspace(-4, -1, case["lambdas"]) * 0.3
    return groups, weights, lambdas


def prepare(case, seed):
    from commit_gb300 import solvers
    from commit_gb300.operator import LinearOperator
    p = _problem(case, seed)
    D, K = _dictionary(p)
    s = dict(kind=case["kind"], A=LinearOperator(D, K), x=p["x"], y=p["y"])
    if case["kind"] == "pair":
        s["arith"] = None if case["arith"] == "ff" else case["arith"]
    elif case["kind"] == "fista":
        rp = _layout(case, p)
        if _lasso(case):
            rp.update(regIC="lasso", lambdaIC=_lasso(case))
        s.update(reg=solvers.init_regularisation(rp), iters=case["iters"])
        if case["host"]:
            s["y"] = s["y"].cpu().numpy()
    elif case["kind"] == "path":
        groups, weights, lambdas = _bundles(case, seed)
        s["regs"] = [solvers.init_regularisation(dict(
            _layout(case, p), regIC="group_lasso", lambdaIC=float(lam),
            dictIC_params={"group_idx_kept": groups, "group_weights": weights})) for lam in lambdas]
        s["iters"] = case["iters"]
    else:
        s["luts"] = [p[k].clone().requires_grad_(True) for k in ("wic", "wec", "wiso")]
        s["x"] = p["x"].requires_grad_(True)
    return s


def run(state):
    A, y = state["A"], state["y"]
    if state["kind"] == "pair":
        return [A.dot(state["x"], arith=state["arith"]), A.T.dot(y, arith=state["arith"])]
    from commit_gb300 import solvers
    if state["kind"] == "fista":
        x, details = solvers.solve(y, A, A.T, tol_fun=0.0, tol_x=0.0, max_iter=state["iters"], verbose=False,
                                   regularisation=state["reg"])
        return [x, details["cost_function"]]
    if state["kind"] == "path":
        fits = solvers.solve_batch(y, A, state["regs"], tol_fun=0.0, tol_x=0.0, max_iter=state["iters"])
        return [[x, details["cost_function"]] for x, details in fits]
    from commit_gb300.autograd import commit_apply
    leaves = [state["x"]] + state["luts"]
    predicted = commit_apply(A, *leaves)
    loss = 0.5 * ((predicted - y) ** 2).sum()
    return [predicted.detach()] + list(torch.autograd.grad(loss, leaves))


# ------------------------------------------------------------------------------ work
def work(case):
    """Bytes and operations of one pass: dictionary items and vectors once per product, one
    multiply-add per item and sample."""
    n, nv, n_s = case["fibers"] * case["segs"], case["voxels"], case["n_s"]
    ec = 2.5 * nv if case["n_ec"] else 0
    iso = nv if case["n_iso"] else 0
    cols = case["fibers"] * case["n_ic"] + ec * case["n_ec"] + iso * case["n_iso"]
    reduced = case["kind"] == "path" or case.get("arith", "ff") != "ff"
    item, word = (12, 4) if reduced else (14, 8)
    byte = n * item + ec * 6 + iso * 4 + cols * word + nv * n_s * word
    flop = 2.0 * n_s * (n * case["n_ic"] + ec * case["n_ec"] + iso * case["n_iso"])
    products = {"pair": 2, "grad": 3}.get(case["kind"], 2 * case.get("iters", 1) + 2) * case.get("lambdas", 1)
    return {"bytes": byte * products, "flops": flop * products}


# ------------------------------------------------------------------------------ in 64 bits
def _dense(p, voxels=1 << 15):
    """(A, A') of the problem in FP64: per run of voxels the summed coefficients of every
    response row, as a dense matrix times the table."""
    x64 = dict(l=p["l"].double(), ic=p["wic"].double(), ec=p["wec"].double(), iso=p["wiso"].double())
    n_ic, n_ec, n_iso = x64["ic"].shape[0], x64["ec"].shape[0], x64["iso"].shape[0]
    nf, ne, ni = p["fibers"], p["ecv"].numel(), p["n_iso"]
    n_s = x64["ic"].shape[-1]
    starts = list(range(0, p["n_vox"], voxels)) + [p["n_vox"]]
    cut = torch.searchsorted(p["v"], torch.tensor(starts, device=p["v"].device)).tolist()
    cute = torch.searchsorted(p["ecv"], torch.tensor(starts, device=p["v"].device)).tolist()
    keep = p["keep"].double()

    def forward(x):
        x = x.double()
        xe = x[:nf * n_ic] * keep
        y = torch.zeros(p["n_vox"], n_s, dtype=torch.float64, device=x.device)
        for k in range(len(starts) - 1):
            a, b = starts[k], starts[k + 1]
            s, e = slice(cut[k], cut[k + 1]), slice(cute[k], cute[k + 1])
            at, ate = (p["v"][s] - a) * NDIRS + p["o"][s], (p["ecv"][e] - a) * NDIRS + p["eco"][e]
            for i in range(n_ic):
                c = torch.zeros((b - a) * NDIRS, dtype=torch.float64, device=x.device)
                c.index_add_(0, at, x64["l"][s] * xe[i * nf + p["f"][s]])
                y[a:b] += c.view(b - a, NDIRS) @ x64["ic"][i]
            for i in range(n_ec):
                c = torch.zeros((b - a) * NDIRS, dtype=torch.float64, device=x.device)
                c.index_add_(0, ate, x[nf * n_ic + i * ne + cute[k]:nf * n_ic + i * ne + cute[k + 1]])
                y[a:b] += c.view(b - a, NDIRS) @ x64["ec"][i]
        for i in range(n_iso):
            o = nf * n_ic + ne * n_ec + i * ni
            y += x[o:o + ni, None] * x64["iso"][i]
        return y.view(-1)

    def adjoint(y):
        y = y.double().view(p["n_vox"], n_s)
        ic = torch.zeros(n_ic, nf, dtype=torch.float64, device=y.device)
        ec = torch.zeros(n_ec, ne, dtype=torch.float64, device=y.device)
        for k in range(len(starts) - 1):
            a, b = starts[k], starts[k + 1]
            s, e = slice(cut[k], cut[k + 1]), slice(cute[k], cute[k + 1])
            at, ate = (p["v"][s] - a) * NDIRS + p["o"][s], (p["ecv"][e] - a) * NDIRS + p["eco"][e]
            for i in range(n_ic):
                ic[i].index_add_(0, p["f"][s], x64["l"][s] * (y[a:b] @ x64["ic"][i].T).view(-1)[at])
            for i in range(n_ec):
                ec[i, e] = (y[a:b] @ x64["ec"][i].T).view(-1)[ate]
        iso = (y @ x64["iso"].T).T if n_iso else y[:0, 0]
        return torch.cat([ic.view(-1) * keep, ec.view(-1), iso.reshape(-1)])

    return forward, adjoint


def _fista(A, At, y, prox, omega, iters, n_cols):
    """FISTA with backtracking for a fixed number of iterations, from zero."""
    xhat = torch.zeros(n_cols, dtype=torch.float64, device=y.device)
    prev = xhat
    r = A(xhat) - y
    grad = At(r)
    objective = 0.5 * float(r.norm()) ** 2
    step = 1.9 / (float(A(grad).norm()) / float(grad.norm())) ** 2
    t_old, f_hat = 1.0, objective
    for it in range(1, iters + 1):
        while True:
            x = prox(xhat - step * grad, step)
            d = x - xhat
            model = f_hat + float(d @ grad) + 0.5 / step * float(d.norm()) ** 2 + omega(x)
            objective = 0.5 * float((A(x) - y).norm()) ** 2 + omega(x)
            if objective <= model:
                break
            step *= 0.9
        if it == iters:
            return x, objective
        t = 0.5 * (1 + math.sqrt(1 + 4 * t_old * t_old))
        xhat = x + (t_old - 1) / t * (x - prev)
        r = A(xhat) - y
        grad = At(r)
        prev, t_old, f_hat = x, t, 0.5 * float(r.norm()) ** 2


def exact(case, seed):
    p = _problem(case, seed)
    A, At = _dense(p)
    if case["kind"] == "pair":
        return [A(p["x"]), At(p["y"])]
    y, n_cols = p["y"], p["x"].numel()
    if case["kind"] == "fista":
        n, lam = p["fibers"] * case["n_ic"], _lasso(case)

        def prox(x, s):
            x[:n] -= s * lam
            return x.clamp_(min=0)
        x, cost = _fista(A, At, y, prox, lambda x: lam * float(x[:n].abs().sum()), case["iters"], n_cols)
        return [x.cpu().numpy() if case["host"] else x, cost]
    if case["kind"] == "path":
        groups, weights, lambdas = _bundles(case, seed)
        at = [torch.from_numpy(g).to(y.device) for g in groups]
        out = []
        for lam in lambdas:
            def prox(x, s):
                for g, w in zip(at, weights):
                    v, m = x[g], s * float(lam) * float(w)
                    x[g] = v * max(0.0, 1 - m / max(float(v.norm()), 1e-300))
                return x.clamp_(min=0)

            def omega(x):
                return float(lam) * sum(float(w) * float(x[g].norm()) for g, w in zip(at, weights))
            out.append(list(_fista(A, At, y, prox, omega, case["iters"], n_cols)))
        return out
    predicted = A(p["x"])
    r = (predicted - y).view(p["n_vox"], -1)
    nf = p["fibers"]
    g_ic = torch.zeros(NDIRS, r.shape[1], dtype=torch.float64, device=y.device)
    for a in range(0, p["f"].numel(), 1 << 20):
        s = slice(a, a + (1 << 20))
        g_ic.index_add_(0, p["o"][s], (p["l"][s].double() * p["x"][p["f"][s]] * p["keep"][p["f"][s]])[:, None] * r[p["v"][s]])
    g_ec = torch.zeros_like(g_ic).index_add_(0, p["eco"], p["x"][nf:nf + p["ecv"].numel(), None] * r[p["ecv"]])
    o = nf + p["ecv"].numel()
    g_iso = torch.stack([p["x"][o + i * p["n_iso"]:o + (i + 1) * p["n_iso"]] @ r for i in range(case["n_iso"])])
    return [predicted, At(r.reshape(-1)), g_ic[None], g_ec[None], g_iso]
