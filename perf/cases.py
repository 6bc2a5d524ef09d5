"""Timed cases of the package: the work its users have it do, each case one
call sequence through the public entry points (geosgs.rand, Plan, Batch,
posterior, the ensemble statistics and the warm-start network's training
step), over the ranges of the repository's workloads and tests.

    listed()            the cases timed by default
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call
    run(state)          one pass, returning its outputs
    work(case)          bytes and FLOPs one pass cannot do without
    exact(case, seed)   the same outputs in plain FP64 torch / numpy
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "geostatsprocesses.jl_gb300"))

import geosgs  # noqa: E402
from geosgs import ensemble, learned  # noqa: E402

VARIOS = {"sph": geosgs.SphericalVariogram, "exp": geosgs.ExponentialVariogram, "gau": geosgs.GaussianVariogram}
QUANTILES = [0.1, 0.5, 0.9]
THRESHOLDS = [-0.5, 0.0, 1.0]


def listed():
    return [
        # the smallest whole call: rand() of a few realizations of a small 2D
        # grid in the plain FP64 precision, arrays back on the host; launches,
        # copies and latency count
        dict(name="rand_fp64_100x100", kind="rand", nx=100, ny=100, nz=1, vario="sph", range=20.0, ratio=1.0,
             nugget=0.0, ball=40.0, ndata=0, k=12, reals=4, path="random", precision="fp64"),
        # the method's defaults (linear path, 26 neighbours, ball of the
        # range, one realization): a long chain of short dependency levels
        dict(name="defaults_300x300", kind="plan", nx=300, ny=300, nz=1, vario="sph", range=30.0, ratio=1.0,
             nugget=0.05, ball=0.0, ndata=0, k=26, reals=1, path="linear", precision="fp32", warm=False),
        # conditional simulation of a smooth model on a 2D map, data at cell
        # centres (some systems are singular): create, prepare, simulate, destroy
        dict(name="conditional_500x500", kind="plan", nx=500, ny=500, nz=1, vario="gau", range=30.0, ratio=1.0,
             nugget=0.1, ball=0.0, ndata=1000, k=32, reals=64, path="random", precision="fp32", warm=False),
        # the large 3D reservoir grid: anisotropic, 5,000 data, 48 neighbours
        # and 256 realizations
        dict(name="reservoir_200x200x100", kind="plan", nx=200, ny=200, nz=100, vario="exp", range=50.0, ratio=2.0,
             rz=5.0, nugget=0.05, ball=1.0, ndata=5000, k=48, reals=256, path="random", precision="fp32", warm=False),
        # the largest grid, unconditional, solved from the learned warm start
        dict(name="learned_256x256x256", kind="plan", nx=256, ny=256, nz=256, vario="sph", range=40.0, ratio=2.0,
             rz=8.0, nugget=0.1, ball=1.0, ndata=0, k=32, reals=64, path="random", precision="fp32", warm=True),
        # many uneven 2D / 3D domains with their own models in one batch
        dict(name="batch_24_domains", kind="batch", domains=24, shapes=6, side0=32, side1=256, depth0=8, depth1=64,
             reals=8),
        # further realizations from a prepared plan, values left on the device
        dict(name="sweep_160x160x48_r100", kind="sweep", nx=160, ny=160, nz=48, vario="exp", range=30.0, ratio=2.0,
             rz=5.0, nugget=0.05, ball=1.0, ndata=500, k=24, reals=100, path="random", precision="fp32"),
        # posterior mean and variance: simple kriging from the data alone
        dict(name="posterior_500x500", kind="krige", nx=500, ny=500, nz=1, vario="exp", range=60.0, ratio=1.0,
             nugget=0.02, ndata=1000, k=10),
        # facies: three categories, conditional, separable indicator model
        dict(name="indicator_256x256", kind="indicator", nx=256, ny=256, nz=1, vario="sph", range=25.0, ratio=1.0,
             nugget=0.0, ball=0.0, ndata=300, k=20, cats=3, reals=32, path="random"),
        # two correlated variables, simple cokriging of a two-structure model
        dict(name="multivariate_160x160", kind="mv", nx=160, ny=160, nz=1, range=20.0, range2=8.0, ndata=200, k=16,
             vars=2, reals=16),
        # statistics of a large ensemble that stays on the device
        dict(name="statistics_1M_r100", kind="stats", nodes=1000000, reals=100),
        # one mini-batch of the warm-start network's training (loss, gradient)
        dict(name="training_16384_k32", kind="train", systems=16384, k=32),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, max_nodes, min_nodes=1500):
    """A 2D or 3D grid of uneven sides, node count spread over its logarithm."""
    n = math.exp(rng.uniform(math.log(min_nodes), math.log(max_nodes)))
    if rng.random() < 0.5:
        nx = max(8, int(math.sqrt(n) * rng.uniform(0.7, 1.4)))
        return dict(nx=nx, ny=max(8, int(n / nx)), nz=1)
    nz = rng.randint(4, max(5, min(100, int(round(n ** (1 / 3))))))
    nx = max(8, int(math.sqrt(n / nz) * rng.uniform(0.7, 1.4)))
    return dict(nx=nx, ny=max(8, int(n / nz / nx)), nz=nz)


def draw(rng):
    kind = rng.choice(["rand", "plan", "plan", "plan", "learned", "batch", "sweep", "krige", "indicator", "mv",
                       "stats", "train"])
    if kind == "rand":
        return dict(kind="rand", **_grid(rng, 20000, 400), vario=rng.choice(["sph", "exp"]),
                    range=round(rng.uniform(5, 20), 2), ratio=1.0, nugget=round(rng.uniform(0, 0.1), 3), ball=0.0,
                    ndata=rng.choice([0, rng.randint(1, 100)]), k=rng.randint(4, 16), reals=rng.randint(1, 8),
                    path="random", precision="fp64")
    if kind in ("plan", "learned", "sweep"):
        g = _grid(rng, 1500000)
        n = g["nx"] * g["ny"] * g["nz"]
        flat = g["nz"] == 1
        case = dict(kind="sweep" if kind == "sweep" else "plan", **g, vario=rng.choice(["sph", "exp"]),
                    range=round(rng.uniform(8, 40), 2), ratio=1.0 if flat else round(rng.uniform(1, 3), 2),
                    rz=round(rng.uniform(3, 10), 2),
                    nugget=round(rng.uniform(0.0, 0.1), 3), ball=0.0 if flat else 1.0,
                    ndata=rng.choice([0, rng.randint(1, 2000)]), k=rng.choice([8, 12, 16, 20, 26, 32, 40, 48, 60]),
                    reals=_logint(rng, 1, max(1, min(256, 150000000 // n))),
                    path="linear" if kind == "plan" and flat and n < 100000 and rng.random() < 0.3 else "random",
                    precision="fp64" if n < 30000 and rng.random() < 0.3 else "fp32")
        if kind != "sweep":
            case["warm"] = kind == "learned" and case["precision"] == "fp32"
        return case
    if kind == "batch":
        s1 = rng.randint(40, 200)
        return dict(kind="batch", domains=rng.randint(1, 24), shapes=rng.randint(0, 10 ** 6), side0=rng.randint(8, 32),
                    side1=s1, depth0=3, depth1=rng.randint(6, 40), reals=_logint(rng, 1, 32))
    if kind == "krige":
        g = _grid(rng, 250000)
        return dict(kind="krige", **{**g, "nz": min(g["nz"], 8)}, vario=rng.choice(["sph", "exp"]),
                    range=round(rng.uniform(10, 60), 2), ratio=1.0, nugget=round(rng.uniform(0.0, 0.1), 3),
                    ndata=_logint(rng, 20, 3000), k=rng.randint(4, 32))
    if kind == "indicator":
        return dict(kind="indicator", **_grid(rng, 200000), vario=rng.choice(["sph", "exp"]),
                    range=round(rng.uniform(8, 25), 2), ratio=1.0, nugget=round(rng.uniform(0.0, 0.1), 3), ball=0.0,
                    ndata=rng.choice([0, rng.randint(10, 500)]), k=rng.randint(6, 32), cats=rng.randint(2, 6),
                    reals=_logint(rng, 1, 64), path="random")
    if kind == "mv":
        L = rng.randint(2, 4)
        g = _grid(rng, 40000)
        return dict(kind="mv", **g, range=round(rng.uniform(8, 20), 2), range2=round(rng.uniform(4, 8), 2),
                    ndata=rng.choice([0, rng.randint(1, 200)]), k=rng.randint(4, 64 // L), vars=L,
                    reals=_logint(rng, 1, 32))
    if kind == "stats":
        r = _logint(rng, 2, 1000)
        return dict(kind="stats", nodes=_logint(rng, 1000, min(4000000, 200000000 // r)), reals=r)
    return dict(kind="train", systems=_logint(rng, 500, 65536), k=rng.randint(8, 48))


# ------------------------------------------------------------------ inputs
def _dims(c):
    return (c["nx"], c["ny"]) if c["nz"] == 1 else (c["nx"], c["ny"], c["nz"])


def _nodes(c):
    return c["nx"] * c["ny"] * c["nz"]


def _ball(c):
    """The model's ellipsoid: ranges r, r / ratio (and rz along z) turned by
    30 degrees about z, or the ball of radius r."""
    dim = len(_dims(c))
    if c["ratio"] == 1.0:
        return geosgs.MetricBall((c["range"],) * dim)
    r = (c["range"], c["range"] / c["ratio"], c["rz"])
    return geosgs.MetricBall(r[:dim], geosgs.RotZ(30.0))


def _data(c, seed):
    """Coordinates and standard normal values; the smooth model's data sit at
    distinct cell centres, the others anywhere in the box."""
    dims = np.asarray(_dims(c), dtype=np.float64)
    rng = np.random.default_rng(1000 + seed)
    n = c["ndata"]
    if c.get("vario") == "gau":
        cells = rng.choice(_nodes(c), min(n, _nodes(c)), replace=False)
        xyz = np.stack(np.unravel_index(cells, _dims(c)[::-1])[::-1], axis=1) + 0.5
    else:
        xyz = rng.uniform(0.0, 1.0, (n, len(dims))) * dims
    return xyz, rng


def _method(c, seed, **kw):
    path = geosgs.LinearPath() if c.get("path") == "linear" else geosgs.RandomPath(seed)
    nb = "range"
    if c.get("ball", 0.0) == 1.0:
        nb = _ball(c)
    elif c.get("ball", 0.0) > 0.0:
        nb = geosgs.MetricBall(c["ball"])
    return geosgs.GPUSEQSIM(path=path, maxneighbors=c["k"], neighborhood=nb, **kw)


def _model(c):
    return VARIOS[c["vario"]](_ball(c), sill=1.0, nugget=c["nugget"])


def _gaussian(c, seed, **kw):
    """(process, grid, data, method) of a univariate case."""
    data = None
    if c["ndata"]:
        xyz, rng = _data(c, seed)
        data = geosgs.georef({"Z": rng.standard_normal(len(xyz))}, xyz)
    return (geosgs.GaussianProcess(_model(c), 0.0), geosgs.CartesianGrid(_dims(c)), data,
            _method(c, seed, precision=c.get("precision", "fp64"), **kw))


def _batch_items(c, seed):
    """Grids, models and neighbourhoods from the case's `shapes`, data and
    paths from the seed."""
    shape, rng = np.random.default_rng(c["shapes"]), np.random.default_rng(2000 + seed)
    for d in range(c["domains"]):
        dims = [int(shape.integers(c["side0"], c["side1"] + 1)) for _ in range(2)]
        if shape.random() < 0.5:
            dims.append(int(shape.integers(c["depth0"], c["depth1"] + 1)))
        cls = VARIOS[("sph", "exp", "gau")[int(shape.integers(3))]]
        gau = cls is VARIOS["gau"]
        model = cls(range=float(shape.uniform(5.0, 80.0)), sill=1.0,
                    nugget=float(shape.uniform(0.12, 0.2) if gau else shape.uniform(0.0, 0.1)))
        nd, k = int(shape.integers(0, 501)), int(shape.choice([8, 16, 32, 48]))
        data = None
        if nd:
            data = geosgs.georef({"Z": rng.standard_normal(nd)}, rng.uniform(0.0, 1.0, (nd, len(dims))) * dims)
        yield (geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid(tuple(dims)), data,
               geosgs.GPUSEQSIM(path=geosgs.RandomPath(100 * seed + d), maxneighbors=k, neighborhood="range"))


def _probabilities(c):
    p = np.arange(c["cats"], 0, -1, dtype=np.float64)
    return p / p.sum()


def _coregionalization(c):
    """Two spherical structures with their own ranges and full-rank
    coregionalization matrices."""
    L = c["vars"]
    i = np.arange(L)
    near = 0.8 ** np.abs(i[:, None] - i[None, :])
    dim = len(_dims(c))
    return geosgs.LinearCoregionalization([
        (0.7 * near, geosgs.SphericalVariogram(geosgs.MetricBall((c["range"],) * dim), sill=1.0)),
        (0.3 * np.eye(L) + 0.05, geosgs.SphericalVariogram(geosgs.MetricBall((c["range2"],) * dim), sill=1.0))])


def _training(c, seed):
    """Features of the systems (lags in the model's frame, covariance,
    nugget, family), neighbour counts and target weights, on the device."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    S, k = c["systems"], c["k"]
    u = torch.randn((S, k, 3), generator=g, device="cuda") * 0.2
    h = u.norm(dim=2)
    nugget = torch.rand((S, 1), generator=g, device="cuda") * 0.2
    family = torch.randint(0, 3, (S, 1), generator=g, device="cuda")
    sph, ex, ga = torch.where(h < 1, 1.5 * h - 0.5 * h ** 3, torch.ones_like(h)), 1 - torch.exp(-3 * h), \
        1 - torch.exp(-3 * h * h)
    cov = 1 - (nugget + (1 - nugget) * torch.where(family == 0, sph, torch.where(family == 1, ex, ga)))
    feat = torch.stack([u[..., 0], u[..., 1], u[..., 2], h, cov, nugget.expand(S, k),
                        (family == 1).float().expand(S, k), (family == 2).float().expand(S, k)], dim=2)
    count = torch.where(torch.rand(S, generator=g, device="cuda") < 0.9, k,
                        torch.randint(1, k + 1, (S,), generator=g, device="cuda")).to(torch.int32)
    live = torch.arange(k, device="cuda")[None, :] < count[:, None]
    target = torch.where(live, torch.softmax(-4 * h + 0.5 * torch.randn((S, k), generator=g, device="cuda"), dim=1), 0)
    params = torch.from_numpy(learned.init_params(seed)).cuda()
    return params, (feat * live[..., None]).contiguous(), count, target.contiguous()


def _ensemble(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    stride = (c["reals"] + 3) // 4 * 4
    return torch.randn((c["nodes"], stride), generator=g, device="cuda"), stride


# ------------------------------------------------------------- preparation
def prepare(case, seed):
    kind, s = case["kind"], dict(case=case, kind=case["kind"], seed=seed)
    if kind == "rand":
        s["args"] = _gaussian(case, seed)
    elif kind in ("plan", "sweep"):
        warm = case.get("warm", False)
        s["problem"] = geosgs.build_problem(*_gaussian(case, seed, **({"warm_start": True} if warm else {})))
        s["network"] = learned.init_params(seed) if warm else None
        if kind == "sweep":
            s["plan"] = geosgs.Plan(*s["problem"]).prepare()
            s["values"] = _values(s["plan"], case)
            s["stream"] = torch.cuda.Stream()
            s["stream"].wait_stream(torch.cuda.current_stream())
    elif kind == "batch":
        s["problems"] = [geosgs.build_problem(*item) for item in _batch_items(case, seed)]
    elif kind == "krige":
        s["args"] = _gaussian(case, seed)[:3]
    elif kind == "indicator":
        cat = None
        xyz, rng = _data(case, seed)
        data = None
        if case["ndata"]:
            cat = rng.choice(case["cats"], case["ndata"], p=_probabilities(case)).astype(np.int32)
            cat[:case["cats"]] = np.arange(case["cats"])  # every category occurs
            data = geosgs.georef({"facies": cat}, xyz)
        s["prob"], s["cat"] = _probabilities(case), cat
        proc = geosgs.IndicatorProcess(_model(case), prob=tuple(s["prob"]))
        s["problem"] = geosgs.build_problem(proc, geosgs.CartesianGrid(_dims(case)), data, _method(case, seed))
    elif kind == "mv":
        func = _coregionalization(case)
        s["mean"], s["coef"] = np.arange(case["vars"], dtype=np.float64), func.coef
        data, s["dval"] = None, None
        if case["ndata"]:
            xyz, rng = _data(case, seed)
            s["dval"] = rng.standard_normal((case["ndata"], case["vars"])) + s["mean"]
            data = geosgs.georef({"v%d" % a: s["dval"][:, a] for a in range(case["vars"])}, xyz)
        s["problem"] = geosgs.build_problem(geosgs.GaussianProcess(func, s["mean"]), geosgs.CartesianGrid(_dims(case)),
                                            data, _method(case, seed))
    elif kind == "stats":
        s["values"], s["stride"] = _ensemble(case, seed)
    else:
        s["train"] = _training(case, seed)
    return s


def _values(plan, case):
    rows = (case["reals"] + 3) // 4 * 4
    return torch.empty((plan.N, rows), dtype=torch.float64 if plan.values_fp64() else torch.float32, device="cuda")


# ---------------------------------------------------------------- one pass
def run(s):
    kind, case, seed = s["kind"], s["case"], s["seed"]
    if kind == "rand":
        process, grid, data, method = s["args"]
        ens = geosgs.rand(np.random.default_rng(seed), process, grid, case["reals"], data=data, method=method)
        return [next(iter(real.values())) for real in ens]
    if kind == "plan":
        plan = geosgs.Plan(*s["problem"])
        if s["network"] is not None:
            plan.set_network(s["network"])
        plan.prepare()
        values = _values(plan, case)
        plan.simulate_device(case["reals"], None, seed, values)
        plan.close()
        return values
    if kind == "sweep":
        with torch.cuda.stream(s["stream"]):
            s["plan"].simulate_device(case["reals"], None, seed, s["values"], stream=s["stream"].cuda_stream)
        return s["values"]
    if kind == "batch":
        batch = geosgs.Batch(s["problems"]).prepare()
        rows, wide = (case["reals"] + 3) // 4 * 4, batch.values_fp64()
        values = torch.empty((batch.nnodes, rows), dtype=torch.float64 if wide else torch.float32, device="cuda")
        batch.simulate_device(case["reals"], seed, values)
        out = []
        for d in range(batch.ndomains):
            v = values[int(batch.first[d]):int(batch.first[d] + batch.sizes[d])]
            # in a batch with FP64 rows the domains that keep FP32 values use
            # the first half of theirs
            out.append(v if not wide or batch.domain_values_fp64(d) else v.view(torch.float32)[:, :rows])
        batch.close()
        return out
    if kind == "krige":
        return list(geosgs.posterior(*s["args"], maxneighbors=case["k"]))
    if kind == "indicator":
        plan = geosgs.Plan(*s["problem"]).set_indicator(s["prob"], s["cat"]).prepare()
        out = plan.simulate_indicator(case["reals"], seed=seed)
        plan.close()
        return out
    if kind == "mv":
        plan = geosgs.Plan(*s["problem"]).set_multivariate(s["mean"], s["coef"], s["dval"]).prepare()
        out = plan.simulate_multivariate(case["reals"], seed=seed)
        plan.close()
        return out
    if kind == "stats":
        v, r, stride = s["values"], case["reals"], s["stride"]
        mean, var = ensemble.mean_var(v, r, stride)
        return [mean, var, ensemble.quantile(v, r, QUANTILES, stride), ensemble.cdf(v, r, THRESHOLDS, stride)]
    loss, grad = learned.loss_and_grad(*s["train"], torch)
    return [loss, grad]


# --------------------------------------------------------------------- work
def work(case):
    """Inputs read once and outputs written once; per kriging system a
    Cholesky factorization and its solves, per value a dot product."""
    kind = case["kind"]
    if kind == "stats":
        n, r = case["nodes"], case["reals"]
        return {"bytes": 4.0 * n * r + 8.0 * n * (2 + len(QUANTILES) + len(THRESHOLDS)),
                "flops": n * r * (4.0 + len(THRESHOLDS) + math.log2(max(2, r)))}
    if kind == "train":
        S, k = case["systems"], case["k"]
        return {"bytes": 4.0 * S * (9 * k + 1) + 8.0 * learned.NPARAMS, "flops": 3 * 2.0 * S * k * (8 * 32 + 32 * 32 + 32)}
    if kind == "batch":
        items = list(_batch_items(case, 0))
        n = sum(g.nelements() for _, g, _, _ in items)
        nd = sum(0 if d is None else d.nrow() for _, _, d, _ in items)
        rows = case["reals"]
        solve = sum(g.nelements() * _system_flops(m.maxneighbors) for _, g, _, m in items)
        dots = sum(2.0 * g.nelements() * m.maxneighbors for _, g, _, m in items)
        return {"bytes": 4.0 * n + 32.0 * nd + 4.0 * n * rows, "flops": solve + dots * rows}
    n, k = _nodes(case), case["k"]
    data = 32.0 * case["ndata"]
    if kind == "krige":
        return {"bytes": data + 16.0 * n, "flops": n * _system_flops(k)}
    R = case["reals"]
    if kind == "mv":
        L = case["vars"]
        return {"bytes": 4.0 * n + data * L + 8.0 * n * L * R,
                "flops": n * (_system_flops(k * L) + 2.0 * (L - 1) * (k * L) ** 2) + 2.0 * n * k * L * L * R}
    if kind == "indicator":
        return {"bytes": 4.0 * n + data + 4.0 * n * R, "flops": n * _system_flops(k) + float(n) * k * R}
    size = 8.0 if kind == "rand" or case["precision"] == "fp64" else 4.0
    dots = 2.0 * n * k * R
    if kind == "sweep":  # the plan's tables, then every value once
        return {"bytes": n * k * 12.0 + n * 24.0 + size * n * R, "flops": dots}
    return {"bytes": 4.0 * n + data + size * n * R, "flops": n * _system_flops(k) + dots}


def _system_flops(k):
    return k ** 3 / 3.0 + 2.0 * k * k


# -------------------------------------------------------- FP64 restatement
def _philox_normals(seed, ids, chunks):
    """Standard normals (len(ids) x 4 chunks): Philox4x32-10 on counter
    (node, realization / 4), Box-Muller on 24-bit uniforms."""
    mask = np.uint64(0xFFFFFFFF)
    ids = ids.astype(np.uint64)[:, None]
    shape = (ids.shape[0], chunks)
    c = [np.broadcast_to(ids & mask, shape), np.broadcast_to(ids >> np.uint64(32), shape),
         np.broadcast_to(np.arange(chunks, dtype=np.uint64)[None, :], shape), np.zeros(shape, dtype=np.uint64)]
    k0, k1 = np.uint64(seed & 0xFFFFFFFF), np.uint64(seed >> 32)
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ k0, b & mask, (a >> np.uint64(32)) ^ c[3] ^ k1, a & mask]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & mask, (k1 + np.uint64(0xBB67AE85)) & mask
    u = [((x >> np.uint64(9)).astype(np.float64) * 2.0 + 1.0) / 16777216.0 for x in c]
    r0, r1 = np.sqrt(-2.0 * np.log(u[0])), np.sqrt(-2.0 * np.log(u[2]))
    z = np.stack([r0 * np.cos(2 * np.pi * u[1]), r0 * np.sin(2 * np.pi * u[1]), r1 * np.cos(2 * np.pi * u[3]),
                  r1 * np.sin(2 * np.pi * u[3])], axis=2)
    return torch.from_numpy(z.reshape(shape[0], 4 * chunks)).cuda()


def _shape_of(lag, ball, vario):
    """The structure's normalized variogram (0 at 0, 1 at the sill) of lags."""
    dim = lag.shape[-1]
    R = torch.from_numpy(np.ascontiguousarray(ball.rotation[:dim, :dim])).cuda()
    r = torch.tensor(ball.padded_radii(dim)[:dim], dtype=torch.float64, device="cuda")
    h = ((lag @ R) / r).square().sum(-1).sqrt()
    if vario == "sph":
        return torch.where(h < 1, 1.5 * h - 0.5 * h ** 3, torch.ones_like(h))
    return 1 - torch.exp(-3 * h) if vario == "exp" else 1 - torch.exp(-3 * h * h)


def _covariance(lag, terms):
    """C_ab(h) of a sum of (matrix, ball, family, sill, nugget): [..., L, L]."""
    zero = (lag == 0).all(-1)
    out = 0.0
    for A, ball, vario, sill, nugget in terms:
        c = sill - torch.where(zero, 0.0, nugget + (sill - nugget) * _shape_of(lag, ball, vario))
        out = out + c[..., None, None] * A
    return out


def _distance2(lag, ball):
    """Squared search distance and its limit: every product and sum rounded
    in axis order; ball: a radius (isotropic), an ellipsoid, or None."""
    dim = lag.shape[-1]
    if ball is None or not isinstance(ball, geosgs.MetricBall):
        s = lag[..., 0] * lag[..., 0]
        for j in range(1, dim):
            s = s + lag[..., j] * lag[..., j]
        return s, math.inf if ball is None else ball * ball
    s = None
    for j in range(dim):
        u = lag[..., 0] * float(ball.rotation[0, j])
        for i in range(1, dim):
            u = u + lag[..., i] * float(ball.rotation[i, j])
        q = u * (1.0 / ball.radii[j])
        s = q * q if s is None else s + q * q
    return s, 1.0


def _cells(ids, dims):
    i = ids % dims[0]
    r = ids // dims[0]
    return torch.stack([i, r] if len(dims) == 2 else [i, r % dims[1], r // dims[1]], dim=-1)


def _neighbours(dims, rank, xyz, ball, k):
    """Per node the k nearest earlier nodes (rank given, None: data only) and
    data inside the ball, ordered by (distance, id): ids (-1: none)."""
    N, dim = int(np.prod(dims)), len(dims)
    out = torch.full((N, k), -1, dtype=torch.int64, device="cuda")
    offs = None
    if rank is not None:
        if isinstance(ball, geosgs.MetricBall):
            ext = np.sqrt(((ball.rotation[:dim, :dim] * np.asarray(ball.radii)[None, :dim]) ** 2).sum(1))
        else:
            ext = [ball] * dim
        e = [min(dims[j] - 1, int(math.floor(ext[j])) + 1) for j in range(dim)]
        o = torch.stack(torch.meshgrid(*[torch.arange(-x, x + 1, device="cuda") for x in e], indexing="ij"), -1)
        o = o.reshape(-1, dim)
        o = o[(o != 0).any(1)]
        d2, lim = _distance2(o.double(), ball)
        o, d2 = o[d2 <= lim], d2[d2 <= lim]
        mult = torch.tensor([1, dims[0], dims[0] * dims[-2]][:dim] if dim == 3 else [1, dims[0]], device="cuda")
        lin = (o * mult).sum(1)
        order = torch.argsort(lin)
        order = order[torch.argsort(d2[order], stable=True)]
        offs, od2, lin = o[order], d2[order], lin[order]
    size = torch.tensor(dims, device="cuda")
    chunk = max(256, 40000000 // max(1 if offs is None else len(offs), 1 if xyz is None else 4 * len(xyz)))
    for a in range(0, N, chunk):
        ids = torch.arange(a, min(a + chunk, N), device="cuda")
        cell = _cells(ids, dims)
        gid = torch.full((len(ids), k + 1), -1, dtype=torch.int64, device="cuda")
        gd = torch.full((len(ids), k + 1), math.inf, dtype=torch.float64, device="cuda")
        if offs is not None:
            c = cell[:, None, :] + offs[None]
            ok = ((c >= 0) & (c < size)).all(2)
            del c
            nb = torch.where(ok, ids[:, None] + lin[None], 0)
            ok &= rank[nb] < rank[ids][:, None]
            place = torch.cumsum(ok, 1, dtype=torch.int32) - 1
            ok &= place < k
            row, col = ok.nonzero(as_tuple=True)
            gid[row, place[row, col].long()] = nb[row, col]
            gd[row, place[row, col].long()] = od2[col]
            del nb, ok, place
        gid, gd = gid[:, :k], gd[:, :k]
        if xyz is not None:
            d2, lim = _distance2(xyz[None] - (cell.double() + 0.5)[:, None, :], ball)
            d2 = torch.where(d2 <= lim, d2, math.inf)
            dd, di = torch.sort(d2, dim=1, stable=True)
            dd, di = dd[:, :k], di[:, :k]
            both = torch.cat([gd, dd], 1)
            idb = torch.cat([gid, torch.where(dd < math.inf, di + N, -1)], 1)
            gd, o = torch.sort(both, dim=1, stable=True)
            gid = torch.gather(idb, 1, o)[:, :k]
        out[ids] = gid
    return out


def _systems(dims, nb, xyz, dval, mean, terms):
    """Per node, simple (co)kriging of the L variables: weights [N, k, L, L],
    constant [N, L] (mean and data folded in), factor of the conditional
    covariance [N, L, L], whether kriged."""
    N, k = nb.shape
    L = terms[0][0].shape[0]
    C0 = _covariance(torch.zeros((1, len(dims)), dtype=torch.float64, device="cuda"), terms)[0]
    tau = 1e-10 * float(C0.diagonal().max())
    W = torch.zeros((N, k, L, L), dtype=torch.float64, device="cuda")
    cst = mean.expand(N, L).clone()
    F = torch.linalg.cholesky(C0).expand(N, L, L).clone()
    kriged = torch.zeros(N, dtype=torch.bool, device="cuda")
    chunk = max(64, 60000000 // (k * L) ** 2)
    for a in range(0, N, chunk):
        ids = torch.arange(a, min(a + chunk, N), device="cuda")
        n, q = len(ids), nb[ids]
        live = q >= 0
        x = _cells(torch.where(q < N, q, 0).clamp(min=0), dims).double() + 0.5
        if xyz is not None:
            x = torch.where((q >= N)[..., None], xyz[(q - N).clamp(min=0)], x)
        x0 = _cells(ids, dims).double() + 0.5
        K = _covariance(x[:, :, None] - x[:, None, :], terms).permute(0, 1, 3, 2, 4).reshape(n, k * L, k * L)
        c = _covariance(x - x0[:, None], terms).reshape(n, k * L, L)
        on = live.repeat_interleave(L, 1)
        K = torch.where(on[:, :, None] & on[:, None, :], K, torch.eye(k * L, dtype=torch.float64, device="cuda"))
        c = torch.where(on[..., None], c, 0.0)
        chol, info = torch.linalg.cholesky_ex(K)
        good = (info == 0) & (chol.diagonal(dim1=1, dim2=2).square().nan_to_num().min(1)[0] > tau) & live.any(1)
        chol = torch.where(good[:, None, None], chol, torch.eye(k * L, dtype=torch.float64, device="cuda"))
        lam = torch.cholesky_solve(c, chol)
        S = C0 - c.transpose(1, 2) @ lam
        f = S.clamp(min=0).sqrt() if L == 1 else torch.linalg.cholesky_ex(S)[0]
        lam = torch.where(good[:, None, None], lam, 0.0).reshape(n, k, L, L)
        F[ids] = torch.where(good[:, None, None], f, F[ids])
        shift = -(lam * mean[None, None, :, None]).sum((1, 2))
        if xyz is not None:
            v = torch.where((q >= N)[..., None], dval[(q - N).clamp(min=0)], 0.0)
            shift = shift + (lam * v[..., None]).sum((1, 2))
        cst[ids] = cst[ids] + shift
        W[ids], kriged[ids] = lam, good
    return W, cst, F, kriged


def _sweep(nb, W, cst, F, z):
    """Values [N, L, R] by dependency levels of the grid neighbours; z alike."""
    N, k = nb.shape
    grid = (nb >= 0) & (nb < N)
    idx = torch.where(grid, nb, 0)
    W = torch.where(grid[..., None, None], W, 0.0)
    level = torch.zeros(N, dtype=torch.int32, device="cuda")
    while True:
        new = torch.where(grid, level[idx] + 1, 0).max(1)[0]
        if torch.equal(new, level):
            break
        level = new
    order = torch.argsort(level, stable=True)
    counts = torch.bincount(level.long()).cpu().tolist()
    V = torch.zeros((N,) + tuple(z.shape[1:]), dtype=torch.float64, device="cuda")
    step = max(1, 50000000 // (k * z.shape[1] * z.shape[2]))
    p = 0
    for m in counts:
        for a in range(p, p + m, step):
            g = order[a:min(a + step, p + m)]
            mu = torch.einsum("njbt,njbr->ntr", W[g], V[idx[g]])
            V[g] = mu + cst[g][..., None] + torch.einsum("ntu,nur->ntr", F[g], z[g])
        p += m
    return V


def _search_ball(c):
    if c.get("ball", 0.0) == 1.0 and c["ratio"] != 1.0:
        return _ball(c)
    return float(c["ball"]) if c.get("ball", 0.0) > 1.0 else float(c["range"])


def exact(case, seed):
    kind = case["kind"]
    if kind == "stats":
        v, _ = _ensemble(case, seed)
        v = v[:, :case["reals"]].double()
        R = case["reals"]
        s = torch.sort(v, dim=1)[0]
        quant = []
        for p in QUANTILES:
            h = (R - 1) * p
            lo = min(int(math.floor(h)), R - 1)
            hi = min(lo + 1, R - 1)
            quant.append(s[:, lo] + (h - math.floor(h)) * (s[:, hi] - s[:, lo]))
        return [v.mean(1), v.var(1), torch.stack(quant, 1),
                torch.stack([(v <= x).double().mean(1) for x in THRESHOLDS], 1)]
    if kind == "train":
        params, feat, count, target = _training(case, seed)
        p = params.double().requires_grad_(True)
        w1, b1, w2a, w2b, b2, w3, b3 = torch.split(p, [256, 32, 1024, 1024, 32, 32, 1])
        live = (torch.arange(case["k"], device="cuda")[None, :] < count[:, None]).double()
        n = count.double()[:, None]
        h = torch.relu(feat.double() @ w1.view(32, 8).T + b1) * live[..., None]
        u = (h.sum(1) / n) @ w2b.view(32, 32).T + b2
        y = torch.relu(h @ w2a.view(32, 32).T + u[:, None]) @ w3 + b3
        loss = (((y - target.double()) * live).square().sum(1, keepdim=True) / n).sum()
        loss.backward()
        return [loss.detach(), p.grad]
    # whole simulations: up to a few 10^5 nodes in plain torch; categories are
    # whole numbers, and a batch is its domains
    if kind in ("batch", "indicator") or _nodes(case) > 300000 or _nodes(case) * case.get("reals", 1) > 20000000:
        return None
    dims, N = _dims(case), _nodes(case)
    xyz = dval = None
    if kind == "mv":
        func = _coregionalization(case)
        L, mean = case["vars"], torch.arange(case["vars"], dtype=torch.float64, device="cuda")
        terms = [(torch.from_numpy(A).cuda(), g.ball, "sph", 1.0, 0.0) for A, g in zip(func.coef, func.structures())]
        ball = max(case["range"], case["range2"])
    else:
        L, mean = 1, torch.zeros(1, dtype=torch.float64, device="cuda")
        one = torch.ones((1, 1), dtype=torch.float64, device="cuda")
        terms = [(one, _ball(case), case["vario"], 1.0, case["nugget"])]
        ball = None if kind == "krige" else _search_ball(case)
    if case["ndata"]:
        at, rng = _data(case, seed)
        xyz = torch.from_numpy(np.ascontiguousarray(at, dtype=np.float64)).cuda()
        if kind == "mv":
            dval = torch.from_numpy(rng.standard_normal((len(at), L))).cuda() + mean
        else:
            dval = torch.from_numpy(rng.standard_normal(len(at))).cuda()[:, None]
    if kind == "krige":
        nb = _neighbours(dims, None, xyz, ball, min(case["k"], case["ndata"]))
        _, cst, F, kriged = _systems(dims, nb, xyz, dval, mean, terms)
        nan = torch.full((N,), math.nan, dtype=torch.float64, device="cuda")
        return [torch.where(kriged, cst[:, 0], nan), torch.where(kriged, F[:, 0, 0].square(), nan)]
    rank = torch.arange(N, device="cuda")
    if case.get("path") != "linear":
        rank[torch.from_numpy(geosgs.RandomPath(seed).permutation(N).astype(np.int64)).cuda()] = \
            torch.arange(N, device="cuda")
    nb = _neighbours(dims, rank, xyz, ball, min(case["k"], N))
    W, cst, F, _ = _systems(dims, nb, xyz, dval, mean, terms)
    # rand() draws the simulation's seed from the generator it is given
    sim = int(np.random.default_rng(seed).integers(0, 2 ** 63 - 1)) if kind == "rand" else seed
    R = case["reals"]
    z = torch.stack([_philox_normals(sim, np.arange(N) + a * N, (R + 3) // 4) for a in range(L)], dim=1)
    V = _sweep(nb, W, cst, F, z)
    if kind == "mv":
        return V[..., :R].permute(2, 1, 0).contiguous()
    if kind == "rand":
        return [V[:, 0, r].contiguous() for r in range(R)]
    return V[:, 0]
