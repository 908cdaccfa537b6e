"""Performance cases of the Gaussian kernel matrix-vector product: what a user's program has this framework do.

A case is a dict of plain values; `kind` names the entry point that is timed:

  one_shot   engine.kmvm: tree, interaction lists and product in one call (the call bench.py times)
  operator   FFM(X, ...) @ b on a new operator, as in the README: the tree is built in the pass
  kept       op @ b on an operator that the program keeps, as every iteration of a CG solve does
  host       engine.kmvm_host: pinned host tensors in, host tensor out
  falkon     F3MGaussianKernel.dmmv: K(X,C)^T (K(X,C) v), one iteration of FALKON
  dense      benchmark_matmul @ b and FFM.grad: the exact product and its lengthscale gradient

Points are drawn as the repository's tests and benchmark draw them: `uniform` on [0, side]^d, `normal` N(0, I_d), and
`clustered` (a mixture of ten Gaussians with means U[-5,5]^d and standard deviations U[0.3,1]).
"""
import math

import torch

from f3m_b200 import engine
from f3m_b200.FFM_classes import FFM, benchmark_matmul
from f3m_b200.solvers import F3MGaussianKernel

DEVICE = "cuda:0"
SQRT12 = 12 ** 0.5


def _case(name, kind, d, n, *, m=0, r=1, dist="uniform", side=1.0, ls=1.0, leaf=1000.0, nodes=64, small=0):
    """m = 0: the sources are the targets.  small = 0: small_field_points equals the node count."""
    c = dict(kind=kind, d=d, n=n, m=m, r=r, dist=dist, side=side, ls=ls, leaf=leaf, nodes=nodes, small=small or nodes)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest calls: a kernel matrix of a few thousand points with the operator's default arguments
        _case("one_shot_2e3", "one_shot", 3, 2000, small=1000),
        # one CG iteration of a GP on a data set of ordinary size (odd count), tree kept between products
        _case("kept_2e4", "kept", 3, 20011, small=1000),
        # the README's use, at the size of the smallest benchmark configuration: build the operator, multiply once
        _case("operator_1e5", "operator", 3, 100_000),
        # K(X, Y) b of two planar point sets with three columns: prediction at other points than the training set
        _case("xy_2d_3col", "one_shot", 2, 150_001, m=60_007, r=3, ls=0.5, leaf=200.0, nodes=36),
        # marginal likelihood of a GP on a data set that the exact op still handles: product and lengthscale gradient
        _case("dense_value_grad", "dense", 3, 20_000, r=3),
        # one FALKON iteration: a million points against Nystrom centres, kernel defaults (leaf size 4^d)
        _case("falkon_2e6_2e4", "falkon", 3, 2_000_000, m=20_000, leaf=64.0),
        # a lengthscale that is short against the domain, 5 nodes per dimension, unit-variance scaling
        _case("short_ls_4e6", "one_shot", 3, 4_000_037, side=SQRT12, ls=0.1, nodes=125),
        # uneven occupancy: the benchmark's mixture
        _case("clustered_1e7", "one_shot", 3, 10_000_000, dist="clustered", ls=0.5, nodes=216),
        # several right-hand sides in four and five dimensions, the benchmark's node counts
        _case("normal4_8col", "one_shot", 4, 1_000_000, r=8, dist="normal", nodes=81),
        _case("normal5_8col", "one_shot", 5, 1_000_000, r=8, dist="normal", nodes=243),
        # a caller whose data live on the host
        _case("host_1e7", "host", 3, 10_000_000, side=SQRT12, nodes=216),
        # the headline benchmark
        _case("uniform_1e8", "one_shot", 3, 100_000_000, side=SQRT12, nodes=216),
    ]


def _log_int(rng, lo, hi):
    """An integer between lo and hi, even over the logarithm, as often odd as even."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one_shot", "one_shot", "one_shot", "operator", "kept", "host", "falkon", "dense", "columns", "columns"])
    ls3 = math.exp(rng.uniform(math.log(0.1), math.log(10.0)))
    if kind == "dense":
        d = rng.randint(1, 5)
        return _case(None, "dense", d, _log_int(rng, 2000, 40_000), r=rng.choice([1, 2, 3, 8]), ls=round(rng.uniform(0.3, 2.0), 4))
    if kind == "falkon":
        return _case(None, "falkon", 3, _log_int(rng, 1e5, 1e7), m=_log_int(rng, 2000, 1e5), leaf=64.0, ls=round(rng.uniform(0.5, 2.0), 4))
    if kind == "columns":
        d = rng.choice([4, 5])
        return _case(None, "one_shot", d, _log_int(rng, 2e4, 1e6), r=rng.randint(2, 8), dist=rng.choice(["normal", "uniform"]),
                     ls=round(rng.uniform(0.8, 2.0), 4), nodes=rng.choice([2, 3]) ** d)
    if kind == "one_shot" and rng.random() < 0.35:
        # two point sets, one to three dimensions, one to four columns
        d = rng.randint(1, 3)
        p = {1: (8, 8), 2: (4, 8), 3: (3, 6)}[d]
        return _case(None, "one_shot", d, _log_int(rng, 2000, 2e6), m=_log_int(rng, 2000, 2e6), r=rng.randint(1, 4),
                     ls=round(rng.uniform(0.2, 2.0), 4), leaf=rng.choice([200.0, 1000.0]), nodes=rng.randint(*p) ** d)
    # one point set in three dimensions, one column
    top = {"one_shot": 3e7, "operator": 5e6, "kept": 5e6, "host": 2e7}[kind]
    p = rng.choice([3, 4, 5, 6])
    dist = rng.choice(["uniform", "uniform", "clustered", "normal"])
    # at unit side the lengthscale is near one; with unit-variance scaling, and for data without a cube, it spans 0.1 to 10
    wide = dist != "uniform" or rng.random() < 0.6
    return _case(None, kind, 3, _log_int(rng, 1500, top), dist=dist, side=SQRT12 if wide else 1.0,
                 ls=round(ls3 if wide else rng.uniform(0.5, 2.0), 4), nodes=p ** 3, small=rng.choice([p ** 3, 1000]))


def _points(case, n, seed, shift=0.0):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    d = case["d"]
    if case["dist"] == "uniform":
        return torch.empty(n, d, device=DEVICE).uniform_(0.0, case["side"], generator=g)
    X = torch.randn(n, d, device=DEVICE, generator=g)
    if case["dist"] == "clustered":
        gm = torch.Generator().manual_seed(7)   # the mixture itself is the same for every seed, as in the benchmark
        means = (torch.rand(10, d, generator=gm) * 10 - 5).to(DEVICE)
        std = (torch.rand(10, generator=gm) * 0.7 + 0.3).to(DEVICE)
        comp = torch.randint(0, 10, (n,), device=DEVICE, generator=g)
        X.mul_(std[comp, None]).add_(means[comp])
    return X


def _operator(case, X, Y):
    return FFM(X, Y, ls=case["ls"], min_points=case["leaf"], nr_of_interpolation=case["nodes"],
               small_field_points=case["small"], device=DEVICE)


def prepare(case, seed):
    kind, n, m = case["kind"], case["n"], case["m"]
    X = _points(case, n, 4 * seed)
    Y = _points(case, m, 4 * seed + 1) if m and kind != "falkon" else None
    g = torch.Generator(device=DEVICE).manual_seed(4 * seed + 2)
    b = torch.randn(m or n, case["r"], device=DEVICE, generator=g)
    s = dict(case=case, X=X, Y=Y, b=b,
             params=engine.make_params(case["ls"], case["leaf"], case["nodes"], False, 0.15, case["small"]))
    if kind == "kept":
        s["op"] = _operator(case, X, Y)
        s["op"].plan()          # the tree of a solve is built once, before its iterations
    elif kind == "host":
        s["X"] = torch.empty(X.shape, pin_memory=True).copy_(X)
        s["b"] = torch.empty(b.shape, pin_memory=True).copy_(b)
        s["out"] = torch.empty(n, case["r"], pin_memory=True)
    elif kind == "falkon":
        s["C"] = X[torch.randperm(n, device=DEVICE, generator=g)[:m]].contiguous()
        s["kernel"] = F3MGaussianKernel(case["ls"], min_points=case["leaf"], interpolation_nr=case["nodes"], device=DEVICE)
        s["kernel"].mmv(X, s["C"], b)   # a fit's first product builds both operators; its iterations reuse them
    elif kind == "dense":
        s["exact"] = benchmark_matmul(X, ls=case["ls"], device=DEVICE)
        s["op"] = _operator(case, X, None)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "one_shot":
        return engine.kmvm(s["X"], s["Y"], s["b"], s["params"])
    if kind == "operator":
        return _operator(case, s["X"], s["Y"]) @ s["b"]
    if kind == "kept":
        return s["op"] @ s["b"]
    if kind == "host":
        return engine.kmvm_host(s["X"], s["Y"], s["b"], s["params"], out=s["out"])
    if kind == "falkon":
        return s["kernel"].dmmv(s["X"], s["C"], s["b"], None)
    return s["exact"] @ s["b"], s["op"].grad(s["b"])


def work(case):
    """Inputs once and outputs once; the multiply-adds of interpolating every source onto, and every target from, its
    box's nodes (the exact op: distance, exponential and column sums of every pair, twice)."""
    d, n, r = case["d"], case["n"], case["r"]
    m = case["m"] or n
    sets = n * d if not case["m"] else (n + m) * d
    if case["kind"] == "dense":
        return {"bytes": 4 * (sets + m * r + 2 * n * r), "flops": 2.0 * n * m * (3 * d + 2 * r)}
    passes = 2 if case["kind"] == "falkon" else 1
    out = m if case["kind"] == "falkon" else n
    return {"bytes": 4 * (sets + m * r + out * r), "flops": passes * 2.0 * case["nodes"] * r * (n + m)}


def tolerance(case):
    """Float32 sums over a tree.  Measured over these cases and drawn ones: the same points given in another order (so that
    every sum runs in another order) 0.1e-6 to 0.5e-6 in the 2-norm and up to 5e-6 in single values; against the same
    algorithm in float64, 0.2e-6 to 0.75e-6 and up to 5.3e-6.  A kernel that is wide against the data (w = lengthscale over
    standard deviation of a coordinate) is worse conditioned: the result is the sum of b but for terms of the order of 1 / w^2,
    and where that sum is small the float32 product is 3e-6 (w = 3.5) to 8e-6 (w = 14) from the float64 one.  About four
    times that.  The exact op with its sums in another order: 0.6e-6, 2.6e-6."""
    spread = {"uniform": case["side"] / SQRT12, "normal": 1.0, "clustered": 3.3}[case["dist"]]
    w = case["ls"] / spread
    if case["kind"] == "dense":
        return {"rel": min(1e-5, max(2.5e-6, 3e-7 * w * w)), "max": 3e-5}
    rel = min(3e-5, max(3e-6, 1e-6 * w * w))
    return {"rel": rel, "max": 13 * rel}


def exact(case, seed):
    """Where every pair is summed directly: the dense op, and a product whose boxes are all small at the first level (the
    tree's own approximation is most of the distance of any other product from K b, so those have no such value)."""
    kind, n = case["kind"], case["n"]
    small = kind in ("one_shot", "kept") and not case["m"] and case["dist"] == "uniform" and n <= 4 * case["small"]
    if not (kind == "dense" or small) or n > 40_000:
        return None
    s = prepare(case, seed)
    X, b = s["X"].double(), s["b"].double()
    val = torch.empty_like(b)
    grad = torch.empty_like(b)
    ls = float(case["ls"])
    for i in range(0, n, 1000):
        D = torch.zeros(min(1000, n - i), n, dtype=torch.float64, device=X.device)
        for k in range(case["d"]):
            D += (X[i:i + 1000, None, k] - X[None, :, k]) ** 2
        K = torch.exp(D / (-2 * ls * ls))
        val[i:i + 1000] = K @ b
        if kind == "dense":
            grad[i:i + 1000] = (K * D) @ b / ls ** 3
    return (val, grad) if kind == "dense" else val
