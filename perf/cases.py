"""Performance cases of the level-wise tree build.

Each case is one call a user's program makes on the build path, with inputs on
the device as a build keeps them: leaf fits (weighted or unweighted batched
ridge), the soft oblique split search of one node or of a level, the routing of
a level's rows, hit-and-run sampling, and prediction with a built tree.  Sizes
follow the repository's workloads (``art.workloads``, ``art.serving``): nodes of
a few hundred to a few hundred thousand rows, d from 2 to 32, affine leaves and
quadratic leaves.

``listed`` are fixed cases, ``draw`` gives more of the same ranges, ``prepare``
makes what the caller holds before the call, ``run`` is one call, ``work`` the
bytes and operations it cannot do without, and ``exact`` the outputs in 64 bits
by plain torch.
"""

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = str(Path(__file__).resolve().parent.parent / "adaptive-regression-trees-art-_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from art.models import (  # noqa: E402
    AffineRidgeModel,
    PolynomialRidgeModel,
    segment_residuals,
    solve_weighted_ridge_batched,
)
from art.sampling import DevicePolytopes, hit_and_run_device  # noqa: E402
from art.splitters import SoftObliqueSplitter, split_level  # noqa: E402
from art.tree import LeafNode, RegressionTree, SplitNode, partition_rows  # noqa: E402

AFFINE, QUADRATIC = 0, 2  # the feature kinds of include/art_b200.h

# (d, feature kind) of the nodes a call mixes.  "job" kinds are a serving
# engine's jobs: quadratic leaves for d <= 8 and affine leaves above.
MIXES = {
    "small": ((2, AFFINE),),
    "jobs": ((2, QUADRATIC), (4, QUADRATIC), (8, QUADRATIC), (16, AFFINE), (32, AFFINE)),
    "narrow_jobs": ((2, QUADRATIC), (4, QUADRATIC), (16, AFFINE)),
    "wide_jobs": ((8, QUADRATIC), (32, AFFINE)),
    "weighted": ((8, AFFINE), (16, AFFINE), (8, QUADRATIC), (16, QUADRATIC)),
    "quadratic": ((8, QUADRATIC), (16, QUADRATIC)),
    "affine": ((16, AFFINE),),
}


def listed():
    return [
        # the root of a small tree: one call, little work, latency counts
        {"name": "fit one node", "op": "fit", "mix": "small", "nodes": 1, "n_min": 4096, "n_max": 4096,
         "weighted": False, "precision": "fp64", "shape": 1},
        # a serving tick: the leaf fits of a level of many jobs, from small
        # nodes to the roots of jobs just admitted
        {"name": "fit a level of jobs", "op": "fit", "mix": "jobs", "nodes": 301, "n_min": 450, "n_max": 400000,
         "weighted": False, "precision": "mixed", "shape": 2},
        # the batched weighted solve in its mixed form (bench.py's workload)
        {"name": "fit weighted mixed", "op": "fit", "mix": "weighted", "nodes": 8192, "n_min": 306, "n_max": 8192,
         "weighted": True, "precision": "mixed", "shape": 3},
        # quadratic leaves in the plain form, the API's default precision
        {"name": "fit quadratic fp64", "op": "fit", "mix": "quadratic", "nodes": 1021, "n_min": 306, "n_max": 8192,
         "weighted": True, "precision": "fp64", "shape": 4},
        # the split of one node, as a depth-first build asks for it
        {"name": "split one node", "op": "split", "mix": "small", "nodes": 1, "n_min": 4096, "n_max": 4096,
         "restarts": 1, "iters": 100, "anneal": 1.0, "temperature": 0.05, "hard": True, "device_start": False,
         "shape": 5},
        # a level searched from 16 restart normals with an annealed temperature
        {"name": "split a level, 16 restarts", "op": "split", "mix": "affine", "nodes": 256, "n_min": 256,
         "n_max": 16384, "restarts": 16, "iters": 30, "anneal": 0.1, "temperature": 0.2, "hard": True,
         "device_start": False, "shape": 6},
        # a serving tick's splits: nodes that fit the warp-per-restart form
        {"name": "split a level of jobs", "op": "split", "mix": "narrow_jobs", "nodes": 203, "n_min": 300,
         "n_max": 65000, "restarts": 1, "iters": 30, "anneal": 1.0, "temperature": 0.1, "hard": False,
         "device_start": True, "shape": 7},
        # ... and those that do not (d = 32, or quadratic models of d = 8)
        {"name": "split a wide level", "op": "split", "mix": "wide_jobs", "nodes": 149, "n_min": 300,
         "n_max": 120000, "restarts": 1, "iters": 15, "anneal": 1.0, "temperature": 0.1, "hard": False,
         "device_start": False, "shape": 8},
        # what follows a level's fits and splits: residuals and the partition
        {"name": "route a level", "op": "route", "mix": "jobs", "nodes": 307, "n_min": 450, "n_max": 400000,
         "shape": 9},
        # many chains, one polytope each (uniform sampling of a whole level)
        {"name": "sample many chains", "op": "sample", "dim": 8, "chains": 16384, "burn_in": 0, "thinning": 10,
         "rounds": 100, "injected": False, "shape": 10},
        # top-ups: few chains, many steps, with the caller's own draws
        {"name": "sample few chains", "op": "sample", "dim": 4, "chains": 61, "burn_in": 100, "thinning": 20,
         "rounds": 100, "injected": True, "shape": 11},
        # prediction of a test set by a built tree (host arrays in and out)
        {"name": "predict", "op": "predict", "dim": 8, "depth": 9, "kind": QUADRATIC, "points": 100003,
         "shape": 12},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["fit", "fit", "fit", "split", "split", "split", "route", "sample", "sample", "predict"])
    shape = rng.randrange(1, 1 << 30)
    if op == "fit":
        if rng.random() < 0.5:  # unweighted nodes of jobs, one to a level of them
            nodes = _log(rng, 1, 400)
            return {"op": op, "mix": rng.choice(["small", "jobs", "narrow_jobs", "wide_jobs"]), "nodes": nodes,
                    "n_min": 450, "n_max": _log(rng, 4096, 400000 if nodes < 300 else 200000), "weighted": False,
                    "precision": rng.choice(["fp64", "mixed"]), "shape": shape}
        nodes = _log(rng, 64, 6000)
        return {"op": op, "mix": rng.choice(["weighted", "quadratic"] if nodes < 2000 else ["weighted"]),
                "nodes": nodes, "n_min": 306, "n_max": _log(rng, 2048, 8192), "weighted": True,
                "precision": rng.choice(["fp64", "mixed"]), "shape": shape}
    if op == "split":
        which = rng.randrange(3)
        if which == 0:  # several restarts
            return {"op": op, "mix": rng.choice(["affine", "small"]), "nodes": _log(rng, 8, 200), "n_min": 256,
                    "n_max": _log(rng, 1024, 16384), "restarts": rng.choice([4, 8, 16]), "iters": rng.randint(15, 30),
                    "anneal": 0.1, "temperature": 0.2, "hard": True, "device_start": False, "shape": shape}
        if which == 1:  # one restart, narrow models
            return {"op": op, "mix": rng.choice(["small", "narrow_jobs", "affine"]), "nodes": _log(rng, 1, 250),
                    "n_min": 300, "n_max": _log(rng, 2048, 65000), "restarts": 1, "iters": rng.randint(15, 50),
                    "anneal": 1.0, "temperature": 0.1, "hard": bool(rng.randrange(2)),
                    "device_start": bool(rng.randrange(2)), "shape": shape}
        return {"op": op, "mix": "wide_jobs", "nodes": _log(rng, 4, 140), "n_min": 300, "n_max": _log(rng, 4096, 110000),
                "restarts": 1, "iters": rng.randint(8, 15), "anneal": 1.0, "temperature": 0.1, "hard": False,
                "device_start": False, "shape": shape}
    if op == "route":
        return {"op": op, "mix": rng.choice(["small", "jobs", "narrow_jobs", "wide_jobs"]), "nodes": _log(rng, 1, 300),
                "n_min": 450, "n_max": _log(rng, 4096, 400000), "shape": shape}
    if op == "sample":
        if rng.random() < 0.6:
            dim = rng.choice([2, 3, 5, 8, 16, 31, 64])
            return {"op": op, "dim": dim, "chains": _log(rng, 1000, 16384 if dim <= 8 else 4096), "burn_in": 0,
                    "thinning": 10, "rounds": rng.randint(40, 100), "injected": False, "shape": shape}
        return {"op": op, "dim": rng.choice([2, 4, 7, 8]), "chains": _log(rng, 1, 100), "burn_in": rng.randint(0, 200),
                "thinning": 20, "rounds": rng.randint(40, 100), "injected": True, "shape": shape}
    return {"op": op, "dim": rng.choice([2, 4, 8, 15]), "depth": rng.randint(4, 9), "kind": rng.choice([AFFINE, QUADRATIC]),
            "points": _log(rng, 1000, 100000), "shape": shape}


# ------------------------------------------------------------------ shapes
def _features(d, kind):
    return d + 1 if kind == AFFINE else 1 + d + d * (d + 1) // 2


def _nodes(case):
    """(dims, kinds, rows) of a case's nodes: the same for every seed."""

    rng = np.random.default_rng([case["shape"], 1])
    mix = MIXES[case["mix"]]
    pick = rng.integers(0, len(mix), case["nodes"])
    d = np.array([mix[i][0] for i in pick], dtype=np.int32)
    kind = np.array([mix[i][1] for i in pick], dtype=np.int32)
    lo, hi = math.log(case["n_min"]), math.log(max(case["n_max"], case["n_min"]))
    n = np.floor(np.exp(rng.uniform(lo, hi, case["nodes"])) + 1e-9).astype(np.int64)
    return d, kind, n


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _rand(g, *size):
    return torch.rand(size, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *size):
    return torch.randn(size, generator=g, device="cuda", dtype=torch.float64)


def _surface(X, g):
    """8 Gaussian bumps plus a tanh ridge on [-1, 1]^d (a serving job's target)."""

    d = X.shape[1]
    c, w = _rand(g, 8, d) * 2.0 - 1.0, (_rand(g, 8) * 0.5 + 0.1) * math.sqrt(d / 2.0)
    a, u = _randn(g, 8), _randn(g, d)
    b = _rand(g, 1) * 0.6 - 0.3
    r2 = (X * X).sum(1, keepdim=True) - 2.0 * X @ c.T + (c * c).sum(1)
    return (a * torch.exp(-r2 / (2.0 * w**2))).sum(1) + torch.tanh(8.0 * (X @ (u / u.norm()) - b))


def _rows(case, seed):
    """Node-sorted rows on the device: x (flat), y, and the host's offsets."""

    d, kind, n = _nodes(case)
    g = _generator(seed)
    ro = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    xo = np.concatenate([[0], np.cumsum(n * d)]).astype(np.int64)
    x = _rand(g, int(xo[-1])) * 2.0 - 1.0
    y = torch.empty(int(ro[-1]), device="cuda", dtype=torch.float64)
    for dim in sorted(set(d.tolist())):  # one target per dimension
        ks = np.flatnonzero(d == dim)
        rows = torch.from_numpy(np.repeat(ro[ks] - (np.cumsum(n[ks]) - n[ks]), n[ks]) + np.arange(n[ks].sum())).cuda()
        flat = torch.from_numpy(np.repeat(xo[ks] - (np.cumsum(n[ks]) - n[ks]) * dim, n[ks])
                                + np.arange(n[ks].sum()) * dim).cuda()
        state = g.get_state()
        for s in range(0, rows.numel(), 1 << 19):
            g.set_state(state)
            X = x[flat[s:s + (1 << 19), None] + torch.arange(dim, device="cuda")]
            y[rows[s:s + (1 << 19)]] = _surface(X, g)
    y += 0.01 * _randn(g, y.numel())
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return {"x": x, "y": y, "ro": t(ro), "xo": t(xo[:-1]), "d": t(d), "kind": t(kind), "g": g,
            "pmax": max(_features(int(a), int(b)) for a, b in zip(d, kind)), "dmax": int(d.max()), "n": int(ro[-1])}


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    return _PREPARE[case["op"]](case, seed)


def _prepare_fit(case, seed):
    s = _rows(case, seed)
    g = s["g"]
    s["w"] = None
    if case["weighted"]:  # products of sigmoid gates, as a soft fit's weights
        s["w"] = torch.sigmoid(4.0 * _randn(g, s["n"])) * torch.sigmoid(2.0 * _randn(g, s["n"]))
    s["ridge"] = torch.exp(_rand(g, case["nodes"]) * math.log(1e4)) * 1e-6
    return s | {"case": case}


def _prepare_split(case, seed):
    s = _rows(case, seed)
    g = s["g"]
    d, kind, n = _nodes(case)
    K, R = case["nodes"], case["restarts"]
    quad = bool((kind == QUADRATIC).all())
    model = PolynomialRidgeModel(degree=2, ridge=1e-6) if quad else AffineRidgeModel(ridge=1e-6)
    s["splitter"] = SoftObliqueSplitter(model, case["temperature"], max_iters=case["iters"], n_restarts=R,
                                        min_side_points=32, min_side_fraction=0.0)
    s["temperature"] = torch.full((K,), case["temperature"], device="cuda", dtype=torch.float64)
    s["ridge"] = torch.full((K,), 1e-6, device="cuda", dtype=torch.float64)
    s["keys"] = (torch.arange(K, device="cuda") * 2654435761 + int(seed)).to(torch.int64)
    s["theta0"] = None
    if not case["device_start"]:  # unit normals through each node's middle
        th = torch.zeros((K, R, s["dmax"] + 1), device="cuda", dtype=torch.float64)
        w = _randn(g, K, R, s["dmax"])
        ro, xo = np.concatenate([[0], np.cumsum(n)]), np.concatenate([[0], np.cumsum(n * d)])
        for k in range(K):
            dim = int(d[k])
            wk = w[k, :, :dim] / w[k, :, :dim].norm(dim=1, keepdim=True)
            X = s["x"][xo[k]:xo[k + 1]].view(-1, dim)
            th[k, :, :dim] = wk
            th[k, :, dim] = (X[:4096] @ wk.T).median(dim=0).values
        s["theta0"] = th
    return s | {"case": case}


def _prepare_route(case, seed):
    s = _rows(case, seed)
    g = s["g"]
    d, _, _ = _nodes(case)
    K = case["nodes"]
    s["beta"] = 0.1 * _randn(g, K, s["pmax"])
    w = _randn(g, K, s["dmax"])
    w *= torch.arange(s["dmax"], device="cuda")[None, :] < s["d"][:, None]
    w /= w.norm(dim=1, keepdim=True)
    th = torch.zeros((K, s["dmax"] + 1), device="cuda", dtype=torch.float64)
    th[:, :-1] = w
    th[torch.arange(K, device="cuda"), s["d"].long()] = _rand(g, K) * 0.4 - 0.2
    s["theta"] = th
    return s | {"case": case}


def _prepare_sample(case, seed):
    g = _generator(seed)
    rng = np.random.default_rng([case["shape"], 2])
    C, d = case["chains"], case["dim"]
    k = torch.from_numpy(rng.integers(4, 13, C)).cuda()  # 4 to 12 oblique rows a polytope
    ro = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), k.cumsum(0)])
    total = int(ro[-1])
    c = _rand(g, C, d) - 0.5
    A = _randn(g, total, d)
    A /= A.norm(dim=1, keepdim=True)
    owner = torch.repeat_interleave(torch.arange(C, device="cuda"), k)
    b = (A * c[owner]).sum(1) + _rand(g, total) * 0.45 + 0.05
    one = torch.ones((C, d), device="cuda", dtype=torch.float64)
    s = {"case": case, "polys": DevicePolytopes(d, -one, one, ro, A, b, 12), "x0": c,
         "chain": torch.arange(C, device="cuda", dtype=torch.int32), "seeds": None, "directions": None,
         "uniforms": None, "owner": owner}
    if case["injected"]:
        steps = case["burn_in"] + case["rounds"] * case["thinning"]
        s["directions"], s["uniforms"] = _randn(g, C, steps, d), _rand(g, C, steps)
    else:
        s["seeds"] = torch.arange(C, device="cuda") + (int(seed) << 20)
    return s


def _prepare_predict(case, seed):
    rng = np.random.default_rng([case["shape"], int(seed)])
    d, kind, depth = case["dim"], case["kind"], case["depth"]
    p = _features(d, kind)

    def leaf(level, node_id):
        if kind == AFFINE:
            m = AffineRidgeModel()
        else:
            m = PolynomialRidgeModel(degree=2)
        m.coef_ = rng.normal(size=p)
        return LeafNode(m, depth=level, node_id=node_id)

    def grow(level, node_id):  # some branches end early
        if level == depth or (level > depth // 2 and rng.random() < 0.1):
            return leaf(level, node_id)
        w = rng.normal(size=d)
        w /= np.linalg.norm(w)
        return SplitNode(w, float(rng.uniform(-0.2, 0.2)), grow(level + 1, node_id + "/L"),
                         grow(level + 1, node_id + "/R"), depth=level, node_id=node_id)

    return {"case": case, "tree": RegressionTree(grow(0, "root")), "X": rng.uniform(-1.0, 1.0, (case["points"], d))}


_PREPARE = {"fit": _prepare_fit, "split": _prepare_split, "route": _prepare_route, "sample": _prepare_sample,
            "predict": _prepare_predict}


# --------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "fit":
        r = solve_weighted_ridge_batched(s["x"], s["y"], s["w"], s["ro"], s["d"], s["kind"], s["ridge"],
                                         x_offsets=s["xo"], precision=case["precision"],
                                         weight_floor=1e-12 if case["weighted"] else 0.0, max_features=s["pmax"],
                                         max_dim=s["dmax"])
        return {"beta": r.beta, "ridge": r.ridge_effective, "status": r.status}
    if op == "split":
        narrow = s["dmax"] <= 23 and s["pmax"] <= 23
        shape = {} if narrow else {"group_restarts": 0, "trial_steps": 0, "ctas_per_sm": 2, "restart_warps": 0}
        r = split_level(s["splitter"], s["x"], s["y"], s["ro"], s["d"], s["kind"], s["temperature"], s["ridge"],
                        x_offsets=s["xo"], theta0=s["theta0"], hard_refit=case["hard"], anneal_ratio=case["anneal"],
                        node_keys=s["keys"], max_dim=s["dmax"], max_features=s["pmax"], traces=case["restarts"] > 1,
                        **shape)
        if case["restarts"] > 1:
            # restarts that reach the same partition, or its mirror image, tie
            # in the last bit of their hard loss, so which of them is chosen
            # is not determined by the inputs; every restart's objective along
            # its search and the loss that was reached are
            return {"objective": r.trace_loss, "loss": r.loss, "failure": r.failure}
        out = {"theta": r.theta, "n_right": r.n_right, "iterations": r.n_iters, "failure": r.failure}
        if case["hard"]:
            out |= {"beta": r.beta, "loss": r.loss, "child_loss": r.child_loss}
        return out
    if op == "route":
        sse, ssy = segment_residuals(s["x"], s["y"], s["ro"], s["d"], s["kind"], s["beta"], x_offsets=s["xo"])
        perm, n_right = partition_rows(s["x"], s["ro"], s["d"], s["theta"], x_offsets=s["xo"])
        return {"sse": sse, "ssy": ssy, "perm": perm, "n_right": n_right}
    if op == "sample":
        samples, x, status = hit_and_run_device(
            s["polys"], s["chain"], s["x0"], burn_in=case["burn_in"], thinning=case["thinning"],
            n_rounds=case["rounds"], mode="batched", seeds=s["seeds"], directions=s["directions"],
            uniforms=s["uniforms"])
        return {"samples": samples, "x": x, "status": status}
    leaf, pred = s["tree"].predict_device(s["X"])
    return {"leaf": leaf, "pred": pred}


# -------------------------------------------------------------------- work
def work(case):
    op = case["op"]
    if op in ("fit", "split", "route"):
        d, kind, n = _nodes(case)
        p = np.array([_features(int(a), int(b)) for a, b in zip(d, kind)], dtype=np.float64)
        n, d = n.astype(np.float64), d.astype(np.float64)
        read = float((n * (d + 1)).sum() * 8)
        if op == "fit":  # the Gram's lower triangle, the right-hand side, Cholesky and two solves
            return {"bytes": read + (float(n.sum() * 8) if case["weighted"] else 0.0) + float(p.sum() * 8),
                    "flops": float((n * p * (p + 1) + 2 * n * p + p**3 / 3 + 2 * p**2).sum())}
        if op == "route":  # residuals read x, y; the partition reads x again and writes the order
            return {"bytes": read + float((n * d).sum() * 8) + float(n.sum() * 8),
                    "flops": float((n * (2 * p + 2 * d + 4)).sum())}
        # per restart and iteration: scores, both sides' Grams, residuals,
        # gradient and one line-search candidate; the rows are read once
        step = 2 * d + p * (p + 1) + 8 * p + 2 * d + 18
        return {"bytes": read, "flops": float((n * step).sum() * case["restarts"] * case["iters"])}
    if op == "sample":
        C, dim = case["chains"], case["dim"]
        steps = case["burn_in"] + case["rounds"] * case["thinning"]
        draws = C * steps * (dim + 1) * 8 if case["injected"] else 0
        return {"bytes": float(C * case["rounds"] * dim * 8 + C * 8 * (dim + 1) * 8 + draws),
                "flops": float(C * steps * (2 * 8 * dim + 7 * dim + 6 * (2 * dim + 8)))}
    p = _features(case["dim"], case["kind"])
    return {"bytes": float(case["points"] * (case["dim"] * 8 + 12)),
            "flops": float(case["points"] * (2 * case["dim"] * case["depth"] + 3 * p))}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    op = case["op"]
    if op == "fit":
        return _exact_fit(case, seed)
    if op == "split":
        d, kind, n = _nodes(case)
        # the framework's own start normals have no value outside it; long
        # searches take too long one restart at a time
        if case["device_start"] or case["restarts"] > 1:
            return None
        return _exact_split(case, seed)
    if op == "route":
        return _exact_route(case, seed)
    if op == "sample":
        return _exact_sample(case, seed) if case["injected"] else None
    return _exact_predict(case, seed)


def _phi(X, kind):
    one = torch.ones((X.shape[0], 1), device=X.device, dtype=X.dtype)
    if kind == AFFINE:
        return torch.cat([X, one], 1)
    i, j = torch.triu_indices(X.shape[1], X.shape[1], device=X.device)
    return torch.cat([one, X, X[:, i] * X[:, j]], 1)


def _each(case, s):
    d, kind, n = _nodes(case)
    ro, xo = np.concatenate([[0], np.cumsum(n)]), np.concatenate([[0], np.cumsum(n * d)])
    for k in range(case["nodes"]):
        yield k, s["x"][xo[k]:xo[k + 1]].view(-1, int(d[k])), s["y"][ro[k]:ro[k + 1]], int(kind[k]), int(ro[k]), int(ro[k + 1])


def _ridge_solve(phi, y, q, ridge):
    p = phi.shape[1]
    wp = phi if q is None else phi * q[:, None]
    G, h = wp.T @ phi, wp.T @ y
    lam = ridge * torch.trace(G) / p
    G.diagonal().add_(lam)
    return torch.cholesky_solve(h[:, None], torch.linalg.cholesky_ex(G).L)[:, 0], lam


def _exact_fit(case, seed):
    s = _prepare_fit(case, seed)
    beta = torch.full((case["nodes"], s["pmax"]), float("nan"), device="cuda", dtype=torch.float64)
    lam = torch.empty(case["nodes"], device="cuda", dtype=torch.float64)
    for k, X, y, kind, r0, r1 in _each(case, s):
        q = None if s["w"] is None else s["w"][r0:r1].clamp(min=1e-12)
        phi = _phi(X, kind)
        beta[k, : phi.shape[1]], lam[k] = _ridge_solve(phi, y, q, s["ridge"][k])
    return {"beta": beta, "ridge": lam, "status": None}


def _exact_route(case, seed):
    s = _prepare_route(case, seed)
    sse = torch.empty(case["nodes"], device="cuda", dtype=torch.float64)
    ssy = torch.empty_like(sse)
    for k, X, y, kind, _, _ in _each(case, s):
        phi = _phi(X, kind)
        sse[k] = (y - phi @ s["beta"][k, : phi.shape[1]]).square().sum()
        ssy[k] = y.square().sum()
    return {"sse": sse, "ssy": ssy, "perm": None, "n_right": None}


def _exact_split(case, seed):
    """The projected-gradient search of each node, one restart, by plain torch."""

    s = _prepare_split(case, seed)
    sp = s["splitter"]
    K, nan = case["nodes"], float("nan")
    theta = torch.full((K, s["dmax"] + 1), nan, device="cuda", dtype=torch.float64)
    beta = torch.full((K, 2, s["pmax"]), nan, device="cuda", dtype=torch.float64)
    loss, child = torch.full_like(theta[:, 0], nan), torch.full_like(theta[:, :2], nan)
    for k, X, y, kind, _, _ in _each(case, s):
        n, dim = X.shape
        phi = _phi(X, kind)

        def fit(th, T):
            pi = torch.sigmoid(((X @ th[:-1] - th[-1]) / T).clamp(-50.0, 50.0))
            bl = _ridge_solve(phi, y, (1.0 - pi).clamp(min=1e-12), 1e-6)[0]
            br = _ridge_solve(phi, y, pi.clamp(min=1e-12), 1e-6)[0]
            el, er = (y - phi @ bl).square(), (y - phi @ br).square()
            c = (er - el) * pi * (1.0 - pi) / n
            gr = torch.cat([X.T @ c / T, -c.sum()[None] / T])
            pg = gr.clone()
            pg[:-1] -= (gr[:-1] @ th[:-1]) * th[:-1]
            return ((1.0 - pi) * el + pi * er).mean().item(), el, er, pg, (gr @ -pg).item()

        def unit(th):
            return torch.cat([th[:-1] / th[:-1].norm(), th[-1:]])

        T = case["temperature"]
        th = unit(s["theta0"][k, 0, : dim + 1])
        f, el, er, pg, slope = fit(th, T)
        tol = sp.grad_atol + sp.grad_rtol * pg.norm().item()
        alpha = sp.alpha0
        for it in range(case["iters"]):
            if pg.norm().item() <= tol or slope >= 0.0:
                break
            ok, failures, a = False, 0, alpha
            while not ok and failures < sp.max_line_search_failures:
                for back in range(sp.max_backtracks + 1):
                    a = a * sp.rho if back else a
                    tc = unit(th - a * pg)
                    pi = torch.sigmoid(((X @ tc[:-1] - tc[-1]) / T).clamp(-50.0, 50.0))
                    if ((1.0 - pi) * el + pi * er).mean().item() <= f + sp.armijo_c * a * slope:
                        ok = True
                        break
                if ok:
                    grow = sp.alpha_grow if back == 0 else (sp.alpha_recovery if back >= sp.heavy_backtrack_threshold
                                                            else 1.0 / sp.rho)
                    alpha = min(max(a * grow, sp.alpha_min), sp.alpha_max)
                else:
                    alpha = min(max(a * sp.rho, sp.alpha_min), sp.alpha_max)
                    failures += 1
                    if alpha <= sp.alpha_min:
                        break
                    a = alpha
            if not ok:
                break
            th = tc
            if case["anneal"] != 1.0 and case["iters"] > 1:
                T = case["temperature"] * case["anneal"] ** ((it + 1) / (case["iters"] - 1))
            f, el, er, pg, slope = fit(th, T)
        th = unit(th)
        theta[k, : dim + 1] = th
        if case["hard"]:
            right = X @ th[:-1] - th[-1] >= 0.0
            for side, m in enumerate((~right, right)):
                b = _ridge_solve(phi[m], y[m], None, 1e-6)[0]
                beta[k, side, : b.numel()] = b
                child[k, side] = (y[m] - phi[m] @ b).square().mean()
            share = right.double().mean()
            loss[k] = (1.0 - share) * child[k, 0] + share * child[k, 1]
    out = {"theta": theta, "n_right": None, "iterations": None, "failure": None}
    if case["hard"]:
        out |= {"beta": beta, "loss": loss, "child_loss": child}
    return out


def _exact_sample(case, seed):
    """Batched hit-and-run with injected draws: chord from the signs of A u."""

    s = _prepare_sample(case, seed)
    P, C, d = s["polys"], case["chains"], case["dim"]
    rows = int((P.row_offsets[1:] - P.row_offsets[:-1]).max())
    slot = torch.arange(P.A.shape[0], device="cuda") - P.row_offsets[:-1][s["owner"]]
    A = torch.zeros((C, rows + 2 * d, d), device="cuda", dtype=torch.float64)
    b = torch.ones((C, rows + 2 * d), device="cuda", dtype=torch.float64)
    A[s["owner"], slot] = P.A
    b[s["owner"], slot] = P.b
    eye = torch.eye(d, device="cuda", dtype=torch.float64)
    A[:, rows:rows + d], A[:, rows + d:] = eye, -eye
    x = s["x0"].clone()
    slack = b - (A @ x[:, :, None])[..., 0]
    steps = case["burn_in"] + case["rounds"] * case["thinning"]
    kept = torch.empty((case["rounds"], C, d), device="cuda", dtype=torch.float64)
    inf = float("inf")
    for step in range(steps):
        u = s["directions"][:, step]
        au = (A @ u[:, :, None])[..., 0]
        q = slack / au
        hi = torch.where(au > 0, q, inf).amin(1)
        lo = torch.where(au < 0, q, -inf).amax(1)
        t = lo + s["uniforms"][:, step] * (hi - lo)
        x = x + t[:, None] * u
        slack = slack - t[:, None] * au
        r = step - case["burn_in"] + 1
        if r > 0 and r % case["thinning"] == 0:
            kept[r // case["thinning"] - 1] = x
    return {"samples": kept, "x": x, "status": None}


def _exact_predict(case, seed):
    s = _prepare_predict(case, seed)
    X = torch.from_numpy(s["X"]).cuda()
    phi = _phi(X, case["kind"])
    pred = torch.empty(X.shape[0], device="cuda", dtype=torch.float64)

    def walk(node, rows):
        if rows.numel() == 0:
            return
        if isinstance(node, LeafNode):
            pred[rows] = phi[rows] @ torch.from_numpy(node.model.coef_).cuda()
            return
        right = X[rows] @ torch.from_numpy(node.w).cuda() - node.z >= 0.0
        walk(node.left, rows[~right])
        walk(node.right, rows[right])

    walk(s["tree"].root, torch.arange(X.shape[0], device="cuda"))
    return {"leaf": None, "pred": pred.cpu().numpy()}
