"""The work that users of this framework have it do, as timed cases.

listed() names them, draw(rng) gives more of the same ranges, prepare(case, seed)
makes what a program has in hand, run(state) is one pass through the public
entry points, work(case) the least such a pass takes, and exact(case, seed) the
outputs in 64 bits from plain torch.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import culof_gb300
from culof_gb300 import _culof
from culof_gb300.autograd import lof_scores


def listed():
    return [
        # A script's small table through the scikit-learn style class on host
        # arrays: latency of one call, launches and copies.
        _case("host_fit_predict_n500_d8_k20", "host_fit_predict", 500, 8, 20, contamination=0.01),
        # A few thousand rows already on the GPU, odd sizes, z-scored.
        _case("scores_n3001_d5_k15_norm", "scores", 3001, 5, 15, normalize=True),
        # The plain exact workload: clusters with 1% uniform outliers.
        _case("fit_predict_n20000_d8_k20", "fit_predict", 20000, 8, 20, contamination=0.01),
        # The same at scale (the headline benchmark's input).
        _case("fit_predict_n200000_d8_k20", "fit_predict", 200000, 8, 20, contamination=0.01),
        # Three features, a ragged row count, more neighbours, z-scored, 'auto'.
        _case("fit_predict_n50021_d3_k35_norm", "fit_predict", 50021, 3, 35, normalize=True),
        # The feature sweep's middle, through the host function lof(X, k).
        _case("host_scores_n20000_d32_k20", "host_scores", 20000, 32, 20),
        # A wide ragged table with correlated features.
        _case("fit_predict_n30011_d100_k30", "fit_predict", 30011, 100, 30, contamination=0.02, data="factor"),
        # The precision workload: rank-16 factor model, the largest call.
        _case("fit_predict_n200000_d128_k50", "fit_predict", 200000, 128, 50, contamination=0.01, data="factor"),
        # More features than the fused paths take (embedding vectors).
        _case("scores_n8000_d200_k20", "scores", 8000, 200, 20, data="factor"),
        # A training step through the scores: forward and backward.
        _case("gradient_n50000_d32_k20", "gradient", 50000, 32, 20, data="mixture"),
        # The same on a small batch of rows.
        _case("gradient_n4000_d8_k20", "gradient", 4000, 8, 20, data="mixture"),
        # Many independent uneven problems in one call.
        _case("batched_256_d16", "batched", 16384, 16, 40, data="groups", problems=256, layout=1),
    ]


def _case(name, entry, n, d, k, normalize=False, contamination=0.0, data="clusters", problems=0, layout=0):
    return {"name": name, "entry": entry, "n": n, "d": d, "k": k, "normalize": normalize,
            "contamination": contamination, "data": data, "problems": problems, "layout": layout}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["host_fit_predict", "host_scores", "fit_predict", "fit_predict", "scores", "gradient",
                        "batched"])
    normalize = rng.random() < 0.3
    if entry == "batched":
        case = _case("", entry, _log_int(rng, 2000, 16384), rng.choice([3, 8, 11, 16, 24]), rng.randint(12, 40),
                     normalize, data="groups", problems=_log_int(rng, 16, 256), layout=rng.randint(1, 10**6))
    else:
        width = rng.choice(["narrow", "narrow", "narrow", "middle", "wide", "over"])
        if width == "narrow":
            d, top, data = rng.randint(2, 8), 200000, "clusters"
        elif width == "middle":
            d, top, data = rng.randint(9, 42), 100000, rng.choice(["clusters", "mixture"])
        elif width == "wide":
            d, top, data = rng.randint(43, 128), 100000, "factor"
        else:
            d, top, data = rng.randint(129, 256), 12000, "factor"
        if entry == "gradient":
            top = min(top, 50000)
        n = _log_int(rng, 500, top)
        case = _case("", entry, n, d, rng.randint(10, 50), normalize, rng.choice([0.0, 0.01, 0.02, 0.05]), data)
    del case["name"]
    return case


def _sizes(case):
    """Rows and neighbours of a batched case's problems: log-uniform rows, fixed by the case alone."""
    rng = np.random.default_rng(case["layout"])
    ns = np.exp(rng.uniform(np.log(128), np.log(case["n"]), size=case["problems"])).astype(np.int64)
    ks = rng.integers(10, case["k"] + 1, size=case["problems"]).astype(np.int32)
    off = np.zeros(case["problems"] + 1, np.int64)
    off[1:] = np.cumsum(ns)
    return off, ks


def _clusters(g, n, d, count, centre, sigma, frac, box):
    """Gaussian clusters of equal weight with a fraction of uniform outliers in random places."""
    dev = "cuda"
    centres = (torch.rand(count, d, generator=g, device=dev) * 2 - 1) * centre
    sig = sigma[0] + (sigma[1] - sigma[0]) * torch.rand(count, generator=g, device=dev)
    lab = torch.randint(0, count, (n,), generator=g, device=dev)
    X = centres[lab] + sig[lab, None] * torch.randn(n, d, generator=g, device=dev)
    m = int(round(n * frac))
    rows = torch.randperm(n, generator=g, device=dev)[:m]
    X[rows] = (torch.rand(m, d, generator=g, device=dev) * 2 - 1) * box
    return X.contiguous()


def _factor(g, n, d):
    """Rank-16 factor model plus noise, shifted by 5; 0.5% of the rows with uniform noise added."""
    dev = "cuda"
    F = torch.randn(n, 16, generator=g, device=dev)
    L = torch.randn(16, d, generator=g, device=dev) / 4.0
    X = F @ L + 0.1 * torch.randn(n, d, generator=g, device=dev) + 5.0
    m = int(round(n * 0.005))
    rows = torch.randperm(n, generator=g, device=dev)[:m]
    X[rows] += (torch.rand(m, d, generator=g, device=dev) * 2 - 1) * 3.0
    return X.contiguous()


def _points(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n, d = case["n"], case["d"]
    if case["data"] == "factor":
        return _factor(g, n, d)
    if case["data"] == "mixture":
        return _clusters(g, n, d, 8, 8.0, (0.5, 1.5), 0.01, 12.0)
    if case["data"] == "groups":
        # three unit clusters and 2% outliers per problem, its own centres
        off, _ = _sizes(case)
        num, ntot = len(off) - 1, int(off[-1])
        pid = torch.repeat_interleave(torch.arange(num, device="cuda"), torch.from_numpy(np.diff(off)).cuda())
        centres = (torch.rand(num, 3, d, generator=g, device="cuda") * 2 - 1) * 6.0
        lab = torch.randint(0, 3, (ntot,), generator=g, device="cuda")
        X = centres[pid, lab] + torch.randn(ntot, d, generator=g, device="cuda")
        out = torch.rand(ntot, generator=g, device="cuda") < 0.02
        X[out] = (torch.rand(int(out.sum()), d, generator=g, device="cuda") * 2 - 1) * 10.0
        return X.contiguous()
    return _clusters(g, n, d, 5, 10.0, (0.5, 2.0), 0.01, 15.0)


def _weights(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1_000_003)
    return torch.randn(case["n"], generator=g, device="cuda")


def prepare(case, seed):
    X = _points(case, seed)
    state = {"case": case}
    entry = case["entry"]
    if entry in ("host_fit_predict", "host_scores"):
        state["X"] = X.cpu().numpy()
        return state
    state["X"] = X
    if entry == "gradient":
        state["X"] = X.requires_grad_(True)
        state["w"] = _weights(case, seed)
        return state
    # device pointers: a context and output buffers that the program keeps
    state["ctx"] = _culof.Context()
    if entry == "batched":
        state["off"], state["ks"] = _sizes(case)
    n = X.shape[0]
    state["scores"] = torch.empty(n, dtype=torch.float32, device="cuda")
    if entry == "fit_predict":
        state["labels"] = torch.empty(n, dtype=torch.int64, device="cuda")
        state["offset"] = torch.empty((), dtype=torch.float64, device="cuda")
    return state


def run(state):
    case, X = state["case"], state["X"]
    n, d, k, normalize = case["n"], case["d"], case["k"], case["normalize"]
    contamination = case["contamination"] if case["contamination"] > 0 else "auto"
    entry = case["entry"]
    if entry == "host_fit_predict":
        model = culof_gb300.LOF(n_neighbors=k, contamination=contamination, normalize=normalize)
        labels = model.fit_predict(X)
        return {"nof": model.negative_outlier_factor_, "labels": labels, "offset": float(model.offset_)}
    if entry == "host_scores":
        return {"scores": culof_gb300.lof(X, k=k, normalize=normalize)}
    if entry == "gradient":
        X.grad = None
        scores = lof_scores(X, k=k, normalize=normalize)
        (scores * state["w"]).sum().backward()
        return {"scores": scores.detach(), "grad": X.grad}
    ctx, scores = state["ctx"], state["scores"]
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    if entry == "batched":
        ctx.lof_batched_device(state["off"], state["ks"], X.data_ptr(), d, normalize, scores.data_ptr())
        return {"scores": scores}
    if entry == "scores":
        ctx.lof_device(X.data_ptr(), n, d, k, normalize, scores.data_ptr())
        return {"scores": scores}
    labels, offset = state["labels"], state["offset"]
    ctx.fit_predict_device(X.data_ptr(), n, d, k, normalize, contamination, scores.data_ptr(), labels.data_ptr(),
                           offset.data_ptr())
    return {"nof": scores, "labels": labels, "offset": offset}


def work(case):
    """Points in and results out once; one 2 d-flop distance per unordered pair of points."""
    d, k = case["d"], case["k"]
    if case["entry"] == "batched":
        off, _ = _sizes(case)
        ns = np.diff(off).astype(np.float64)
        return {"bytes": float((4 * d + 4) * ns.sum()), "flops": float((d * ns * (ns - 1)).sum())}
    n = case["n"]
    out = {"fit_predict": 12 * n + 8, "host_fit_predict": 12 * n + 8, "gradient": 8 * n + 8 * n * d}.get(
        case["entry"], 4 * n)
    flops = float(d) * n * (n - 1)
    if case["entry"] == "gradient":
        flops += 6.0 * n * k * d
    return {"bytes": float(4 * n * d + out), "flops": flops}


def _neighbours(Z, k):
    """The k nearest rows of every row of Z (64 bits), by blocks of rows."""
    n = Z.shape[0]
    sq = (Z * Z).sum(1)
    idx = torch.empty(n, k, dtype=torch.int64, device=Z.device)
    step = max(1, min(n, (1 << 29) // n))
    for r in range(0, n, step):
        e = min(n, r + step)
        D = torch.addmm(sq[None, :], Z[r:e], Z.T, alpha=-2.0)
        D[torch.arange(e - r, device=Z.device), torch.arange(r, e, device=Z.device)] = math.inf
        idx[r:e] = torch.topk(D, k, dim=1, largest=False, sorted=True).indices
    return idx


def _lof64(X, k, normalize):
    """LOF scores of the rows of X in 64 bits, neighbour sets held fixed."""
    Z = X - X.mean(0)
    if normalize:
        sd = Z.square().mean(0).sqrt()
        Z = Z / torch.where(sd > 1e-12, sd, torch.ones_like(sd))
    idx = _neighbours(Z.detach(), k)
    d2 = torch.cat([(Z[i, None, :] - Z[j]).square().sum(2)
                    for i, j in zip(torch.arange(len(Z), device=Z.device).split(16384), idx.split(16384))])
    kd2 = d2[:, k - 1]
    reach = torch.maximum(kd2[idx], d2).sqrt()
    lrd = 1.0 / (reach.mean(1) + 1e-10)
    return lrd[idx].mean(1) / lrd


def exact(case, seed):
    n, d, k = case["n"], case["d"], case["k"]
    if case["entry"] == "batched":
        off, ks = _sizes(case)
        X = _points(case, seed).double()
        parts = [_lof64(X[off[p]:off[p + 1]], int(ks[p]), case["normalize"]) for p in range(len(ks))]
        return {"scores": torch.cat(parts)}
    if float(n) * n * d > 1.0e12:  # minutes in 64 bits
        return None
    X = _points(case, seed).double()
    if case["entry"] == "gradient":
        X.requires_grad_(True)
        scores = _lof64(X, k, case["normalize"])
        (scores * _weights(case, seed).double()).sum().backward()
        return {"scores": scores.detach(), "grad": X.grad}
    scores = _lof64(X, k, case["normalize"])
    if "fit_predict" not in case["entry"]:
        return {"scores": scores}
    c = case["contamination"]
    offset = float(np.percentile(-scores.cpu().numpy(), 100.0 * c)) if c > 0 else -1.5
    return {"nof": -scores, "labels": None, "offset": offset}
