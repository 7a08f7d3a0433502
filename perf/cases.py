"""Performance cases of the fit core and of prediction, over the range that users run.

A case is a dict of plain values; ``prepare`` makes its inputs on the GPU from a seed (or in
host memory where the entry point takes host arrays), ``run`` makes one pass through the public
entry points, ``work`` states what that pass cannot do without, and ``exact`` gives the computed
floating outputs in 64 bits where that is quick.

Kinds of case:
 * ``fit``: ``Context.fit_core_device`` on resident rows (kNN core distances and the MST);
 * ``pack``: ``Context.fit_core_packed``, the small fits of a request stream, host arrays;
 * ``estimator``: ``HDBSCAN(...).fit(X)`` on a host array, labels and trees included;
 * ``predict``: ``approximate_predict`` of a host batch against a prepared predictor;
 * ``round``: the backend operations of one Borůvka round as a host driver calls them
   (exact neighbours, per-row candidates, per-component reduction).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cuscan_gb300 as cg
from cuscan_gb300 import _lib

STREAM_FEATURES = (16, 32, 64, 128)   # feature counts of the fit-request stream
LEGACY_STREAM = 1                     # cudaStreamLegacy: the stream torch uses by default


def listed():
    return [
        # the smallest benchmark workload: a plain f32 fit of 2,000 blob points in 10 features,
        # where launches, synchronisations and single-CTA steps count
        dict(name="fit_blobs_2k_d10", kind="fit", family="noisy_blobs", n=2000, d=10, clusters=8,
             min_samples=5, precision="fp32"),
        # a server's pack: eight small fits of the request stream (500 to 2,047 rows) in one call
        dict(name="pack_8_small", kind="pack", fits=8, n_lo=500, n_hi=2047, min_samples=5,
             precision="fp16_refined"),
        # an ordinary request of the stream, ragged rows
        dict(name="fit_stream_9k_d32", kind="fit", family="mixture", n=9001, d=32, clusters=16,
             min_samples=5, precision="bf16_refined"),
        # the largest request of the stream
        dict(name="fit_stream_50k_d128", kind="fit", family="mixture", n=50_000, d=128,
             clusters=30, min_samples=5, precision="fp16_refined"),
        # the anisotropic mixture workload, screened and in plain f32
        dict(name="fit_aniso_100k_d64", kind="fit", family="aniso", n=100_000, d=64, clusters=50,
             min_samples=10, precision="bf16_refined"),
        dict(name="fit_aniso_100k_d64_fp32", kind="fit", family="aniso", n=100_000, d=64,
             clusters=50, min_samples=10, precision="fp32"),
        # the headline workload: unit vectors, 500,000 x 128
        dict(name="fit_vmf_500k_d128", kind="fit", family="vmf", n=500_000, d=128, clusters=100,
             min_samples=15, precision="bf16_refined"),
        # embeddings wider than 128 features (the library takes up to 256)
        dict(name="fit_vmf_20k_d200", kind="fit", family="vmf", n=20_000, d=200, clusters=40,
             min_samples=15, precision="bf16_refined"),
        # the estimator as most users call it: only min_cluster_size set, so min_samples is the
        # same 50 and the arithmetic the default f32; host array in, labels and trees out
        dict(name="estimator_20k_d32", kind="estimator", family="mixture", n=20_011, d=32,
             clusters=20, min_cluster_size=50, min_samples=0, precision="fp32"),
        # approximate_predict against a resident predictor of 100,000 rows: a small batch and
        # the largest batch of the mixed request stream
        dict(name="predict_64_of_100k_d64", kind="predict", n=100_000, d=64, clusters=40, m=63,
             min_samples=5),
        dict(name="predict_4096_of_100k_d64", kind="predict", n=100_000, d=64, clusters=40,
             m=4096, min_samples=5),
        # the backend operations of one round, called one by one (the reference's driver loop)
        dict(name="round_ops_10k_d64", kind="round", n=10_007, d=64, clusters=24, min_samples=10),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges; odd sizes are as likely as round ones."""
    kind = rng.choice(["fit", "fit", "fit", "fit", "estimator", "predict", "predict", "pack",
                       "round"])
    if kind == "pack":
        lo = _log_uniform(rng, 300, 900)
        return dict(kind=kind, fits=rng.randint(2, 10), n_lo=lo,
                    n_hi=min(2047, lo * rng.randint(1, 4) + rng.randint(0, 99)),
                    min_samples=rng.choice([3, 5, 10]),
                    precision=rng.choice(["fp32", "fp16_refined", "bf16_refined"]))
    if kind == "estimator":
        return dict(kind=kind, family=rng.choice(["mixture", "noisy_blobs"]),
                    n=_log_uniform(rng, 1000, 30_000), d=_log_uniform(rng, 2, 128),
                    clusters=rng.randint(4, 30), min_cluster_size=rng.choice([5, 15, 25, 50, 100]),
                    min_samples=rng.choice([0, 0, 5, 10]),
                    precision=rng.choice(["fp32", "bf16_refined", "fp16_refined"]))
    if kind == "predict":
        return dict(kind=kind, n=_log_uniform(rng, 2000, 100_000),
                    d=rng.choice(STREAM_FEATURES + (10, 50)), clusters=rng.randint(4, 40),
                    m=_log_uniform(rng, 1, 4096), min_samples=rng.choice([5, 5, 10, 15, 25]))
    if kind == "round":
        return dict(kind=kind, n=_log_uniform(rng, 1000, 20_000), d=_log_uniform(rng, 4, 128),
                    clusters=rng.randint(4, 60), min_samples=rng.choice([5, 10, 15, 30]))
    family = rng.choice(["mixture", "aniso", "vmf", "noisy_blobs"])
    precision = rng.choice(["bf16_refined", "bf16_refined", "fp16_refined", "fp32"])
    wide = rng.random() < 0.15
    d = rng.randint(129, 256) if wide else rng.choice(STREAM_FEATURES + (rng.randint(2, 128),))
    min_samples = rng.choice([1, 3, 5, 5, 10, 10, 15, 15, 25, 32, 50, 100])
    # plain f32, wide rows and long neighbour lists are used on smaller sets
    top = 50_000 if precision == "fp32" else 300_000
    if wide or min_samples > 32:
        top = 25_000
    return dict(kind=kind, family=family, n=_log_uniform(rng, 500, top), d=d,
                clusters=rng.randint(2, 60), min_samples=min_samples, precision=precision)


# ---- inputs ----

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 2654435761 % (1 << 62))


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float32)


def _with_noise(g, pts, n_noise):
    lo, hi = pts.amin(0), pts.amax(0)
    return torch.cat([pts, lo + (hi - lo) * _uniform(g, n_noise, pts.shape[1])])


def _points(family, n, d, clusters, seed):
    """Device rows of one of the benchmark's point-set families (cuscan_gb300.synthetic states
    them on the host): noisy isotropic blobs, isotropic mixtures, anisotropic mixtures with
    noise, and clustered unit vectors with noise."""
    g = _generator(seed)
    centres = 20.0 * _uniform(g, clusters, d) - 10.0
    if family == "noisy_blobs":
        m = n - n // 20
        at = torch.randint(clusters, (m,), generator=g, device="cuda")
        x = _with_noise(g, centres[at] + _normal(g, m, d), n - m)
    elif family == "mixture":
        std = 0.5 + 1.5 * _uniform(g, clusters)
        at = torch.randint(clusters, (n,), generator=g, device="cuda")
        x = centres[at] + _normal(g, n, d) * std[at, None]
    elif family == "aniso":
        m = n - n // 50
        w = -torch.log(_uniform(g, clusters) + 1e-9)          # Dirichlet(1) weights
        at = torch.multinomial(w, m, replacement=True, generator=g).sort().values
        parts = []
        for c, count in enumerate(torch.bincount(at, minlength=clusters).tolist()):
            q, _ = torch.linalg.qr(_normal(g, d, d))
            lam = torch.exp(math.log(0.1) + math.log(20.0) * _uniform(g, d))
            parts.append(centres[c] + (_normal(g, count, d) * lam.sqrt()) @ q.T)
        x = _with_noise(g, torch.cat(parts), n - m)
    else:
        m = n - n // 100
        mu = torch.nn.functional.normalize(_normal(g, clusters, d))
        kappa = 20.0 + 180.0 * _uniform(g, clusters)
        at = torch.randint(clusters, (m,), generator=g, device="cuda")
        x = torch.cat([mu[at] + _normal(g, m, d) / kappa[at, None].sqrt(), _normal(g, n - m, d)])
        x = torch.nn.functional.normalize(x)
    return x[torch.randperm(n, generator=g, device="cuda")].contiguous()


def _pack_shapes(case):
    """(n, d) of a pack's fits: rows log-spaced from n_lo to n_hi, features cycling."""
    f = case["fits"]
    ratio = case["n_hi"] / case["n_lo"]
    return [(int(case["n_lo"] * ratio ** (i / (f - 1))), STREAM_FEATURES[i % 4]) for i in range(f)]


def _pack_points(case, seed):
    return [_points("mixture", n, d, 2 + 3 * i, seed * 64 + i)
            for i, (n, d) in enumerate(_pack_shapes(case))]


def _round_inputs(case, seed):
    n = case["n"]
    x = _points("mixture", n, case["d"], case["clusters"], seed)
    g = _generator(seed + 1)
    core = 0.5 * case["d"] * _uniform(g, n)
    # components of a middle round: many more than clusters, of uneven sizes
    count = max(2, n // 20)
    comp = (count * _uniform(g, n) ** 2).to(torch.int64).clamp_(max=count - 1)
    _, comp = torch.unique(comp, return_inverse=True)
    return x, core, comp.to(torch.int32)


def _plan(components, width=512):
    """The component reduction plan (stable CSR members, tiles of at most `width` members)."""
    comp = components.cpu().numpy()
    members = np.argsort(comp, kind="stable").astype(np.int32)
    sizes = np.bincount(comp)
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    tiles = -(-sizes // width)
    first = np.concatenate([[0], np.cumsum(tiles)])
    owner = np.repeat(np.arange(sizes.size), tiles)
    starts = offsets[owner] + (np.arange(owner.size) - first[owner]) * width
    ends = np.minimum(starts + width, offsets[owner + 1])
    return [torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda()
            for a in (members, starts, ends, first)]


def prepare(case, seed):
    kind = case["kind"]
    ctx = cg.context(0)
    if kind == "pack":
        prec = _lib.PRECISIONS[case["precision"]]
        fits = [(x.cpu().numpy(), case["min_samples"], prec) for x in _pack_points(case, seed)]
        return dict(kind=kind, ctx=ctx, fits=fits)
    if kind == "predict":
        # one draw of the mixture: the first n rows are the training set, the rest the batch
        x = _points("mixture", case["n"] + case["m"], case["d"], case["clusters"], seed)
        x = x.cpu().numpy()
        model = cg.HDBSCAN(min_cluster_size=max(5, case["n"] // 200),
                           min_samples=case["min_samples"], precision="fp16_refined")
        model.fit(x[:case["n"]])
        return dict(kind=kind, predictor=model.to_predictor(),
                    batch=np.ascontiguousarray(x[case["n"]:]))
    if kind == "estimator":
        x = _points(case["family"], case["n"], case["d"], case["clusters"], seed)
        model = cg.HDBSCAN(min_cluster_size=case["min_cluster_size"],
                           min_samples=case["min_samples"] or None, precision=case["precision"])
        return dict(kind=kind, x=x.cpu().numpy(), model=model)
    n, d = case["n"], case["d"]
    k = min(case["min_samples"], n - 1)
    i32 = dict(dtype=torch.int32, device="cuda")
    f32 = dict(dtype=torch.float32, device="cuda")
    if kind == "round":
        x, core, comp = _round_inputs(case, seed)
        members, starts, ends, partial = _plan(comp)
        c = partial.numel() - 1
        state = dict(kind=kind, ctx=ctx, n=n, d=d, k=k, x=x, core=core, comp=comp,
                     plan=(members, starts, ends, partial), p=starts.numel(), c=c,
                     ids=torch.empty((n, k), **i32), dist=torch.empty((n, k), **f32),
                     w=torch.empty(n, **f32), dst=torch.empty(n, **i32),
                     win_w=torch.empty(c, **f32), win_meta=torch.empty((c, 5), **i32))
    else:
        x = _points(case["family"], n, d, case["clusters"], seed)
        state = dict(kind=kind, ctx=ctx, n=n, d=d, x=x, min_samples=case["min_samples"],
                     precision=_lib.PRECISIONS[case["precision"]],
                     ids=torch.empty((n, k), **i32), dist=torch.empty((n, k), **f32),
                     core=torch.empty(n, **f32), src=torch.empty(n - 1, **i32),
                     dst=torch.empty(n - 1, **i32), w=torch.empty(n - 1, **f32))
    torch.cuda.synchronize()  # the fit runs on the context's own stream
    return state


def run(state):
    kind = state["kind"]
    s = state
    if kind == "fit":
        s["ctx"].fit_core_device(s["x"].data_ptr(), s["n"], s["d"], s["min_samples"],
                                 s["precision"], s["ids"].data_ptr(), s["dist"].data_ptr(),
                                 s["core"].data_ptr(), s["src"].data_ptr(), s["dst"].data_ptr(),
                                 s["w"].data_ptr())
        return {key: s[key] for key in ("ids", "dist", "core", "src", "dst", "w")}
    if kind == "pack":
        return [{key: o[key] for key in ("knn_ids", "knn_sq", "core_sq", "src", "dst", "wsq")}
                for o in s["ctx"].fit_core_packed(s["fits"])]
    if kind == "estimator":
        m = s["model"].fit(s["x"])
        mst, tree = m.minimum_spanning_tree_, m.condensed_tree_
        return {"labels": m.labels_, "probabilities": m.probabilities_,
                "core": m.core_distances_, "mst": mst,
                "tree": {key: tree[key] for key in tree.dtype.names},
                "linkage": m.single_linkage_tree_, "neighbors": m.neighbors_}
    if kind == "predict":
        labels, strengths, points = s["predictor"].approximate_predict(s["batch"], True)
        return {"labels": labels, "strengths": strengths, "points": points}
    ctx, x, n = s["ctx"], s["x"].data_ptr(), s["n"]
    ctx.exact_knn(x, n, x, n, s["d"], s["k"], True, 0, True, s["ids"].data_ptr(),
                  s["dist"].data_ptr(), LEGACY_STREAM)
    ctx.boruvka_candidates(x, s["core"].data_ptr(), s["comp"].data_ptr(), n, s["d"],
                           s["w"].data_ptr(), s["dst"].data_ptr(), LEGACY_STREAM)
    ctx.component_reduce(s["w"].data_ptr(), s["dst"].data_ptr(),
                         *[t.data_ptr() for t in s["plan"]], n, s["p"], s["c"],
                         s["win_w"].data_ptr(), s["win_meta"].data_ptr(), LEGACY_STREAM)
    return {key: s[key] for key in ("ids", "dist", "w", "dst", "win_w", "win_meta")}


# ---- what a pass cannot do without ----

def _fit_work(n, d, k):
    # rows in; kNN ids and distances, cores and MST edges out; every unordered pair of rows
    # compared once (a multiply and an add per feature)
    return 4 * n * d + 8 * n * k + 4 * n + 12 * (n - 1), float(n) * n * d


def work(case):
    kind = case["kind"]
    if kind == "pack":
        parts = [_fit_work(n, d, min(case["min_samples"], n - 1)) for n, d in _pack_shapes(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    n, d = case["n"], case["d"]
    if kind == "predict":
        m = case["m"]
        # batch and training rows in; label, strength and connecting point out
        return {"bytes": 4 * d * (n + m) + 24 * m, "flops": 2.0 * m * n * d}
    k = min(case["min_samples"] or case.get("min_cluster_size", 0), n - 1)
    b, f = _fit_work(n, d, k)
    if kind == "round":
        # exact neighbours and candidates share the pairs; core, components and the plan in,
        # candidates and winners out
        b = 4 * n * d + 8 * n * k + 12 * n + 8 * n + 24 * max(2, n // 20)
    if kind == "estimator":
        b += 4 * n * k + 40 * n + 56 * n + 28 * n  # 64-bit neighbours, tree, linkage, labels
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits ----

def _neighbours64(x, k, core=None, comp=None):
    """Sorted squared distances of every row's k nearest other rows, and with cores and
    components the smallest mutual-reachability weight to another component, in 64 bits."""
    x = x.double()
    n, norm = x.shape[0], x.square().sum(1)
    rows = max(1, min(n, (1 << 27) // n))
    near = torch.empty((n, k), dtype=torch.float64, device="cuda")
    low = torch.empty(n, dtype=torch.float64, device="cuda")
    for a in range(0, n, rows):
        b = min(n, a + rows)
        at = torch.arange(a, b, device="cuda")
        sq = (norm[a:b, None] + norm[None, :] - 2.0 * (x[a:b] @ x.T)).clamp_(min=0.0)
        if core is not None:
            w = torch.maximum(sq, torch.maximum(core[a:b, None], core[None, :]).double())
            w.masked_fill_(comp[a:b, None] == comp[None, :], math.inf)
            low[a:b] = w.amin(1)
        sq[at - a, at] = math.inf
        near[a:b] = sq.topk(k, dim=1, largest=False, sorted=True).values
    return near, low


def _core64(near, n, min_samples):
    if min_samples >= n:
        return torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
    if min_samples == 1:
        return torch.zeros(n, dtype=torch.float64, device="cuda")
    return near[:, min_samples - 1].clone()


def exact(case, seed):
    """Distances, core distances and component weights; edge lists, labels and strengths follow
    from them through comparisons and have no value of their own in 64 bits."""
    kind = case["kind"]
    if kind == "predict":
        return None
    if kind == "pack":
        out = []
        for x in _pack_points(case, seed):
            n = x.shape[0]
            k = min(case["min_samples"], n - 1)
            near, _ = _neighbours64(x, k)
            out.append({"knn_ids": None, "knn_sq": near,
                        "core_sq": _core64(near, n, case["min_samples"]), "src": None,
                        "dst": None, "wsq": None})
        return out
    n = case["n"]
    if float(n) * n * case["d"] > 2e12:
        return None
    if kind == "round":
        x, core, comp = _round_inputs(case, seed)
        near, low = _neighbours64(x, min(case["min_samples"], n - 1), core, comp)
        win = torch.full((int(comp.max()) + 1,), math.inf, dtype=torch.float64, device="cuda")
        win.scatter_reduce_(0, comp.long(), low, "amin")
        return {"ids": None, "dist": near, "w": low, "dst": None, "win_w": win, "win_meta": None}
    x = _points(case["family"], n, case["d"], case["clusters"], seed)
    if kind == "estimator":
        ms = case["min_samples"] or case["min_cluster_size"]
        near, _ = _neighbours64(x, min(ms, n - 1))
        return {"labels": None, "probabilities": None, "core": _core64(near, n, ms).sqrt(),
                "mst": None, "tree": None, "linkage": None, "neighbors": None}
    near, _ = _neighbours64(x, min(case["min_samples"], n - 1))
    return {"ids": None, "dist": near, "core": _core64(near, n, case["min_samples"]),
            "src": None, "dst": None, "w": None}
