"""The work that users have this framework do, as cases that can be timed.

A case is a dict of plain values; `prepare` makes what a program has in hand
(inputs from a seed, and the jobs it keeps), `run` takes it once through the
public entry points, `exact` gives the same results in 64 bits from plain
torch, and `work` the bytes and operations one pass cannot do without.

What is run:

  iterate   a stretch of gradient iterations of one device-resident job: the
            coordinates set, `iters` iterations, the coordinates read back.
            This is how a program advances an embedding and shows or stores
            it every so often.  The stretches are short: the gains' sign rule
            turns rounding into a difference of whole steps in longer ones.
  batch     the same for many independent jobs advanced together.
  embed     the library call: host kNN graph in, lambda rescaling,
            symmetrisation, iterations, host embedding out.
  graph     P built from points on the device: exact kNN, lambda rescaling
            or perplexity equalisation, (P + P^T)/(2n).
  affinity  P built from given kNN distances: perplexity equalisation and
            symmetrisation.

Graphs are kNN graphs of Gaussian mixtures in 20 to 100 dimensions (the
mixtures of the benchmark's configurations: centres far enough apart that all
neighbours lie in the point's own component).  Components above 65,536 points
are searched in pieces of that size, so those neighbours are approximate, as
the reference's FLANN search returns them.  Coordinates are the mixture's
components laid out as blobs, a random projection of each component inside
its blob, scaled to a given extent.  The extents are those that runs of these
sizes pass through: 1000 iterations of a 2,000-point job end 73 wide, of
100,000 points 48, of 1.3 million 15.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..",
                                "gpu-sg-sne_b200", "python"))
import sgtsne_b200 as S  # noqa: E402

DEV = "cuda"
SEARCH_MAX = 65536  # points searched together within a component
H = {1: 0.5, 2: 0.7, 3: 1.2}
FORMATS = {"csr": S.FORMAT_CSR, "coo": S.FORMAT_COO, "hybrid": S.FORMAT_HYBRID}


def listed():
    return [
        # the smallest requests of the serving range, near the end of a run
        {"name": "iterate-2k-2d", "what": "iterate", "n": 2000, "d": 2, "k": 30, "dim": 50,
         "comps": 10, "format": "csr", "extent": 40.0, "alpha": 1.0, "iters": 8},
        # the 10,000-point configuration (10-component mixture, k = 30) in mid-run
        {"name": "iterate-10k-2d", "what": "iterate", "n": 10000, "d": 2, "k": 30, "dim": 50,
         "comps": 10, "format": "csr", "extent": 24.0, "alpha": 1.0, "iters": 8},
        # a one-dimensional embedding (-d 1)
        {"name": "iterate-20k-1d", "what": "iterate", "n": 20011, "d": 1, "k": 30, "dim": 50,
         "comps": 10, "format": "csr", "extent": 33.0, "alpha": 1.0, "iters": 8},
        # the 60,000-point configuration (k = 90) shortly after the exaggeration
        {"name": "iterate-60k-2d-k90", "what": "iterate", "n": 60000, "d": 2, "k": 90, "dim": 50,
         "comps": 10, "format": "csr", "extent": 18.0, "alpha": 1.0, "iters": 20},
        # the library's default storage format, a point count that is no round number
        {"name": "iterate-100k-2d-coo", "what": "iterate", "n": 99991, "d": 2, "k": 30, "dim": 50,
         "comps": 40, "format": "coo", "extent": 31.0, "alpha": 1.0, "iters": 20},
        # a three-dimensional embedding of the batched and served ranges
        {"name": "iterate-100k-3d", "what": "iterate", "n": 100000, "d": 3, "k": 30, "dim": 50,
         "comps": 20, "format": "csr", "extent": 18.5, "alpha": 1.0, "iters": 20},
        # a spread-out embedding on the largest grid (512 points per axis)
        {"name": "iterate-400k-2d-wide", "what": "iterate", "n": 400000, "d": 2, "k": 30,
         "dim": 50, "comps": 40, "format": "csr", "extent": 352.0, "alpha": 1.0, "iters": 20},
        # the benchmark's 1.3M-point configuration; its runs stay on small grids
        {"name": "iterate-1300k-2d", "what": "iterate", "n": 1300000, "d": 2, "k": 30, "dim": 50,
         "comps": 40, "format": "csr", "extent": 2.0, "alpha": 1.0, "iters": 20},
        # independent embeddings of uneven size together, half 2-D and half 3-D
        {"name": "batch-24", "what": "batch", "jobs": 24, "n_lo": 2000, "n_hi": 40000, "k": 30,
         "dim": 40, "comps": 10, "extent": 22.0, "alpha": 1.0, "iters": 8},
        # the drop-in library call from host memory
        {"name": "embed-20k-2d", "what": "embed", "n": 20000, "d": 2, "k": 30, "dim": 50,
         "comps": 10, "extent": 16.0, "alpha": 1.0, "iters": 16, "lambda": 10.0},
        # P of a mid-sized data set from its points
        {"name": "graph-100k", "what": "graph", "n": 100000, "k": 30, "dim": 50, "comps": 40,
         "lambda": 10.0},
        # P of the 60,000-image configuration (784 pixels of 0..255, k = 90, perplexity 30)
        {"name": "graph-60k-images", "what": "graph", "n": 60000, "k": 90, "dim": 784,
         "comps": 10, "perplexity": 30.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    what = rng.choice(["iterate"] * 6 + ["batch", "embed", "graph", "affinity"])
    dim, comps = rng.randint(20, 100), rng.randint(5, 40)
    if what == "iterate":
        d = rng.choice([1, 2, 2, 2, 3, 3])
        n = int(_log(rng, 1000, 500000 if d == 3 else 1200000))
        k = 30 if n > 150000 else rng.choice([15, 30, 30, 90])
        # later states are wider, and fewer points spread further
        widest = 75.0 if n < 10000 else (55.0 if n < 300000 else 25.0)
        widest = widest * (0.7 if d == 3 else 1.0)
        return {"what": what, "n": n, "d": d, "k": k, "dim": dim, "comps": comps,
                "format": rng.choice(["csr", "csr", "csr", "coo", "hybrid"]),
                "extent": round(_log(rng, 1.0, widest), 2),
                "alpha": rng.choice([1.0, 1.0, 12.0]) if n > 20000 else 1.0,
                "iters": rng.choice([8, 8, 16, 20]) if n > 50000 else rng.choice([4, 8])}
    if what == "batch":
        return {"what": what, "jobs": rng.randint(4, 48), "n_lo": 1000,
                "n_hi": int(_log(rng, 5000, 60000)), "k": 30, "dim": dim, "comps": comps,
                "extent": round(_log(rng, 4.0, 40.0), 2), "alpha": 1.0, "iters": 8}
    if what == "embed":
        return {"what": what, "n": int(_log(rng, 2000, 100000)), "d": rng.choice([2, 2, 3]),
                "k": rng.choice([15, 30]), "dim": dim, "comps": comps,
                "extent": round(_log(rng, 8.0, 40.0), 2), "alpha": 1.0, "iters": 12,
                "lambda": rng.choice([1.0, 10.0])}
    if what == "graph":
        n = int(_log(rng, 2000, 130000))
        if rng.random() < 0.3:
            k = rng.randint(30, 96)
            return {"what": what, "n": n // 3, "k": k, "dim": rng.randint(65, 784),
                    "comps": rng.randint(5, 10), "perplexity": float(k // 3)}
        return {"what": what, "n": n, "k": rng.choice([10, 30, 30]), "dim": dim, "comps": comps,
                "lambda": rng.choice([1.0, 5.0])}
    k = rng.randint(30, 96)
    return {"what": what, "n": int(_log(rng, 2000, 120000)), "k": k, "dim": dim, "comps": comps,
            "perplexity": float(k // 3)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _points(n, dim, comps, gen):
    """n points of a mixture with Zipf(1.1) sizes in random order, by component."""
    w = torch.arange(1, comps + 1, dtype=torch.float64) ** -1.1
    size = (w / w.sum() * n).floor().to(torch.int64).clamp_min(1)
    size[0] += n - int(size.sum())
    centre = torch.randn(comps, dim, generator=gen, device=DEV) * 5.0
    lab = torch.repeat_interleave(torch.arange(comps, device=DEV), size.to(DEV))
    off = torch.randn(n, dim, generator=gen, device=DEV)
    return centre[lab] + off, off, lab, size.tolist()


def _images(n, dim, comps, gen):
    """n vectors of whole numbers 0..255: noisy copies of templates with about
    a fifth of their coordinates active, in random order."""
    active = torch.rand(comps, dim, generator=gen, device=DEV) < 0.19
    template = active * torch.rand(comps, dim, generator=gen, device=DEV) * 255.0
    lab = torch.randint(comps, (n,), generator=gen, device=DEV)
    x = template[lab] * (torch.rand(n, dim, generator=gen, device=DEV) < 0.9)
    x += 20.0 * torch.randn(n, dim, generator=gen, device=DEV)
    return x.clamp_(0.0, 255.0).floor_().contiguous()


def _knn(x, size, k, gen):
    """(idx, d2): k nearest neighbours in the own component, rows by distance."""
    n = x.shape[0]
    idx = torch.empty(n, k, dtype=torch.int64, device=DEV)
    d2 = torch.empty(n, k, device=DEV)
    at = 0
    for m in size:
        pieces = max(1, -(-m // SEARCH_MAX))
        order = at + (torch.randperm(m, generator=gen, device=DEV) if pieces > 1 else
                      torch.arange(m, device=DEV))
        parts = torch.chunk(order, pieces)
        for p, rows in enumerate(parts):
            cand = parts[(p + 1) % pieces]
            # a component with fewer than k + 1 points takes its neighbours from all points
            if len(cand) <= k:
                cand = torch.arange(n, device=DEV)
            xc = x[cand]
            sq = (xc * xc).sum(1)
            for b in torch.split(rows, 4096):
                q = x[b]
                dist = (q * q).sum(1)[:, None] + sq[None] - 2.0 * (q @ xc.T)
                dist.masked_fill_(b[:, None] == cand[None], float("inf"))
                v, j = torch.topk(dist, k, dim=1, largest=False)
                idx[b], d2[b] = cand[j], v.clamp_min(0.0)
        at += m
    return idx, d2


def _symmetric(n, idx, w):
    """(P + P^T)/(2n) as CSR, from row-normalised weights of the neighbour lists."""
    k = idx.shape[1]
    row = torch.arange(n, device=DEV).repeat_interleave(k)
    col = idx.reshape(-1)
    key, order = torch.sort(torch.cat([row * n + col, col * n + row]), stable=True)
    val = torch.cat([w.reshape(-1), w.reshape(-1)])[order]
    key, inv = torch.unique_consecutive(key, return_inverse=True)
    out = torch.zeros(key.numel(), dtype=w.dtype, device=DEV).index_add_(0, inv, val) / (2.0 * n)
    rowptr = torch.searchsorted(key, torch.arange(n + 1, device=DEV) * n).to(torch.int32)
    return rowptr, (key % n).to(torch.int32), out


def _layout(off, lab, size, d, extent, gen):
    """Coordinates: a blob per component, `extent` wide over all."""
    comps, n = len(size), off.shape[0]
    y = off @ (torch.randn(off.shape[1], d, generator=gen, device=DEV) / math.sqrt(off.shape[1]))
    radius = (torch.tensor(size, dtype=torch.float32, device=DEV) / n) ** (1.0 / d)
    centre = torch.rand(comps, d, generator=gen, device=DEV) * 2.0 - 1.0
    y = centre[lab] + y * (0.25 * radius)[lab][:, None]
    y -= y.mean(0)
    return (y * (extent / (y.max(0)[0] - y.min(0)[0]).max())).contiguous()


def _inputs(case, seed, n=None, d=None):
    """Points, neighbours, P and coordinates of one embedding, in random point order."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    tf32 = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    try:
        n = n or case["n"]
        if case["what"] == "graph" and "perplexity" in case:
            return {"n": n, "x": _images(n, case["dim"], case["comps"], gen)}
        x, off, lab, size = _points(n, case["dim"], case["comps"], gen)
        out = {"n": n, "x": x}
        perm = torch.randperm(n, generator=gen, device=DEV)  # new place -> place by component
        if case["what"] == "graph":
            out["x"] = x[perm].contiguous()
            return out
        idx, d2 = _knn(x, size, case["k"], gen)
        place = torch.empty_like(perm)
        place[perm] = torch.arange(n, device=DEV)
        out["x"], out["idx"], out["d2"] = None, place[idx[perm]], d2[perm].contiguous()
        if case["what"] != "affinity":
            d = d or case["d"]
            out["y"] = _layout(off, lab, size, d, case["extent"], gen)[perm].contiguous()
        if case["what"] in ("iterate", "batch"):
            near = out["d2"] - out["d2"][:, :1]
            w = torch.exp(-near / near.mean(1, keepdim=True).clamp_min(1e-20))
            out["p"] = _symmetric(n, out["idx"], w / w.sum(1, keepdim=True))
            out["idx"] = out["d2"] = None
        return out
    finally:
        torch.backends.cuda.matmul.allow_tf32 = tf32


def _batch_sizes(case):
    """Sizes of a batch's jobs: even steps over the logarithm of the range, 2-D and 3-D in turn."""
    lo, hi, m = math.log(case["n_lo"]), math.log(case["n_hi"]), case["jobs"]
    return [(int(math.exp(lo + (hi - lo) * i / max(1, m - 1))), 2 + i % 2) for i in range(m)]


# ---------------------------------------------------------------------------
# what a program holds, and one pass
# ---------------------------------------------------------------------------
_CTX = []


def _ctx():
    if not _CTX:
        _CTX.append(S.Context(0))
    return _CTX[0]


def _params(case, d, fmt):
    p = S.default_params(d=d, format=FORMATS[fmt], alpha=case["alpha"], max_iter=case["iters"],
                         h=H[d])
    p.lambda_ = case.get("lambda", 1.0)
    return p


def _job(ctx, case, inp, d, fmt):
    rowptr, col, val = inp["p"]
    torch.cuda.synchronize()
    job = S.Job(ctx, _params(case, d, fmt), rowptr, col, val.float(), device_mem=True)
    job.prepare()
    return job


def prepare(case, seed):
    ctx, what = _ctx(), case["what"]
    s = {"ctx": ctx, "case": case}
    if what == "iterate":
        inp = _inputs(case, seed)
        s["job"], s["y"] = _job(ctx, case, inp, case["d"], case["format"]), inp["y"]
        s["out"] = torch.empty_like(inp["y"])
    elif what == "batch":
        s["jobs"], s["ys"] = [], []
        for i, (n, d) in enumerate(_batch_sizes(case)):
            inp = _inputs(case, seed * 1000 + i, n, d)
            s["jobs"].append(_job(ctx, case, inp, d, "csr"))
            s["ys"].append(inp["y"])
        s["outs"] = [torch.empty_like(y) for y in s["ys"]]
        s["batch"] = S.Batch(ctx, s["jobs"])
    elif what == "embed":
        inp = _inputs(case, seed)
        n, k = case["n"], case["k"]
        s["rowptr"] = np.arange(0, (n + 1) * k, k, dtype=np.int32)
        s["col"] = inp["idx"].reshape(-1).to(torch.int32).cpu().numpy()
        s["val"] = inp["d2"].reshape(-1).cpu().numpy()
        if case["lambda"] == 1.0:  # rescaling is skipped: the values are probabilities
            s["val"] = (np.exp(-s["val"] / s["val"].reshape(n, k).mean(1).repeat(k)) / k).astype(
                np.float32)
        s["y"] = np.ascontiguousarray(inp["y"].T.cpu().numpy())
        s["params"] = _params(case, case["d"], "csr")
    elif what == "graph":
        n, k = case["n"], case["k"]
        s["x"] = _inputs(case, seed)["x"]
        s["idx"] = torch.empty(n, k, dtype=torch.int32, device=DEV)
        s["d2"] = torch.empty(n, k, device=DEV)
        s["p"] = torch.empty(n, k, device=DEV)
        s["beta"] = torch.zeros(n, device=DEV)
        s["rowptr"] = torch.arange(0, (n + 1) * k, k, dtype=torch.int32, device=DEV)
        _symmetric_buffers(s, n, k)
    else:
        n, k = case["n"], case["k"]
        inp = _inputs(case, seed)
        s["d2"], s["idx"] = inp["d2"], inp["idx"].to(torch.int32).contiguous()
        s["p"] = torch.empty(n, k, device=DEV)
        s["beta"] = torch.empty(n, device=DEV)
        s["rowptr"] = torch.arange(0, (n + 1) * k, k, dtype=torch.int32, device=DEV)
        _symmetric_buffers(s, n, k)
    torch.cuda.synchronize()
    return s


def _symmetric_buffers(s, n, k):
    s["srp"] = torch.empty(n + 1, dtype=torch.int32, device=DEV)
    # the upper bound of P's size; the entries behind P stay zero
    s["sc"] = torch.zeros(2 * n * k, dtype=torch.int32, device=DEV)
    s["sv"] = torch.zeros(2 * n * k, device=DEV)


def run(s):
    case, ctx = s["case"], s["ctx"]
    what = case["what"]
    if what == "iterate":
        s["job"].set_y(s["y"], S.LAYOUT_POINT_MAJOR, True)
        s["job"].run(case["iters"])
        return s["job"].get_y(s["out"], S.LAYOUT_POINT_MAJOR, True)
    if what == "batch":
        for job, y in zip(s["jobs"], s["ys"]):
            job.set_y(y, S.LAYOUT_POINT_MAJOR, True)
        s["batch"].run(case["iters"])
        return [job.get_y(o, S.LAYOUT_POINT_MAJOR, True) for job, o in zip(s["jobs"], s["outs"])]
    if what == "embed":
        return ctx.embed(s["rowptr"], s["col"], s["val"], s["params"], y_in=s["y"])[0]
    n, k = case["n"], case["k"]
    if what == "graph":
        ctx.knn(n, case["dim"], s["x"], k, s["idx"], s["d2"])
    if "perplexity" in case:
        ctx.perplexity(n, k, s["d2"], case["perplexity"], s["p"], s["beta"])
    else:
        s["p"].copy_(s["d2"])  # the rescaling works in place
        torch.cuda.current_stream().synchronize()
        ctx.lambda_bisect(n, s["rowptr"], s["p"], case["lambda"], 1, s["beta"])
    s["nnz"] = ctx.symmetrize(n, n * k, s["rowptr"], s["idx"], s["p"], 1.0 / (2 * n), s["srp"],
                              s["sc"], s["sv"])
    return {key: s[key] for key in ("idx", "d2", "p", "beta", "srp", "sc", "sv", "nnz")}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
SYM = 1.65  # nonzeros of P + P^T per neighbour-list entry of these graphs


def _iteration_work(n, k, d):
    """P, coordinates, momentum and gains read, the last three written."""
    nnz = SYM * n * k
    return (8.0 * nnz + 4.0 * n + 6 * 4.0 * n * d,
            nnz * (4.0 * d + 2) + 2 * n * 4.0 ** d * (d + 1) * 2)


def work(case):
    what = case["what"]
    if what in ("iterate", "embed", "batch"):
        jobs = _batch_sizes(case) if what == "batch" else [(case["n"], case["d"])]
        per = [_iteration_work(n, case["k"], d) for n, d in jobs]
        b, f = (case["iters"] * sum(v) for v in zip(*per))
        if what == "embed":  # the graph in; the embedding out
            b += 8.0 * case["n"] * case["k"] + 8.0 * case["n"] * case["d"]
        return {"bytes": b, "flops": f}
    n, k = case["n"], case["k"]
    if what == "graph":  # points in; lists, rescaled lists and P out
        return {"bytes": 4.0 * n * case["dim"] + 12.0 * n * k + 8.0 * SYM * n * k + 4.0 * n,
                "flops": 2.0 * n * n * case["dim"]}
    return {"bytes": 12.0 * n * k + 8.0 * SYM * n * k + 8.0 * n, "flops": 20 * 3.0 * n * k}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
# points per axis that the interpolation grid is rounded up to (sizes of the
# reference's transform table)
GRID = [8, 9, 10, 11, 12, 13, 14, 15, 16, 20, 25, 26, 28, 32, 33, 35, 36, 39, 40, 42, 44, 45, 48,
        49, 50, 52, 54, 55, 56, 60, 63, 64, 65, 66, 70, 72, 75, 77, 78, 80, 84, 88, 90, 91, 96, 98,
        99, 100, 104, 105, 108, 110, 112, 117, 120, 125, 126, 130, 132, 135, 140, 144, 147, 150,
        154, 156, 160, 165, 168, 175, 176, 180, 182, 189, 192, 195, 196, 198, 200, 208, 210, 216,
        220, 224, 225, 231, 234, 240, 245, 250, 252, 260, 264, 270, 273, 275, 280, 288, 294, 297,
        300, 308, 312, 315, 320, 325, 330, 336, 343, 350, 351, 352, 360, 364, 375, 378, 385, 390,
        392, 396, 400, 416, 420, 432, 440, 441, 448, 450, 455, 462, 468, 480, 490, 495, 500, 504,
        512]


def _repulsion64(y, h, most):
    """Interpolated repulsive force (cubic Lagrange nodes) over its Z."""
    n, d = y.shape
    lo = torch.minimum(y.min(0)[0], torch.full((d,), 100.0, dtype=y.dtype, device=DEV))
    s = y - lo
    maxy = float(s.max())
    want = max(int(math.ceil(np.float32(maxy) / np.float32(h))), 14) + 2
    N = next((g for g in GRID if g >= want and g <= most), most)
    step = maxy / (N - 3)
    t = (s / maxy).clamp_max(1.0 - float(np.finfo(np.float32).eps)) * (N - 3)
    f = t.floor()
    u = t - f
    f = f.to(torch.int64)

    def l1(v):
        return 0.5 * v ** 3 - v ** 2 - 0.5 * v + 1.0

    def l2(v):
        return -v ** 3 / 6.0 + v ** 2 - 11.0 / 6.0 * v + 1.0

    w = [l2(1.0 + u), l1(u), l1(1.0 - u), l2(2.0 - u)]
    c = s - 0.5 * maxy
    q = torch.cat([torch.ones(n, 1, dtype=y.dtype, device=DEV), c], 1)
    places = []
    for e in range(4 ** d):
        a = [(e >> (2 * k)) & 3 for k in range(d)]
        wt, at = w[a[0]][:, 0], f[:, 0] + a[0]
        for k in range(1, d):
            wt, at = wt * w[a[k]][:, k], at + (f[:, k] + a[k]) * N ** k
        places.append((at, wt))
    grid = torch.zeros(d + 1, N ** d, dtype=y.dtype, device=DEV)
    for at, wt in places:
        for ch in range(d + 1):
            grid[ch] += torch.bincount(at, wt * q[:, ch], N ** d)
    M = 2 * N
    r = torch.arange(M, device=DEV)
    r = torch.minimum(r, M - r).to(y.dtype) * step
    r2 = torch.zeros((M,) * d, dtype=y.dtype, device=DEV)
    for k in range(d):
        r2 = r2 + (r ** 2).reshape([-1 if j == k else 1 for j in range(d)])
    dims = tuple(range(1, d + 1))
    spec = torch.fft.rfftn((1.0 / (1.0 + r2) ** 2)[None], dim=dims)
    phi = torch.fft.irfftn(torch.fft.rfftn(grid.reshape((d + 1,) + (N,) * d), s=(M,) * d, dim=dims)
                           * spec, s=(M,) * d, dim=dims)
    phi = phi[(slice(None),) + (slice(0, N),) * d].reshape(d + 1, -1)
    p = torch.zeros(n, d + 1, dtype=y.dtype, device=DEV)
    for at, wt in places:
        for ch in range(d + 1):
            p[:, ch] += wt * phi[ch][at]
    z = float(((1.0 + 2.0 * (c * c).sum(1)) * p[:, 0] - 2.0 * (c * p[:, 1:]).sum(1)).sum()) - n
    return (c * p[:, :1] - p[:, 1:]) / z


def _attraction64(y, row, col, val):
    out = torch.zeros_like(y)
    for a in range(0, col.numel(), 1 << 24):
        r, c = row[a:a + (1 << 24)], col[a:a + (1 << 24)].to(torch.int64)
        df = y[r] - y[c]
        pq = val[a:a + (1 << 24)].to(y.dtype) / (1.0 + (df * df).sum(1))
        for k in range(y.shape[1]):
            out[:, k] += torch.bincount(r, pq * df[:, k], y.shape[0])
    return out


def _iterate64(case, p, y, d):
    rowptr, col, val = p
    n = y.shape[0]
    row = torch.repeat_interleave(torch.arange(n, device=DEV), (rowptr[1:] - rowptr[:-1]).long())
    y = y.double()
    vel, gain = torch.zeros_like(y), torch.ones_like(y)
    for _ in range(case["iters"]):
        y = y - y.mean(0)
        dy = case["alpha"] * _attraction64(y, row, col, val) - _repulsion64(
            y, H[d], 512 if d < 3 else 128)
        gain = torch.where(torch.sign(dy) != torch.sign(vel), gain + 0.2, gain * 0.8)
        gain = gain.clamp_min(0.01)
        vel = 0.5 * vel - 200.0 * gain * dy
        y = y + vel
    return y - y.mean(0)


def _perplexity64(d2, perplexity):
    """(P, beta) by the bisection on the entropy, tolerance 1e-5."""
    d2 = d2.double()
    n = d2.shape[0]
    beta = torch.ones(n, dtype=torch.float64, device=DEV)
    lo, hi = torch.zeros_like(beta), torch.full_like(beta, math.inf)
    found, used = torch.zeros(n, dtype=torch.bool, device=DEV), beta.clone()
    has_lo = torch.zeros_like(found)
    total = torch.ones_like(beta)
    for _ in range(200):
        e = torch.exp(-beta[:, None] * d2)
        sums = e.sum(1) + float(np.finfo(np.float64).tiny)
        diff = (beta[:, None] * d2 * e).sum(1) / sums + torch.log(sums) - math.log(perplexity)
        used, total = torch.where(found, used, beta), torch.where(found, total, sums)
        found = found | (diff.abs() < 1e-5)
        if bool(found.all()):
            break
        up = diff > 0
        lo, hi = torch.where(~found & up, beta, lo), torch.where(~found & ~up, beta, hi)
        has_lo = has_lo | (~found & up)
        step = torch.where(up, torch.where(torch.isinf(hi), beta * 2.0, (beta + hi) / 2.0),
                           torch.where(has_lo, (beta + lo) / 2.0, beta / 2.0))
        beta = torch.where(found, beta, step)
    return torch.exp(-used[:, None] * d2) / total[:, None], used


def _lambda64(d2, lam):
    """(rows of exp(-s d2) / sum, s) with sum exp(-s d2) = lam, bisection to 1e-5."""
    d2 = d2.double()
    n = d2.shape[0]
    sig = torch.ones(n, dtype=torch.float64, device=DEV)
    a, c = torch.full_like(sig, -1e3), torch.full_like(sig, math.inf)
    f = torch.exp(-d2).sum(1) - lam
    for _ in range(100):
        on = f.abs() > 1e-5
        if not bool(on.any()):
            break
        up = on & (f > 0)
        dn = on & ~(f > 0)
        a, c = torch.where(up, sig, a), torch.where(dn, sig, c)
        new = torch.where(up & torch.isinf(c), 2.0 * a, 0.5 * (a + c))
        sig = torch.where(on, new, sig)
        f = torch.where(on, torch.exp(-sig[:, None] * d2).sum(1) - lam, f)
    e = torch.exp(-sig[:, None] * d2)
    return e / e.sum(1, keepdim=True), sig


def exact(case, seed):
    what = case["what"]
    if what == "iterate":
        inp = _inputs(case, seed)
        return _iterate64(case, inp["p"], inp["y"], case["d"])
    if what == "batch":
        outs = []
        for i, (n, d) in enumerate(_batch_sizes(case)):
            inp = _inputs(case, seed * 1000 + i, n, d)
            outs.append(_iterate64(case, inp["p"], inp["y"], d))
        return outs
    n, k = case["n"], case["k"]
    inp = _inputs(case, seed)
    if what == "embed":
        val = inp["d2"].double()
        if case["lambda"] == 1.0:
            w = torch.exp(-inp["d2"] / inp["d2"].mean(1, keepdim=True)).double() / k
        else:
            w = _lambda64(val, case["lambda"])[0]
        y = _iterate64(case, _symmetric(n, inp["idx"], w), inp["y"], case["d"])
        return y.cpu().numpy()
    if what == "graph":
        x = inp["x"].double()
        d2 = torch.empty(n, k, dtype=torch.float64, device=DEV)
        for a in range(0, n, 2048):
            q = x[a:a + 2048]
            dist = (q * q).sum(1)[:, None] + (x * x).sum(1)[None] - 2.0 * (q @ x.T)
            dist[torch.arange(q.shape[0], device=DEV),
                 torch.arange(a, a + q.shape[0], device=DEV)] = math.inf
            d2[a:a + 2048] = torch.topk(dist, k, dim=1, largest=False)[0]
    else:
        d2 = inp["d2"].double()
    p, beta = (_perplexity64(d2, case["perplexity"]) if "perplexity" in case else
               _lambda64(d2, case["lambda"]))
    sv = None
    if what == "affinity":
        val = _symmetric(n, inp["idx"], p)[2]
        sv = torch.zeros(2 * n * k, dtype=torch.float64, device=DEV)
        sv[:val.numel()] = val
    return {"idx": None, "d2": d2, "p": p, "beta": beta, "srp": None, "sc": None, "sv": sv,
            "nnz": None}
