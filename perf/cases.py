"""What the framework is timed on: passes through its public entry points, from a thumbnail
to the largest grids of its benchmark.

Images follow the construction of ``synth.py`` (12 filled ellipses, Gaussian blur of sigma 3,
N(0, 8) noise; t-links 100 * (score_bg - score_fg) under colour models of two ellipses;
n-links 50 * exp(-beta |dI|^2)), made on the GPU so that making them is quick.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("cl-util_b200"))

import strokes  # noqa: E402
from gmm_tlinks import Mixture, components  # noqa: E402
from GMM import GMM  # noqa: E402
from GraphCut import GraphCut  # noqa: E402
from GraphCutBatch import GraphCutBatch  # noqa: E402
from IncrementalTileList import IncrementalTileList, Logical, Operator  # noqa: E402
from PrefixSum import PrefixSum  # noqa: E402
from session_pool import SessionPool, tiles_of  # noqa: E402
from StreamCompact import StreamCompact  # noqa: E402


def listed():
    return [
        # a thumbnail or preview cut, from ready capacity planes: latency and launches
        {"name": "cut_256x192", "kind": "cut", "w": 256, "h": 192},
        # the plain single cut of a small picture
        {"name": "cut_512x512", "kind": "cut", "w": 512, "h": 512},
        # the benchmark's single grid
        {"name": "cut_2048x2048", "kind": "cut", "w": 2048, "h": 2048},
        # a picture of no round size, weighted by the reference's own lamda rule, whose n-links
        # are large against the t-links: a solve of many cycles
        {"name": "lamda_803x607", "kind": "image", "w": 803, "h": 607, "lamda": 60},
        # a 16.8 Mpix photo straight from its RGBA words and t-links
        {"name": "image_4096x4096", "kind": "image", "w": 4096, "h": 4096, "lamda": 0},
        # a video frame with two fitted colour models: t-links, n-links and cut on the device
        {"name": "models_1920x1080", "kind": "models", "w": 1920, "h": 1080, "k": 4},
        # the colour model of a stroke's pixels (65 iterations of 4 components, as the
        # reference's fit test runs it)
        {"name": "gmm_fit_10000x4", "kind": "fit", "n": 10000, "k": 4, "iters": 65},
        # a job of many uneven pictures solved together
        {"name": "batch_64", "kind": "batch", "n": 64, "lo": 256, "hi": 1536, "step": 128},
        # an interactive edit of a large photo: one stroke, then the warm cut
        {"name": "stroke_4096x4096", "kind": "stroke", "w": 4096, "h": 4096},
        # one tick of a server: some new images and some strokes on resident ones, one solve
        {"name": "serve_12", "kind": "serve", "n": 12, "new": 4, "lo": 256, "hi": 2048},
        # the tile list of an 8192^2 image with 16^2 tiles, the largest the reference timed
        {"name": "tiles_8192x8192", "kind": "tiles", "w": 8192, "h": 8192, "tile": 16},
        # the primitives beneath it at a length that no vector width divides
        {"name": "scan_3000017", "kind": "scan", "n": 3000017},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cut", "cut", "image", "image", "models", "fit", "batch", "stroke", "serve",
                       "tiles", "scan"])
    if kind == "fit":
        return {"kind": kind, "n": _log_int(rng, 500, 20000), "k": rng.randint(2, 5),
                "iters": rng.randint(20, 65)}
    if kind == "batch":
        return {"kind": kind, "n": rng.randint(4, 48), "lo": rng.randint(60, 300),
                "hi": rng.randint(400, 1536), "step": rng.choice([1, 7, 32, 128])}
    if kind == "serve":
        n = rng.randint(2, 12)
        return {"kind": kind, "n": n, "new": rng.randint(0, min(n, 4)), "lo": rng.randint(100, 300),
                "hi": rng.randint(500, 2048)}
    if kind == "tiles":
        return {"kind": kind, "w": _log_int(rng, 400, 8192), "h": _log_int(rng, 300, 8192),
                "tile": rng.choice([16, 32])}
    if kind == "scan":
        return {"kind": kind, "n": _log_int(rng, 450, 3000000)}
    case = {"kind": kind, "w": _log_int(rng, 100, 4096), "h": _log_int(rng, 100, 4096)}
    if kind == "image":
        # the lamda rule up to 1 Mpix: its solves take many more cycles a pixel
        case["lamda"] = rng.choice([0, 0, rng.randint(1, 120)])
        if case["lamda"]:
            case["w"], case["h"] = min(case["w"], 1024), min(case["h"], 1024)
    if kind == "models":
        case["k"] = rng.randint(1, 6)
    return case


# ---- inputs ---------------------------------------------------------------------------------
def _picture(w, h, seed):
    """int32 RGBA words [h, w], and two boxes (x, y, a, b) inside two of the ellipses."""
    rng = np.random.default_rng(seed)
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    img = torch.empty((3, h, w), dtype=torch.float32, device=dev)
    img[:] = torch.tensor(rng.integers(0, 256, 3), dtype=torch.float32, device=dev)[:, None, None]
    short = min(w, h)
    boxes = []
    for _ in range(12):
        cx, cy = rng.uniform(0, w), rng.uniform(0, h)
        a, b = rng.uniform(0.05, 0.30, 2) * short
        th = rng.uniform(0.0, math.pi)
        colour = torch.tensor(rng.integers(0, 256, 3), dtype=torch.float32, device=dev)
        r = max(a, b)
        x0, x1 = max(0, int(cx - r)), min(w, int(cx + r) + 1)
        y0, y1 = max(0, int(cy - r)), min(h, int(cy + r) + 1)
        ys = torch.arange(y0, y1, device=dev, dtype=torch.float32)[:, None] - cy
        xs = torch.arange(x0, x1, device=dev, dtype=torch.float32)[None, :] - cx
        u = (xs * math.cos(th) + ys * math.sin(th)) / a
        v = (ys * math.cos(th) - xs * math.sin(th)) / b
        part = img[:, y0:y1, x0:x1]
        part.copy_(torch.where((u * u + v * v <= 1.0)[None], colour[:, None, None], part))
        boxes.append((cx, cy, 0.6 * min(a, b)))
    tap = np.exp(-0.5 * (np.arange(-12, 13) / 3.0) ** 2)
    tap /= tap.sum()
    for axis in (1, 2):
        pad = (0, 0, 12, 12) if axis == 1 else (12, 12, 0, 0)
        p = torch.nn.functional.pad(img[None], pad, mode="replicate")[0]
        img = torch.zeros_like(img)
        for k in range(25):
            img.add_(p.narrow(axis, k, h if axis == 1 else w), alpha=float(tap[k]))
    img += 8.0 * torch.randn(img.shape, generator=gen, device=dev)
    q = torch.clamp(torch.floor(img + 0.5), 0, 255).to(torch.int32)
    words = q[0] | (q[1] << 8) | (q[2] << 16) | (-1 << 24)
    two = rng.choice(12, 2, replace=False)
    return words.contiguous(), [boxes[i] for i in two], rng


def _stroke_pixels(words, box, n, rng):
    """Colours [n, 3] under a stroke inside the ellipse (clipped to the picture)."""
    h, w = words.shape
    cx, cy, r = box
    x = np.clip(cx + rng.uniform(-r, r, n), 0, w - 1).astype(np.int64)
    y = np.clip(cy + rng.uniform(-r, r, n), 0, h - 1).astype(np.int64)
    return words.reshape(-1)[torch.from_numpy(y * w + x).to(words.device)]


def _rgb(words):
    v = words.cpu().numpy().astype(np.int64)
    return np.stack([v & 255, (v >> 8) & 255, (v >> 16) & 255], 1).astype(np.float64)


def _model(x, k, rng):
    """A k-component full-covariance mixture of the colours x: a few EM steps."""
    mu = x[rng.choice(len(x), k, replace=False)] + rng.normal(0, 1, (k, 3))
    cov = np.stack([np.cov(x.T) + np.eye(3)] * k)
    wt = np.full(k, 1.0 / k)
    for _ in range(8):
        lp = np.empty((len(x), k))
        for j in range(k):
            d = x - mu[j]
            lp[:, j] = (np.log(wt[j]) - 0.5 * np.linalg.slogdet(cov[j])[1]
                        - 0.5 * np.einsum("ni,ij,nj->n", d, np.linalg.inv(cov[j]), d))
        r = np.exp(lp - lp.max(1, keepdims=True))
        r /= r.sum(1, keepdims=True)
        nk = r.sum(0) + 1e-6
        wt = nk / nk.sum()
        mu = (r.T @ x) / nk[:, None]
        for j in range(k):
            d = x - mu[j]
            cov[j] = (r[:, j, None] * d).T @ d / nk[j] + np.eye(3)
    return wt, mu, cov


def _score(words, model):
    """-log p of every pixel under the mixture, float64 [h, w]."""
    ch = [((words >> s) & 255).double() for s in (0, 8, 16)]
    terms = []
    for c in components(*model):
        c = [float(v) for v in c]
        d = [ch[i] - c[1 + i] for i in range(3)]
        y0 = c[4] * d[0]
        y1 = c[5] * d[0] + c[6] * d[1]
        y2 = c[7] * d[0] + c[8] * d[1] + c[9] * d[2]
        terms.append(c[0] - 0.5 * (y0 * y0 + y1 * y1 + y2 * y2))
    return -torch.logsumexp(torch.stack(terms), 0)


def _tlinks(words, models):
    t = torch.floor(100.0 * (_score(words, models[1]) - _score(words, models[0])) + 0.5)
    return torch.clamp(t, -10 ** 6, 10 ** 6).to(torch.int32)


def _planes(words, excess):
    """The five int32 capacity planes of a picture."""
    ch = [(words >> s) & 255 for s in (0, 8, 16)]
    dv = sum((c[1:] - c[:-1]) ** 2 for c in ch)
    dh = sum((c[:, 1:] - c[:, :-1]) ** 2 for c in ch)
    mean = float(dv.sum() + dh.sum()) / max(1, dv.numel() + dh.numel())
    beta = 1.0 / (2.0 * mean) if mean > 0 else 0.0
    wv = torch.floor(50.0 * torch.exp(-beta * dv.double()) + 0.5).to(torch.int32)
    wh = torch.floor(50.0 * torch.exp(-beta * dh.double()) + 0.5).to(torch.int32)
    up, down, left, right = (torch.zeros_like(excess) for _ in range(4))
    up[1:], down[:-1], left[:, 1:], right[:, :-1] = wv, wv, wh, wh
    return up, down, left, right, excess


def _scene(w, h, seed, k=2):
    words, boxes, rng = _picture(w, h, seed)
    models = [_model(_rgb(_stroke_pixels(words, b, 1000, rng)), k, rng) for b in boxes]
    return words, models, rng


def _sides(case, rng):
    """Sizes of a batch's or a server's images."""
    sides = np.arange(case["lo"], case["hi"] + 1, case.get("step", 1))
    return [(int(rng.choice(sides)), int(rng.choice(sides))) for _ in range(case["n"])]


def _shapes(case):
    """Sizes that go with the case, not with the inputs' seed: every pass costs alike."""
    return _sides(case, np.random.default_rng([case["n"], case["lo"], case["hi"]]))


def _edits(w, h, rng, n=24):
    return [strokes.random_stroke(rng, w, h) for _ in range(n)]


def _edit(target, args, edits, k):
    """The k-th edit of a session: the list again and again, each round with the signs
    turned, so that every pass changes its pixels."""
    s = edits[k % len(edits)]
    target(*args, s.xs, s.ys, s.radius, -s.value if (k // len(edits)) & 1 else s.value)


def prepare(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda")
    if kind in ("cut", "image", "models", "stroke"):
        w, h = case["w"], case["h"]
        words, models, rng = _scene(w, h, seed, case.get("k", 2))
        gc = GraphCut(w, h)
        out = torch.empty((h, w), dtype=torch.uint8, device=dev)
        state = {"kind": kind, "gc": gc, "out": out, "words": words}
        if kind == "models":
            state["models"] = tuple(Mixture(*m) for m in models)
            return state
        excess = _tlinks(words, models)
        if kind == "image":
            state.update(excess=excess, lamda=case["lamda"] or None)
            return state
        state["planes"] = _planes(words, excess)
        if kind == "stroke":
            gc.upload_capacities(*state.pop("planes"))
            gc.cut_labels(out=out)
            state.update(edits=_edits(w, h, rng), k=0)
        return state
    if kind == "batch":
        shapes = _shapes(case)
        graphs = []
        for i, (w, h) in enumerate(shapes):
            words, models, _ = _scene(w, h, 1000 * seed + i)
            graphs.append(_planes(words, _tlinks(words, models)))
        flat = torch.empty(sum(w * h for w, h in shapes), dtype=torch.uint8, device=dev)
        outs = [v.view(h, w) for v, (w, h) in zip(flat.split([w * h for w, h in shapes]), shapes)]
        return {"kind": kind, "batch": GraphCutBatch(shapes), "graphs": graphs, "flat": flat,
                "outs": outs}
    if kind == "serve":
        shapes = _shapes(case)
        rng = np.random.default_rng(seed)
        pool = SessionPool(sum(tiles_of(w, h) for w, h in shapes), len(shapes))
        state = {"kind": kind, "pool": pool, "slots": list(range(len(shapes))), "new": case["new"],
                 "inputs": [], "edits": [], "k": 0, "outs": []}
        for s, (w, h) in enumerate(shapes):
            pool.open(s, w, h, pool.alloc_tiles(w, h))
            words, models, _ = _scene(w, h, 1000 * seed + s)
            inputs = (words, _tlinks(words, models))
            pool.upload_image(s, *inputs)
            state["inputs"].append(inputs if s < case["new"] else None)
            state["edits"].append(_edits(w, h, rng))
            state["outs"].append(torch.empty((h, (w + 7) // 8), dtype=torch.uint8, device=dev))
        pool.solve_labels(state["slots"], state["outs"])
        return state
    rng = np.random.default_rng(seed)
    if kind == "fit":
        n = case["n"]
        words, boxes, rng = _picture(512, 384, seed)
        return {"kind": kind, "samples": _stroke_pixels(words, boxes[0], n, rng),
                "gmm": GMM(case["iters"], case["k"])}
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    if kind == "tiles":
        tl = IncrementalTileList((case["w"], case["h"]), (case["tile"], case["tile"]))
        tl.d_tiles.copy_(torch.randint(-1, 1, tl.d_tiles.shape, generator=gen, device=dev))
        other = torch.randint(0, 20, tl.d_tiles.shape, generator=gen, device=dev, dtype=torch.int32)
        return {"kind": kind, "list": tl, "other": other}
    n = case["n"]
    flags = (torch.rand(n, generator=gen, device=dev) < 0.35).to(torch.int32)
    sc = StreamCompact(n)
    return {"kind": kind, "flags": flags, "compact": sc, "scan": PrefixSum(n),
            "list": sc.listFactory(), "array": torch.empty_like(flags),
            "length": torch.zeros(1, dtype=torch.int32, device=dev),
            "total": torch.zeros(1, dtype=torch.int32, device=dev)}


# ---- one pass -------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "cut":
        gc = state["gc"]
        gc.upload_capacities(*state["planes"])
        return {"labels": gc.cut_labels(out=state["out"]), "flow": gc.flow}
    if kind == "image":
        gc = state["gc"]
        gc.upload_image(state["words"], state["excess"], lamda=state["lamda"])
        return {"labels": gc.cut_labels(out=state["out"]), "flow": gc.flow}
    if kind == "models":
        gc = state["gc"]
        gc.upload_image(state["words"], state["models"])
        return {"labels": gc.cut_labels(out=state["out"]), "flow": gc.flow}
    if kind == "stroke":
        gc, k = state["gc"], state["k"]
        _edit(gc.edit_stroke, (), state["edits"], k)
        state["k"] = k + 1
        return {"labels": gc.cut_labels(out=state["out"]), "flow": gc.flow}
    if kind == "batch":
        b = state["batch"]
        for i, planes in enumerate(state["graphs"]):
            b.upload(i, *planes)
        b.cut()
        for i, out in enumerate(state["outs"]):
            b.labels(i, out=out)
        return {"labels": state["flat"],
                "flow": np.array([b.flow(i) for i in range(len(b))], np.int64)}
    if kind == "serve":
        pool, k = state["pool"], state["k"]
        for s in state["slots"]:
            if s < state["new"]:
                pool.upload_image(s, *state["inputs"][s])
            else:
                _edit(pool.edit_stroke, (s,), state["edits"][s], k)
        state["k"] = k + 1
        outs = pool.solve_labels(state["slots"], state["outs"])
        return {"labels": outs, "flow": np.array([pool.flow(s) for s in state["slots"]], np.int64)}
    if kind == "fit":
        gmm = state["gmm"]
        weights, means, covars = gmm.fit(state["samples"], retParams=True)
        return {"weights": weights, "means": means, "covars": covars,
                "log_likelihood": gmm.log_likelihood, "iterations": gmm.iterations}
    if kind == "tiles":
        tl = state["list"]
        tl.increment()
        tl.incorporate(state["other"], Operator.GTE, 0, Operator.GTE, 10, Logical.AND)
        tl.build()
        return {"length": tl.length, "list": tl.d_list}
    state["compact"].compact(state["flags"], state["list"], state["length"])
    state["array"].copy_(state["flags"])   # the scan works in place
    state["scan"].scan(state["array"], state["total"])
    return {"list": state["list"], "length": state["length"], "scan": state["array"],
            "total": state["total"]}


def work(case):
    kind = case["kind"]
    if kind == "cut":        # five planes in, one label byte out
        return {"bytes": 21 * case["w"] * case["h"], "flops": 0}
    if kind == "image":      # RGBA word and t-link in, label out
        return {"bytes": 9 * case["w"] * case["h"], "flops": 0}
    if kind == "models":     # RGBA word in, label out; two mixtures of k components a pixel
        n = case["w"] * case["h"]
        return {"bytes": 5 * n, "flops": 2 * case["k"] * 24 * n}
    if kind == "stroke":     # the labels come whole
        return {"bytes": case["w"] * case["h"], "flops": 0}
    if kind == "batch":
        return {"bytes": 21 * sum(w * h for w, h in _shapes(case)), "flops": 0}
    if kind == "serve":
        px = [w * h for w, h in _shapes(case)]
        return {"bytes": 8 * sum(px[:case["new"]]) + sum(px) // 8, "flops": 0}
    if kind == "fit":        # a density, a responsibility and ten moments a sample and component
        return {"bytes": 4 * case["n"], "flops": 60 * case["n"] * case["k"] * case["iters"]}
    if kind == "tiles":      # two maps read, half the stamps written, the list written
        t = (case["w"] // case["tile"]) * (case["h"] // case["tile"])
        return {"bytes": 12 * t, "flops": 0}
    return {"bytes": 8 * case["n"] + int(1.4 * case["n"]) + 4 * case["n"], "flops": 0}


def exact(case, seed):
    """The fit in float64 numpy; the other outputs are whole numbers."""
    if case["kind"] != "fit":
        return None
    x = _rgb(prepare(case, seed)["samples"])
    n, k, iters = case["n"], case["k"], case["iters"]
    mu = x[[j * (n - 1) // (k - 1) if k > 1 else 0 for j in range(k)]].copy()
    var, wt, last, t = np.full((k, 3), 30.0), np.full(k, 1.0 / k), 0.0, 0
    while True:
        with np.errstate(divide="ignore"):
            c = np.log(wt) - 0.5 * (3 * np.log(2 * np.pi) + np.log(var).sum(1))
        e = c - 0.5 * ((x[:, None] - mu) ** 2 / var).sum(2)
        m = e.max(1, keepdims=True)
        lp = m + np.log(np.exp(e - m).sum(1, keepdims=True))
        like = math.fsum(lp[:, 0])
        done = t >= 1 and t - 1 > 1 and abs(like - last) < 0.01
        last = like if t >= 1 else last
        if done or t == iters:
            break
        r = np.exp(e - lp)
        nk = r.sum(0)
        live = nk > 0
        wt = np.where(live, nk / nk.sum(), 0.0)
        for j in np.flatnonzero(live):
            mu[j] = (r[:, j, None] * x).sum(0) / nk[j]
            var[j] = (r[:, j, None] * x * x).sum(0) / nk[j] - mu[j] ** 2 + 1e-3
        t += 1
    return {"weights": wt, "means": mu, "covars": var, "log_likelihood": like, "iterations": None}
