"""Workloads for timing the framework through its public entry points.

Three kinds of call: one field through ``compute_dmsc`` (on the device, or as
a CPU tensor, the reference's calling convention), a list of uneven fields
through ``compute_dmsc_batched``, and a forward and backward pass of the
topological denoising loss. Sizes, bump counts and noise levels are those of
the benchmark, the tests and the synthetic generators of this repository; the
fields are made on the GPU from the seed alone.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from dmsc_b200 import compute_dmsc, compute_dmsc_batched
from dmsc_b200.autograd import topological_loss

# Fields of one complex whose sizes depend on the values, and those of the
# image's size (the image shape apart).
_LISTS = ("max_pts", "min_pts", "sad_pts", "e_max", "e_min", "p_max", "p_min", "ppairs_max", "ppairs_min", "ridges",
          "ridge_offsets", "ridge_arc_offsets", "valleys", "valley_offsets", "valley_arc_offsets")
_MAPS = ("grad_indices", "peaks", "basins")


def _one(name, H, W, field, thr, **more):
    return dict(name=name, kind="one", H=H, W=W, field=field, thr=thr, **more)


def listed():
    return [
        # the reference's fixture size: a call whose time is launches and host round trips
        _one("landscape_32", 32, 32, "landscape", 0.1, dual=False),
        # one patch, analysed as it comes: the smallest configuration of the benchmark
        _one("bumps_256", 256, 256, "bumps", 0.1, sigma_lo=8.0, sigma_hi=32.0, noise=0.05, per_bump=2730, dual=False),
        # an odd-sized scan (no row is a multiple of 16 bytes), dual orientation
        _one("scan_509x1531_dual", 509, 1531, "bumps", 0.05, sigma_lo=4.0, sigma_hi=32.0, noise=0.03, per_bump=8000,
             dual=True),
        # an 8-bit video frame converted to float: large plateaus, most comparisons are ties
        _one("frame8bit_1080x1920", 1080, 1920, "bumps", 0.05, sigma_lo=4.0, sigma_hi=64.0, noise=0.02, per_bump=8389,
             levels=256, dual=False),
        # a CPU caller wanting gradient and segmentation: input uploaded, every output back in host memory
        _one("host_1024", 1024, 1024, "bumps", 0.05, sigma_lo=4.0, sigma_hi=64.0, noise=0.02, per_bump=8389,
             dual=False, arcs=False, host=True),
        # the resolution and the larger threshold of the reference's own benchmark script
        _one("bumps_2048_thr0.25", 2048, 2048, "bumps", 0.25, sigma_lo=4.0, sigma_hi=64.0, noise=0.02, per_bump=8389,
             dual=False),
        # the headline field, simplified: cancellation, replay and arc geometry
        _one("bumps_4096", 4096, 4096, "bumps", 0.05, sigma_lo=4.0, sigma_hi=64.0, noise=0.02, per_bump=8389,
             dual=False),
        # the headline field, unsimplified, dual: every saddle survives into the outputs
        _one("bumps_4096_dual_raw", 4096, 4096, "bumps", 0.0, sigma_lo=4.0, sigma_hi=64.0, noise=0.02, per_bump=8389,
             dual=True),
        # watershed segmentation only (labels and pairs; no gradient, no arcs) of an odd-sized mosaic
        _one("segment_3001x4099", 3001, 4099, "bumps", 0.05, sigma_lo=4.0, sigma_hi=64.0, noise=0.02, per_bump=8389,
             dual=False, gradient=False, arcs=False),
        # the densest critical cells a field can have: i.i.d. uniform values, the largest call
        _one("uniform_8192", 8192, 8192, "uniform", 0.0, dual=False),
        # a data set of uneven images, thresholds and orientations analysed in one call
        dict(name="batch_48_uneven", kind="batch", n=48, lo=64, hi=2048),
        # one step of topological denoising: forward and backward of the persistence loss
        dict(name="train_8x512", kind="train", B=8, H=512, W=512, noise=0.05, dual=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    u = rng.random()
    if u < 0.15:
        return dict(kind="batch", n=_log_int(rng, 2, 64), lo=64, hi=_log_int(rng, 128, 2048))
    if u < 0.3:
        return dict(kind="train", B=_log_int(rng, 1, 12), H=_log_int(rng, 48, 512), W=_log_int(rng, 48, 512),
                    noise=rng.choice([0.02, 0.05]), dual=rng.random() < 0.5)
    H, W = _log_int(rng, 24, 4096), _log_int(rng, 24, 4096)
    if rng.random() < 0.3:
        H, W = 16 * max(2, H // 16), 16 * max(2, W // 16)
    dual, v = rng.random() < 0.5, rng.random()
    if v < 0.2:  # unsimplified (a threshold above 0 joins nearly all of a uniform field's arcs into one)
        return dict(kind="one", H=H, W=W, field="uniform", thr=0.0, dual=dual, gradient=rng.random() < 0.5)
    case = dict(kind="one", H=H, W=W, field="bumps", thr=rng.choice([0.0, 0.02, 0.05, 0.1, 0.2]), dual=dual,
                sigma_lo=4.0, sigma_hi=rng.choice([32.0, 64.0]), noise=rng.choice([0.02, 0.03, 0.05]),
                per_bump=rng.choice([2730, 8000, 8389]))
    if v < 0.35:
        case["levels"] = rng.choice([256, 4096])
    elif v < 0.55:
        case.update(gradient=False, arcs=False)
    elif v < 0.65:
        case.update(host=True, arcs=False, thr=rng.choice([0.05, 0.1, 0.2]))
    return case


def _generators(seed):
    return torch.Generator().manual_seed(seed), torch.Generator(device="cuda").manual_seed(seed)


def _bumps(H, W, per_bump, sigma_lo, sigma_hi, noise, gens):
    """Gaussian bumps of amplitude U[-1, 1] with N(0, noise^2) noise, one bump
    per ``per_bump`` pixels; a bump is separable, so the sum is one product."""
    g, gd = gens
    n = max(1, math.ceil(H * W / per_bump))
    cy, cx, a, s = (torch.rand(n, generator=g) for _ in range(4))
    cy, cx, a, s = (t.to("cuda") for t in (cy * H, cx * W, a * 2 - 1, s * (sigma_hi - sigma_lo) + sigma_lo))
    ys, xs = torch.arange(H, device="cuda"), torch.arange(W, device="cuda")
    ey = a[:, None] * torch.exp(-((ys[None, :] - cy[:, None]) ** 2) / (2 * s * s)[:, None])
    ex = torch.exp(-((xs[None, :] - cx[:, None]) ** 2) / (2 * s * s)[:, None])
    return ey.t() @ ex + noise * torch.randn(H, W, generator=gd, device="cuda")


def _landscape(H, W, gens):
    """Two peaks and two valleys with U[-0.05, 0.05) noise (the fixtures' field)."""
    y, x = torch.meshgrid(torch.linspace(-2, 2, H), torch.linspace(-2, 2, W), indexing="ij")
    z = (torch.exp(-((x - 1) ** 2 + y ** 2) / 0.5) + torch.exp(-((x + 1) ** 2 + y ** 2) / 0.5)
         - 0.5 * torch.exp(-(x ** 2 + (y - 1) ** 2) / 0.5) - torch.exp(-(x ** 2 + (y + 1) ** 2) / 0.5))
    return z.to("cuda") + 0.1 * (torch.rand(H, W, generator=gens[1], device="cuda") - 0.5)


def _field(case, seed):
    gens = _generators(seed)
    H, W = case["H"], case["W"]
    if case["field"] == "uniform":
        return torch.rand(H, W, generator=gens[1], device="cuda")
    if case["field"] == "landscape":
        return _landscape(H, W, gens)
    z = _bumps(H, W, case["per_bump"], case["sigma_lo"], case["sigma_hi"], case["noise"], gens)
    if "levels" in case:
        n = case["levels"] - 1
        lo, hi = z.min(), z.max()
        z = torch.round((z - lo) / (hi - lo) * n) / n
    return z


def _batch(case, seed):
    """The batch's sizes, thresholds and orientations go with the case, its
    images' values with the seed."""
    mix = torch.Generator().manual_seed(7919 * case["n"] + case["hi"])
    gens = _generators(seed)
    images, thr, dual = [], [], []
    span = math.log(case["hi"] / case["lo"])
    for _ in range(case["n"]):
        h, w, t, d = torch.rand(4, generator=mix).tolist()
        h, w = (int(round(case["lo"] * math.exp(u * span))) for u in (h, w))
        images.append(_bumps(h, w, 8000, 4.0, 32.0, 0.03, gens))
        thr.append(0.02 + 0.18 * t)
        dual.append(d < 0.5)
    return images, thr, dual


def _train_batch(case, seed):
    gens = _generators(seed)
    B, H, W = case["B"], case["H"], case["W"]
    x = torch.stack([_bumps(H, W, 1311, 4.0, 32.0, case["noise"], gens) for _ in range(B)])
    rank = torch.rand(B, H * W, generator=gens[1], device="cuda").argsort(dim=1).reshape(B, H, W)
    return x + 1e-6 * rank / (H * W)


def _record(npx, device):
    """Buffer of one call's lists back to back: all of them together have
    less than 10 entries per pixel on these fields."""
    return torch.zeros(10 * npx + 4096, dtype=torch.int32, device=device)


def prepare(case, seed):
    if case["kind"] == "batch":
        images, thr, dual = _batch(case, seed)
        return dict(kind="batch", images=images, thr=thr, dual=dual,
                    record=_record(sum(x.numel() for x in images), "cuda"))
    if case["kind"] == "train":
        return dict(kind="train", x=_train_batch(case, seed).requires_grad_(), dual=case["dual"])
    img = _field(case, seed)
    if case.get("host"):
        img = img.cpu()
    arcs = case.get("arcs", True)
    return dict(kind="one", img=img, thr=case["thr"], record=_record(img.numel(), img.device),
                options=dict(is_dual=case["dual"], return_gradient=case.get("gradient", True), trace_valleys=arcs,
                             trace_ridges=arcs))


def _pack(complexes, record):
    """The lists of the complexes, whole, back to back in ``record`` (a
    program that analyses one field after the other keeps them in records of
    one size), and the length of each."""
    parts = [getattr(c, f).reshape(-1) for f in _LISTS for c in complexes]
    n = [t.numel() for t in parts]
    torch.cat([t.view(torch.int32) for t in parts], out=record[: sum(n)])
    return torch.tensor(n)


def run(state):
    if state["kind"] == "one":
        c = compute_dmsc(state["img"], state["thr"], **state["options"])
        out = {f: getattr(c, f) for f in _MAPS}
        out["lengths"] = _pack([c], state["record"])
        out["lists"] = state["record"]
        return out
    if state["kind"] == "batch":
        complexes = compute_dmsc_batched(state["images"], state["thr"], is_dual=state["dual"])
        out = {f: torch.cat([getattr(c, f).reshape(-1) for c in complexes]) for f in _MAPS}
        out["lengths"] = _pack(complexes, state["record"])
        out["lists"] = state["record"]
        return out
    x = state["x"]
    x.grad = None
    loss = topological_loss(x, is_dual=state["dual"])
    loss.backward()
    return {"loss": loss.detach(), "grad": x.grad}


def _complex_bytes(H, W, gradient=True):
    """Input once, and the outputs whose size does not depend on the values
    (gradient and the two label maps); the lists come on top."""
    return 4 * H * W + (16 * (H + 1) * (W + 1) if gradient else 0) + 4 * (H + 1) * (W + 1) + 4 * H * W


def work(case):
    if case["kind"] == "one":
        n = _complex_bytes(case["H"], case["W"], case.get("gradient", True))
    elif case["kind"] == "batch":  # mean side of a log-uniform size
        side = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        n = case["n"] * _complex_bytes(side, side)
    else:  # field in, gradient out
        n = 8 * case["B"] * case["H"] * case["W"]
    return {"bytes": n, "flops": 0}


def _merges(order, a, b, birth):
    """Kruskal over the edges ``order`` with the elder rule: (edge, oldest
    node of the dying component) of every merge. The smaller a node's
    ``birth``, the older it is."""
    link = list(range(len(birth)))
    edges, dead = [], []
    for e in order:
        r, s = a[e], b[e]
        while link[r] != r:
            link[r] = link[link[r]]
            r = link[r]
        while link[s] != s:
            link[s] = link[link[s]]
            s = link[s]
        if r == s:
            continue
        if birth[r] < birth[s]:
            r, s = s, r
        link[r] = s  # r is the younger one
        edges.append(e)
        dead.append(r)
    return np.array(edges, dtype=np.int64), np.array(dead, dtype=np.int64)


def _pixel_pairs(z, dual):
    """The (plus, minus) pixels of every persistence pair of a tie-free field,
    pairs of one pixel with itself included: merges of the components of the
    sublevel sets over the pixel grid, whose outside is older than every
    pixel, and of the superlevel sets over the grid of pixel corners."""
    z = -z if dual else z
    H, W = z.shape
    at = np.argsort(z.reshape(-1)[:: -1 if dual else 1], kind="stable")  # pixel of each rank
    at = H * W - 1 - at if dual else at  # ties by pixel id, in the dual the other way round
    rank = np.empty(H * W, dtype=np.int64)
    rank[at] = np.arange(H * W)
    r = np.full((H + 2, W + 2), -1, dtype=np.int64)
    r[1:-1, 1:-1] = rank.reshape(H, W)
    px = np.full((H + 2, W + 2), H * W, dtype=np.int64)  # H * W: the outside
    px[1:-1, 1:-1] = np.arange(H * W).reshape(H, W)
    # H-edges lie between the pixels (y, x-1) and (y, x) and the corners (y, x)
    # and (y+1, x); V-edges between (y-1, x) and (y, x) and the corners (y, x)
    # and (y, x+1). An edge's value is that of its higher pixel.
    top = np.concatenate([np.maximum(r[1:-1, :-1], r[1:-1, 1:]).ravel(), np.maximum(r[:-1, 1:-1], r[1:, 1:-1]).ravel()])
    a = np.concatenate([px[1:-1, :-1].ravel(), px[:-1, 1:-1].ravel()])
    b = np.concatenate([px[1:-1, 1:].ravel(), px[1:, 1:-1].ravel()])
    e, d = _merges(np.argsort(top, kind="stable").tolist(), a.tolist(), b.tolist(), rank.tolist() + [-1])
    low = (at[top[e]], d)
    corner = np.maximum(np.maximum(r[:-1, :-1], r[:-1, 1:]), np.maximum(r[1:, :-1], r[1:, 1:])).reshape(-1)
    cid = np.arange((H + 1) * (W + 1)).reshape(H + 1, W + 1)
    a = np.concatenate([cid[:-1].ravel(), cid[:, :-1].ravel()])
    b = np.concatenate([cid[1:].ravel(), cid[:, 1:].ravel()])
    e, d = _merges(np.argsort(-top, kind="stable").tolist(), a.tolist(), b.tolist(), (-corner).tolist())
    high = (at[corner[d]], at[top[e]])
    return [(m, p) if dual else (p, m) for p, m in (low, high)]


def exact(case, seed):
    if case["kind"] != "train":
        return None  # list orders and labels are whole numbers; a persistence is one difference of two inputs
    x = _train_batch(case, seed).cpu().double().numpy()
    grad = np.zeros_like(x)
    loss = 0.0
    for k in range(case["B"]):
        z, g = x[k].reshape(-1), grad[k].reshape(-1)
        for plus, minus in _pixel_pairs(x[k], case["dual"]):
            p = z[plus] - z[minus]
            keep = p < 0.1
            p = np.where(keep, p, 0.0)
            loss += float((p * p).sum())
            np.add.at(g, plus, 2 * p)
            np.add.at(g, minus, -2 * p)
    return {"loss": torch.tensor(loss, dtype=torch.float64), "grad": torch.from_numpy(grad)}
