"""Performance cases: what a user of the package has it do, through its public entry points.

Twelve listed cases and a generator of more of the same ranges.  A case is a dict of plain
values; ``kind`` names the family (one prepare / run / work / exact each):

  grey     flat grey morphology of (B, 1, *spatial) float32 batches, one call
  train    differentiable grey morphology inside a training step: forward and backward
  binary   binary morphology of bool masks, one call
  edt      exact Euclidean distance transform of bool masks
  ragged   a pipeline over images of uneven sizes packed in one RaggedBatch
  ot       SinkhornSolver as a loss on histograms sharing one cost: distances and gradients
  clouds   PointCloudSinkhorn as a loss on ragged point-cloud pairs: costs and gradients
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

import torchmorph_gb300 as tm
from torchmorph_gb300 import ragged

DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one operator on a small batch of images, as an augmentation or a loss term calls
        # it in every step: launch and host latency
        dict(name="grey_3x3_small", kind="grey", op="dilation", size=3, mode="reflect", shape="8,256,256"),
        # the same operator on whole slides or frames: memory bandwidth
        dict(name="grey_3x3_large", kind="grey", op="dilation", size=3, mode="reflect", shape="8,4096,4096"),
        # background subtraction of photographs or micrographs, rows of odd length
        dict(name="tophat_15_odd", kind="grey", op="white_tophat", size=15, mode="reflect", shape="6,1023,1535"),
        # a morphological layer of a network: forward and backward of one training step
        dict(name="grey_5x5_train", kind="train", op="dilation", size=5, mode="reflect", shape="16,512,512"),
        # clean-up of 3-D segmentation masks (removes specks thinner than the default cross)
        dict(name="binary_open_3d", kind="binary", op="opening", element="cross", shape="4,96,160,200", fill=0.5),
        # dense seeds: 10 % background voxels everywhere, with the feature indices
        dict(name="edt_dense_3d", kind="edt", shape="4,128,128,128", mask="noise", fill=0.9, sampling="",
             indices=True),
        # distance maps of organ-like masks on a scanner's grid (slices thicker than pixels)
        dict(name="edt_scan_3d", kind="edt", shape="2,88,180,214", mask="blobs", fill=0.5, sampling="2.5,1,1",
             indices=False),
        # distance maps of 2-D instance masks (boundary weights, watershed seeds)
        dict(name="edt_masks_2d", kind="edt", shape="8,1000,1333", mask="blobs", fill=0.5, sampling="",
             indices=False),
        # images of uneven sizes through a fixed pipeline: two erosions and a binary opening
        dict(name="ragged_256", kind="ragged", count=256, low=32, high=1024, sizes=0, small=5, big=15),
        # OT loss between small grey images on one grid cost, gradients w.r.t. both sides
        dict(name="ot_images_16", kind="ot", n=16, grid=28, points=0, epsilon=0.05, iterations=100, log=False),
        # many histograms over one large shared support
        dict(name="ot_shared_256x8192", kind="ot", n=256, grid=0, points=8192, epsilon=0.05, iterations=20,
             log=False),
        # OT loss between hundreds of ragged point clouds, gradient w.r.t. the source points
        dict(name="clouds_512", kind="clouds", count=512, low=64, high=2048, sizes=0, iterations=100),
    ]


def _log_int(rng: random.Random, lo: float, hi: float) -> int:
    return max(int(lo), min(int(hi), int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _batch_of(rng, dims, voxels):
    """A (B, *dims) shape text of about `voxels` voxels, at least one item."""
    n = 1
    for d in dims:
        n *= d
    return ",".join(str(v) for v in (max(1, min(64, voxels // n)), *dims))


def draw(rng: random.Random):
    kind = rng.choice(["grey", "grey", "train", "binary", "edt", "edt", "edt", "ragged", "ot", "clouds"])
    if kind == "grey":
        op = rng.choice(["dilation", "erosion", "opening", "closing", "gradient", "white_tophat", "black_tophat"])
        mode = rng.choice(["reflect", "reflect", "nearest", "mirror", "constant"])
        if rng.random() < 0.25:
            dims, size = [_log_int(rng, 24, 200) for _ in range(3)], rng.choice([3, 3, 5])
            voxels = _log_int(rng, 2e5, 2e7)
        else:
            dims, size = [_log_int(rng, 48, 4096) for _ in range(2)], rng.choice([3, 3, 5, 7, 9, 15, 21])
            voxels = _log_int(rng, 2e5, 1e8)
            if op == "gradient" and size > 7:
                size = 7
        return dict(kind=kind, op=op, size=size, mode=mode, shape=_batch_of(rng, dims, voxels))
    if kind == "train":
        dims = [_log_int(rng, 48, 2048) for _ in range(2)]
        return dict(kind=kind, op=rng.choice(["dilation", "erosion"]), size=rng.choice([3, 5, 7]),
                    mode=rng.choice(["reflect", "nearest", "constant"]),
                    shape=_batch_of(rng, dims, _log_int(rng, 2e5, 3e7)))
    if kind == "binary":
        if rng.random() < 0.6:
            dims, voxels = [_log_int(rng, 24, 256) for _ in range(3)], _log_int(rng, 2e5, 5e7)
        else:
            dims, voxels = [_log_int(rng, 48, 4096) for _ in range(2)], _log_int(rng, 2e5, 1e8)
        return dict(kind=kind, op=rng.choice(["erosion", "dilation", "opening", "closing"]),
                    element=rng.choice(["cross", "cross", "box"]), shape=_batch_of(rng, dims, voxels),
                    fill=round(rng.uniform(0.2, 0.8), 3))
    if kind == "edt":
        if rng.random() < 0.6:
            dims, voxels = [_log_int(rng, 24, 256) for _ in range(3)], _log_int(rng, 2e5, 1.5e7)
            sampling = rng.choice(["", "", "2.5,1,1", "1,1,2.5"])
        else:
            dims, voxels = [_log_int(rng, 64, 2048) for _ in range(2)], _log_int(rng, 2e5, 2e7)
            sampling = ""
        mask = rng.choice(["blobs", "blobs", "noise"])
        fill = round(rng.uniform(0.2, 0.8) if mask == "blobs" else rng.choice([0.5, 0.9, 0.99]), 3)
        return dict(kind=kind, shape=_batch_of(rng, dims, voxels), mask=mask, fill=fill, sampling=sampling,
                    indices=sampling == "" and rng.random() < 0.5)
    if kind == "ragged":
        return dict(kind=kind, count=_log_int(rng, 16, 256), low=32, high=_log_int(rng, 256, 1024),
                    sizes=rng.randrange(1, 1 << 20), small=rng.choice([3, 5]), big=rng.choice([9, 15]))
    if kind == "ot":
        if rng.random() < 0.6:
            return dict(kind=kind, n=_log_int(rng, 1, 48), grid=rng.randint(8, 40), points=0,
                        epsilon=rng.choice([0.05, 0.1]), iterations=rng.choice([50, 100]),
                        log=rng.random() < 0.3)
        return dict(kind=kind, n=_log_int(rng, 32, 256), grid=0, points=_log_int(rng, 512, 8192), epsilon=0.05,
                    iterations=20, log=False)
    return dict(kind=kind, count=_log_int(rng, 16, 512), low=64, high=_log_int(rng, 256, 2048),
                sizes=rng.randrange(1, 1 << 20), iterations=100)


# ------------------------------------------------------------------- inputs
def _dims(case):
    return [int(v) for v in case["shape"].split(",")]


def _numel(case):
    return math.prod(_dims(case))


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _blobs(dims, fill, gen):
    """(B, 1, *spatial) bool masks with the extent and smoothness of segmented objects: a coarse
    random field (a node every 24 voxels) interpolated to the grid; `fill` of the voxels are foreground."""
    b, sp = dims[0], dims[1:]
    coarse = [max(2, -(-s // 24) + 1) for s in sp]
    field = torch.randn((b, 1, *coarse), generator=gen, device=DEV)
    field = torch.nn.functional.interpolate(field, size=sp, mode="trilinear" if len(sp) == 3 else "bilinear",
                                            align_corners=True)
    flat = field.reshape(b, -1)
    pick = torch.linspace(0, flat.shape[1] - 1, min(flat.shape[1], 100001), device=DEV).long()
    level = torch.quantile(flat[:, pick], 1.0 - fill, dim=1)
    return field > level.view(b, 1, *([1] * len(sp)))


def _ragged_shapes(case):
    r = np.random.default_rng(case["sizes"])
    return [tuple(int(v) for v in r.integers(case["low"], case["high"] + 1, 2)) for _ in range(case["count"])]


def _cloud_sizes(case):
    r = np.random.default_rng(case["sizes"])
    k = np.rint(np.exp(r.uniform(math.log(case["low"]), math.log(case["high"]), (2, case["count"]))))
    return [int(v) for v in k[0]], [int(v) for v in k[1]]


def _cloud_points(sizes, means, gen):
    """Points of a 4-component Gaussian mixture in R^3 per problem, packed (sum k, 3)."""
    owner = torch.repeat_interleave(torch.arange(len(sizes), device=DEV), torch.tensor(sizes, device=DEV))
    part = torch.randint(0, 4, (owner.numel(),), generator=gen, device=DEV)
    return means[owner, part] + 0.2 * torch.randn((owner.numel(), 3), generator=gen, device=DEV)


def _ot_inputs(case, seed):
    gen = _gen(seed)
    n = case["n"]
    if case["grid"]:
        s = case["grid"]
        cost = tm.build_cost_matrix((s, s), device=DEV)
        # images: three soft spots on a faint background
        at = torch.arange(s, device=DEV, dtype=torch.float32) / s
        img = []
        for _ in range(2):
            c = torch.rand((n, 3, 2), generator=gen, device=DEV)
            gy = torch.exp(-((at - c[..., :1]) ** 2) / 0.02)
            gx = torch.exp(-((at - c[..., 1:]) ** 2) / 0.02)
            img.append(torch.einsum("nky,nkx->nyx", gy, gx).reshape(n, s * s) + 1e-3)
        a, b = img
    else:
        d = case["points"]
        x = torch.rand((d, 3), generator=gen, device=DEV, dtype=torch.float64)
        y = torch.rand((d, 3), generator=gen, device=DEV, dtype=torch.float64)
        cost = ((x * x).sum(1)[:, None] + (y * y).sum(1)[None] - 2.0 * (x @ y.T)).clamp_(min=0)
        # Dirichlet(1) histograms: normalised exponential variables
        a, b = (-torch.log1p(-torch.rand((n, d), generator=gen, device=DEV)) + 1e-7 for _ in range(2))
    cost = (cost / cost.max()).float().contiguous()
    return a, b, cost


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("grey", "train"):
        b, *sp = _dims(case)
        gen = _gen(seed)
        x = torch.rand((b, 1, *sp), generator=gen, device=DEV)
        if kind == "grey":
            return dict(case, x=x)
        return dict(case, x=x.requires_grad_(), grad=torch.randn((b, 1, *sp), generator=gen, device=DEV))
    if kind == "binary":
        dims = _dims(case)
        gen = _gen(seed)
        x = _blobs(dims, case["fill"], gen)
        # a few per cent of salt and pepper, what a clean-up is there to remove
        x = x ^ (torch.rand(x.shape, generator=gen, device=DEV) < 0.02)
        element = None if case["element"] == "cross" else torch.ones((3,) * (len(dims) - 1), dtype=torch.bool)
        return dict(case, x=x, structure=element)
    if kind == "edt":
        b, *sp = _dims(case)
        gen = _gen(seed)
        if case["mask"] == "noise":
            x = torch.rand((b, 1, *sp), generator=gen, device=DEV) < case["fill"]
        else:
            x = _blobs([b, *sp], case["fill"], gen)
        sampling = [float(v) for v in case["sampling"].split(",")] if case["sampling"] else None
        return dict(case, x=x, spacing=sampling)
    if kind == "ragged":
        shapes = _ragged_shapes(case)
        data = torch.rand(sum(h * w for h, w in shapes), generator=_gen(seed), device=DEV)
        batch = tm.RaggedBatch(data, shapes)
        batch.plan  # noqa: B018  (laid out once per batch of shapes, as a program keeps it)
        return dict(case, batch=batch, mask=batch.map(lambda v: v > 0.5))
    if kind == "ot":
        a, b, cost = _ot_inputs(case, seed)
        solver = tm.SinkhornSolver(epsilon=case["epsilon"], max_iter=case["iterations"], log_space=case["log"],
                                   reuse_solves=False)
        return dict(case, a=a.requires_grad_(), b=b.requires_grad_(), cost=cost, solver=solver)
    nx, ny = _cloud_sizes(case)
    gen = _gen(seed)
    means = torch.rand((case["count"], 4, 3), generator=gen, device=DEV) * 2 - 1
    x, y = _cloud_points(nx, means, gen), _cloud_points(ny, means, gen)
    solver = tm.PointCloudSinkhorn(epsilon=0.05, max_iter=case["iterations"], threshold=0.0)
    return dict(case, x=x.requires_grad_(), y=y, nx=nx, ny=ny, solver=solver)


# ---------------------------------------------------------------------- runs
_GREY = {
    "dilation": tm.grey_dilation,
    "erosion": tm.grey_erosion,
    "opening": tm.grey_opening,
    "closing": tm.grey_closing,
    "gradient": tm.morphological_gradient,
    "white_tophat": tm.white_tophat,
    "black_tophat": tm.black_tophat,
}
_BINARY = {
    "dilation": tm.binary_dilation,
    "erosion": tm.binary_erosion,
    "opening": tm.binary_opening,
    "closing": tm.binary_closing,
}


def run(state):
    kind = state["kind"]
    if kind == "grey":
        return _GREY[state["op"]](state["x"], size=state["size"], mode=state["mode"])
    if kind == "train":
        out = _GREY[state["op"]](state["x"], size=state["size"], mode=state["mode"], differentiable=True)
        return out, torch.autograd.grad(out, state["x"], state["grad"])[0]
    if kind == "binary":
        return _BINARY[state["op"]](state["x"], structure=state["structure"])
    if kind == "edt":
        return tm.euclidean_distance_transform(state["x"], sampling=state["spacing"],
                                               return_indices=state["indices"])
    if kind == "ragged":
        batch = state["batch"]
        return (ragged.grey_erosion(batch, size=state["small"]).data,
                ragged.grey_erosion(batch, size=state["big"]).data,
                ragged.binary_opening(state["mask"]).data)
    if kind == "ot":
        dist = state["solver"](state["a"], state["b"], state["cost"])
        return (dist, *torch.autograd.grad(dist.sum(), (state["a"], state["b"])))
    cost = state["solver"](state["x"], state["y"], state["nx"], state["ny"])
    return cost, torch.autograd.grad(cost.sum(), state["x"])[0]


# --------------------------------------------------------------------- work
def work(case):
    """Bytes: each input read once, each output written once.  Operations: the products of the
    Sinkhorn iterations (two per iteration), or the pair evaluations of the point clouds (an
    inner product, an exponential and a sum: about 10 operations a pair)."""
    kind = case["kind"]
    if kind == "grey":
        return dict(bytes=8 * _numel(case), flops=0)
    if kind == "train":  # forward: in, out; backward: gradient of the output, of the input
        return dict(bytes=16 * _numel(case), flops=0)
    if kind == "binary":
        return dict(bytes=2 * _numel(case), flops=0)
    if kind == "edt":
        nd = len(_dims(case)) - 1
        return dict(bytes=(5 + (4 * nd if case["indices"] else 0)) * _numel(case), flops=0)
    if kind == "ragged":
        return dict(bytes=18 * sum(h * w for h, w in _ragged_shapes(case)), flops=0)
    if kind == "ot":
        d = case["grid"] ** 2 or case["points"]
        n = case["n"]
        return dict(bytes=4 * d * d + 16 * n * d + 4 * n, flops=2 * (2 * case["iterations"] + 1) * n * d * d)
    nx, ny = _cloud_sizes(case)
    pairs = sum(a * b for a, b in zip(nx, ny))
    return dict(bytes=4 * (6 * sum(nx) + 3 * sum(ny)), flops=10 * pairs * (2 * case["iterations"] + 1))


# -------------------------------------------------- the same in 64 bits, torch
def _source(n, offset, mode):
    """Index read at i + offset for i = 0 .. n-1 under a border mode (-1: the constant)."""
    i = torch.arange(n, device=DEV) + offset
    if mode == "constant":
        return torch.where((i < 0) | (i >= n), torch.full_like(i, -1), i)
    if mode == "nearest":
        return i.clamp(0, n - 1)
    if mode == "mirror":
        p = max(1, 2 * n - 2)
        i = i % p
        return torch.minimum(i, p - i) if n > 1 else torch.zeros_like(i)
    i = i % (2 * n)  # reflect
    return torch.minimum(i, 2 * n - 1 - i)


def _box64(x, size, mode, dilation):
    """Flat box extremum of the trailing dims of x in float64, axis by axis (border constant 0)."""
    pick = torch.maximum if dilation else torch.minimum
    for axis in range(2, x.dim()):
        n, best = x.shape[axis], None
        for k in range(size):
            off = k - size // 2
            src = _source(n, -off if dilation else off, mode)
            v = x.index_select(axis, src.clamp(min=0))
            if mode == "constant":
                out = (src < 0).view([-1 if a == axis else 1 for a in range(x.dim())])
                v = v.masked_fill(out, 0.0)
            best = v if best is None else pick(best, v)
        x = best
    return x


def _grey64(x, op, size, mode):
    ero = lambda v: _box64(v, size, mode, False)  # noqa: E731
    dil = lambda v: _box64(v, size, mode, True)  # noqa: E731
    return {
        "dilation": dil,
        "erosion": ero,
        "opening": lambda v: dil(ero(v)),
        "closing": lambda v: ero(dil(v)),
        "gradient": lambda v: dil(v) - ero(v),
        "white_tophat": lambda v: v - dil(ero(v)),
        "black_tophat": lambda v: ero(dil(v)) - v,
    }[op](x)


def _train64(x, grad, op, size, mode):
    """Extremum and the gradient routed to the first tap (raster order) that attains it."""
    h, w = x.shape[2:]
    best = arg = None
    for ky in range(size):
        for kx in range(size):
            s = -1 if op == "dilation" else 1
            sy = _source(h, s * (ky - size // 2), mode)
            sx = _source(w, s * (kx - size // 2), mode)
            v = x.index_select(2, sy.clamp(min=0)).index_select(3, sx.clamp(min=0))
            at = (sy[:, None] * w + sx[None]).expand_as(v)
            if mode == "constant":
                out = (sy[:, None] < 0) | (sx[None] < 0)
                v, at = v.masked_fill(out, 0.0), at.masked_fill(out, h * w)
            if best is None:
                best, arg = v, at
            else:
                new = v > best if op == "dilation" else v < best
                best, arg = torch.where(new, v, best), torch.where(new, at, arg)
    b = x.shape[0]
    gin = torch.zeros((b, h * w + 1), dtype=torch.float64, device=DEV)
    gin.scatter_add_(1, arg.reshape(b, -1), grad.double().reshape(b, -1))
    return best, gin[:, :-1].reshape(x.shape)


def _edt64(x, spacing):
    """Distances by min-plus products along each axis in float64."""
    d2 = torch.where(x, torch.full(x.shape, 1e12, dtype=torch.float64, device=DEV),
                     torch.zeros(x.shape, dtype=torch.float64, device=DEV))
    for axis in range(2, x.dim()):
        n = x.shape[axis]
        s = 1.0 if spacing is None else spacing[axis - 2]
        q = torch.arange(n, device=DEV, dtype=torch.float64) * s
        pair = (q[:, None] - q[None]) ** 2
        lines = d2.movedim(axis, -1).contiguous()
        flat = lines.view(-1, n)
        step = max(1, (1 << 27) // (n * n))
        for i in range(0, flat.shape[0], step):
            flat[i:i + step] = (flat[i:i + step, None, :] + pair).amin(-1)
        d2 = lines.movedim(-1, axis)
    return d2.sqrt().contiguous()


def _ot64(case, seed):
    a, b, cost = _ot_inputs(case, seed)
    a, b, cost = a.double(), b.double(), cost.double()
    eps = case["epsilon"]
    sa, sb = a.sum(-1, keepdim=True), b.sum(-1, keepdim=True)
    a, b = a / sa, b / sb
    kern = torch.exp(-cost / eps)
    tiny = 0.0 if case["log"] else 1e-12
    u, v = torch.ones_like(a), torch.ones_like(b)
    for _ in range(case["iterations"]):
        u = a / (v @ kern.T + tiny)
        v = b / (u @ kern + tiny)
    dist = (u * (v @ (kern * cost).T)).sum(-1)
    out = [dist]
    for w, h, total in ((u, a, sa), (v, b, sb)):
        pot = eps * w.log()
        pot = pot - pot.mean(-1, keepdim=True)
        out.append((pot - (pot * h).sum(-1, keepdim=True)) / total)  # through the normalisation of the row
    return tuple(out)


def _clouds64(state):
    eps = 0.05
    x, y = state["x"].detach().double(), state["y"].double()
    costs, grads = [], []
    ox = oy = 0
    for n, m in zip(state["nx"], state["ny"]):
        xp, yp = x[ox:ox + n], y[oy:oy + m]
        ox, oy = ox + n, oy + m
        # log-domain iterations with the marginal weights 1/n, 1/m, from log u = log v = 0
        k = -((xp[:, None] - yp[None]) ** 2).sum(-1) / eps
        la, lb = -math.log(n), -math.log(m)
        g = torch.full((m,), -lb, dtype=torch.float64, device=DEV)
        for _ in range(state["iterations"]):
            f = -torch.logsumexp(k + (g + lb), 1)
            g = -torch.logsumexp(k + (f + la)[:, None], 0)
        costs.append(eps * (f.mean() + g.mean()))
        p = torch.exp(k + (f + la)[:, None] + (g + lb))
        grads.append(2 * (p.sum(1, keepdim=True) * xp - p @ yp))
    return torch.stack(costs), torch.cat(grads)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ot":
        return _ot64(case, seed)
    if kind == "binary":
        return None
    s = prepare(case, seed)
    if kind == "grey":
        return _grey64(s["x"].double(), case["op"], case["size"], case["mode"])
    if kind == "train":
        return _train64(s["x"].detach().double(), s["grad"], case["op"], case["size"], case["mode"])
    if kind == "edt":
        d = _edt64(s["x"], s["spacing"])
        return (d, None) if case["indices"] else d
    if kind == "ragged":
        small, big = [], []
        for im in s["batch"].images():
            v = im.double()[None, None]
            small.append(_box64(v, case["small"], "reflect", False).reshape(-1))
            big.append(_box64(v, case["big"], "reflect", False).reshape(-1))
        return torch.cat(small), torch.cat(big), None
    return _clouds64(s)
