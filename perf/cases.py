"""The work that users of this package have it do, as timed cases.

Each case is a dict of plain values.  `kind` names the path:

  mttkrp    MTTKRP of every mode of a tensor resident on the GPU (one sweep of
            an ALS or gradient program), COO or HiCOO, FP32 or BF16 factors
  first     a new tensor: device COO arrays -> handle -> HiCOO conversion ->
            the first MTTKRP of every mode (schedules are built on the way)
  als       CPD-ALS iterations of one tensor
  gradient  gradient CP through autograd: loss and the gradient of every factor
  ttm       tensor times matrix along every mode
  batch     CPD-ALS of many small uneven tensors at once
  host      the drop-in call on host arrays (copies in, schedule, copy back)

Coordinates are unique and seeded, uniform per mode or Zipf(1.1) over a
permutation of each mode; values and factors follow the benchmark workloads.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from hiparti_b200.api import COOTensor, DeviceTensor
from hiparti_b200.autograd import cp_loss
from hiparti_b200.batched import Batch
from hiparti_b200.synth import coords_torch


def listed():
    return [
        # a small tensor inside a larger program: calls of a few microseconds
        dict(name="mttkrp_coo_small", kind="mttkrp", fmt="coo", d0=120, d1=90, d2=70, nnz=5_000, rank=10,
             dtype="fp32", zipf=False),
        # the plain COO workload: 1000^3, a million uniform nonzeros, R = 16
        dict(name="mttkrp_coo_1m", kind="mttkrp", fmt="coo", d0=1000, d1=1000, d2=1000, nnz=1_000_000, rank=16,
             dtype="fp32", zipf=False),
        # a wide factorisation of a power-law 4-D tensor with ragged sizes
        dict(name="mttkrp_coo_4d_wide", kind="mttkrp", fmt="coo", d0=30_011, d1=12_007, d2=5_003, d3=97,
             nnz=3_000_001, rank=150, dtype="fp32", zipf=True),
        # the headline workload: 50M Zipf nonzeros in HiCOO, R = 32
        dict(name="mttkrp_hicoo_50m", kind="mttkrp", fmt="hicoo", d0=200_000, d1=150_000, d2=20_000,
             nnz=50_000_000, rank=32, dtype="fp32", zipf=True),
        # the mixed-precision sweep: 4-D, BF16 factors, a rank that fills no power of two
        dict(name="mttkrp_hicoo_4d_bf16", kind="mttkrp", fmt="hicoo", d0=20_000, d1=20_000, d2=20_000, d3=500,
             nnz=10_000_000, rank=40, dtype="bf16", zipf=False),
        # a tensor seen for the first time: conversion, schedules, first results
        dict(name="first_use_10m", kind="first", d0=200_000, d1=150_000, d2=20_000, nnz=10_000_000, rank=32,
             zipf=True),
        # ALS of a 4-D tensor in HiCOO at the usual rank
        dict(name="als_hicoo_4d", kind="als", fmt="hicoo", d0=20_000, d1=20_000, d2=20_000, d3=500,
             nnz=10_000_000, rank=32, iters=3, precision="fp32", zipf=False),
        # ALS at a large rank, where the dense steps weigh as much as the MTTKRP
        dict(name="als_coo_rank64", kind="als", fmt="coo", d0=30_000, d1=20_000, d2=3_000, nnz=2_000_000, rank=64,
             iters=3, precision="fp32", zipf=False),
        # gradient CP: 100,000^3, 20M nonzeros, R = 64
        dict(name="gradient_20m", kind="gradient", d0=100_000, d1=100_000, d2=100_000, nnz=20_000_000, rank=64),
        # TTM of a power-law tensor along every mode (a Tucker sweep)
        dict(name="ttm_5m", kind="ttm", d0=200_000, d1=150_000, d2=20_000, nnz=5_000_000, rank=16, zipf=True),
        # many small tensors of uneven size and rank
        dict(name="batch_128", kind="batch", tensors=128, nnz_max=500_000, iters=10, precision="fp32"),
        # the C library's call with host arrays, as a program linked against it makes it
        dict(name="host_hicoo_1m", kind="host", d0=20_000, d1=15_000, d2=2_000, nnz=1_000_000, rank=16, zipf=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, n, lo, hi):
    return {f"d{m}": _log(rng, lo, hi) for m in range(n)}


def draw(rng):
    kind = rng.choice(["mttkrp"] * 5 + ["first", "als", "als", "gradient", "ttm", "batch", "host"])
    if kind == "mttkrp":
        fmt = rng.choice(["coo", "hicoo"])
        n = rng.choice([3, 3, 4, 4, 5] if fmt == "coo" else [3, 4])
        zipf = rng.random() < 0.5
        rank = _log(rng, 4, 200)
        most = 3_000_000 if rank > 128 or n > 4 else 20_000_000
        nnz = _log(rng, 5_000, max(20_000, min(most, 400_000_000 // rank)))
        dims = _dims(rng, n, 2_000, 200_000) if nnz > 200_000 else _dims(rng, n, 300, 30_000)
        return dict(kind=kind, fmt=fmt, **dims, nnz=nnz, rank=rank, dtype=rng.choice(["fp32", "bf16"]), zipf=zipf)
    if kind == "first":
        n = rng.choice([3, 4])
        return dict(kind=kind, **_dims(rng, n, 2_000, 200_000), nnz=_log(rng, 100_000, 10_000_000),
                    rank=_log(rng, 8, 64), zipf=rng.random() < 0.5)
    if kind == "als":
        n = rng.choice([3, 4])
        return dict(kind=kind, fmt=rng.choice(["coo", "hicoo"]), **_dims(rng, n, 500, 20_000),
                    nnz=_log(rng, 200_000, 4_000_000), rank=_log(rng, 8, 128), iters=3,
                    precision=rng.choice(["fp32", "fp32", "bf16"]), zipf=False)
    if kind == "gradient":
        return dict(kind=kind, **_dims(rng, 3, 1_000, 100_000), nnz=_log(rng, 100_000, 10_000_000),
                    rank=_log(rng, 8, 100))
    if kind == "ttm":
        n = rng.choice([3, 4])
        return dict(kind=kind, **_dims(rng, n, 2_000, 200_000), nnz=_log(rng, 50_000, 4_000_000),
                    rank=_log(rng, 2, 32), zipf=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, tensors=rng.randint(8, 128), nnz_max=_log(rng, 20_000, 500_000), iters=10,
                    precision=rng.choice(["fp32", "bf16"]))
    return dict(kind=kind, **_dims(rng, rng.choice([3, 4]), 2_000, 20_000), nnz=_log(rng, 20_000, 2_000_000),
                rank=_log(rng, 8, 64), zipf=rng.random() < 0.5)


def _case_dims(case):
    return [case[f"d{m}"] for m in range(8) if f"d{m}" in case]


def _stride(rank):
    return (rank + 7) // 8 * 8


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _coords(case, seed):
    dims, zipf = _case_dims(case), 1.1 if case.get("zipf") else None
    if case["kind"] != "ttm":
        return coords_torch(dims, case["nnz"], seed, zipf_s=zipf)
    # one pattern, its modes rotated by the seed: as many fibers for every seed
    rng = np.random.default_rng(seed)
    inds = coords_torch(dims, case["nnz"], case["nnz"], zipf_s=zipf)
    return [((i.long() + int(rng.integers(d))) % d).to(torch.int32) for i, d in zip(inds, dims)]


def _factors(dims, rank, g, normal=0.0):
    """Row-major factors, rows padded to a multiple of 8 with zeros; U(0,1), or
    N(0, normal^2)."""
    out = []
    for d in dims:
        a = torch.zeros((d, _stride(rank)), device="cuda")
        a[:, :rank] = (normal * torch.randn((d, rank), generator=g, device="cuda") if normal
                       else torch.rand((d, rank), generator=g, device="cuda"))
        out.append(a)
    return out


def _planted(dims, inds, rank, noise, g):
    """Values of a positive Kruskal model of the given rank at the coordinates,
    scaled to a mean of 1, plus noise."""
    n = inds[0].numel()
    facs = [torch.rand((d, rank), generator=g, device="cuda") + 0.1 for d in dims]
    w = torch.rand(rank, generator=g, device="cuda") + 0.5
    vals = torch.empty(n, device="cuda")
    for z in range(0, n, 1 << 22):
        p = w.expand(min(1 << 22, n - z), rank)
        for a, ix in zip(facs, inds):
            p = p * a[ix[z:z + (1 << 22)].long()]
        vals[z:z + (1 << 22)] = p.sum(1)
    vals /= vals.mean()
    return vals + noise * torch.randn(n, generator=g, device="cuda")


def _batch_inputs(case, seed):
    """Tensors of a batch: mode sizes U{50..5000}, nonzeros log-uniform, ranks
    from {8, 16, 32}.  Sizes belong to the case, coordinates and values to the
    seed."""
    rng = np.random.default_rng(case["tensors"])
    tensors, ranks = [], []
    g = _gen(seed)
    steps = np.linspace(math.log(1_000), math.log(case["nnz_max"]), case["tensors"])
    for b in range(case["tensors"]):
        dims = [int(x) for x in rng.integers(50, 5001, 3)]
        nnz = min(int(math.exp(steps[b])), int(np.prod(dims, dtype=np.float64)) // 4)
        inds = coords_torch(dims, nnz, seed * 1000 + b)
        tensors.append((dims, inds, torch.rand(nnz, generator=g, device="cuda")))
        ranks.append((8, 16, 32)[b % 3])
    return tensors, ranks, g


def _batch_views(flat, tensors, ranks):
    views, at = [], 0
    for (dims, _, _), r in zip(tensors, ranks):
        fs = []
        for d in dims:
            n = d * _stride(r)
            fs.append(flat[at:at + n].view(d, _stride(r)))
            at += (n + 63) // 64 * 64
        views.append(fs)
    return views


def _inputs(case, seed):
    """The seeded inputs of a case, the same for prepare and exact."""
    kind, g = case["kind"], _gen(seed + 1)
    if kind == "batch":
        tensors, ranks, g = _batch_inputs(case, seed)
        size = sum((d * _stride(r) + 63) // 64 * 64 for (dims, _, _), r in zip(tensors, ranks) for d in dims)
        flat = torch.zeros(size, device="cuda")
        for fs, r in zip(_batch_views(flat, tensors, ranks), ranks):
            for f in fs:
                f[:, :r] = torch.rand((f.shape[0], r), generator=g, device="cuda")
        return dict(tensors=tensors, ranks=ranks, flat=flat)
    dims = _case_dims(case)
    inds = _coords(case, seed)
    s = dict(dims=dims, inds=inds)
    if kind == "als":
        s["vals"] = _planted(dims, inds, 10, 0.05, g)
    elif kind == "gradient":
        s["vals"] = _planted(dims, inds, 16, 0.05, g)
    else:
        s["vals"] = torch.rand(case["nnz"], generator=g, device="cuda")
    if kind == "ttm":
        s["mats"] = [torch.rand((d, case["rank"]), generator=g, device="cuda") for d in dims]
    else:
        s["mats"] = _factors(dims, case["rank"], g, normal=0.1 if kind == "gradient" else 0.0)
    if case.get("dtype") == "bf16":
        s["mats"] = [m.to(torch.bfloat16) for m in s["mats"]]
    return s


def prepare(case, seed):
    kind = case["kind"]
    s = _inputs(case, seed)
    s["case"] = case
    if kind == "batch":
        s["batch"] = Batch(s["tensors"], s["ranks"])
        s["work"] = torch.empty_like(s["flat"])
        s["views"] = _batch_views(s["work"], s["tensors"], s["ranks"])
        del s["tensors"]
        return s
    if kind == "first":
        return s
    if kind == "host":
        coo = COOTensor(s["dims"], [i.cpu().numpy().view(np.uint32) for i in s["inds"]], s["vals"].cpu().numpy())
        s["tensor"] = coo.to_hicoo()
        s["mats"] = [m.cpu().numpy() for m in s["mats"]]
        del s["inds"], s["vals"]
        return s
    dt = DeviceTensor.from_torch_coo(s["dims"], s["inds"], s["vals"])
    if case.get("fmt") == "hicoo":
        dt = dt.to_hicoo()
    if kind == "ttm":
        for m, u in enumerate(s["mats"]):
            dt.ttm(u, m)
    elif len(s["dims"]) <= 4:
        dt.prepare()
    if kind == "als":
        s["work"] = [torch.empty_like(m) for m in s["mats"]]
    if kind == "gradient":
        s["mats"] = [m.requires_grad_(True) for m in s["mats"]]
    else:
        del s["vals"]
    del s["inds"]
    s["tensor"] = dt
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "mttkrp":
        return [s["tensor"].mttkrp(s["mats"], m, rank=case["rank"]) for m in range(len(s["dims"]))]
    if kind == "first":
        h = DeviceTensor.from_torch_coo(s["dims"], s["inds"], s["vals"]).to_hicoo()
        out = [h.mttkrp(s["mats"], m, rank=case["rank"]) for m in range(len(s["dims"]))]
        return out + [h.nb, h.max_nnzb]
    if kind == "als":
        for w, m in zip(s["work"], s["mats"]):
            w.copy_(m)
        lam, fits = s["tensor"].cpd_als(s["work"], case["iters"], precision=case["precision"], rank=case["rank"])
        return [*s["work"], lam, np.array(fits)]
    if kind == "gradient":
        for f in s["mats"]:
            f.grad = None
        loss = cp_loss(s["tensor"], s["vals"], s["mats"], rank=case["rank"])
        loss.backward()
        return [loss.detach(), *(f.grad for f in s["mats"])]
    if kind == "ttm":
        out = []
        for m, u in enumerate(s["mats"]):
            finds, y = s["tensor"].ttm(u, m)
            out += [f for f in finds if f is not None] + [y]
        return out
    if kind == "batch":
        s["work"].copy_(s["flat"])
        lams, fits, _ = s["batch"].cpd_als(s["views"], case["iters"], precision=case["precision"])
        return [s["work"], torch.cat(lams), fits]
    return [s["tensor"].mttkrp(s["mats"], case["rank"], m) for m in range(len(s["dims"]))]


def work(case):
    """Each input read once and each output written once: coordinates (4 bytes
    a mode in COO; a byte of element offset a mode in HiCOO, its block
    coordinates left out), values, factors, results.  The arithmetic is that
    of the products and sums."""
    kind = case["kind"]
    if kind == "batch":
        steps = [math.log(1_000) + (math.log(case["nnz_max"]) - math.log(1_000)) * b / max(1, case["tensors"] - 1)
                 for b in range(case["tensors"])]
        ranks = [(8, 16, 32)[b % 3] for b in range(case["tensors"])]
        per_b = sum(3 * math.exp(x) * 7 + 3 * 2525 * 3 * 4 * r for x, r in zip(steps, ranks))
        per_f = sum(3 * math.exp(x) * 3 * r + 3 * 2525 * 4 * r * r for x, r in zip(steps, ranks))
        return {"bytes": int(case["iters"] * per_b), "flops": int(case["iters"] * per_f)}
    dims, nnz, rank = _case_dims(case), case["nnz"], case["rank"]
    n = len(dims)
    fsize = 2 if case.get("dtype") == "bf16" else 4
    hicoo = case.get("fmt") == "hicoo" or kind == "host"
    nz = n + 4 if hicoo else 4 * n + 4
    sweep_b = n * nnz * nz + sum(4 * rank * d + fsize * rank * (sum(dims) - d) for d in dims)
    sweep_f = n * nnz * n * rank
    if kind == "first":
        return {"bytes": nnz * (4 * n + 4) + nnz * (n + 4) * (n + 1) + 4 * rank * sum(dims) * n, "flops": sweep_f}
    if kind == "als":
        dense_b = 8 * rank * sum(dims)
        dense_f = 4 * rank * rank * sum(dims)
        return {"bytes": case["iters"] * (sweep_b + dense_b), "flops": case["iters"] * (sweep_f + dense_f)}
    if kind == "gradient":
        return {"bytes": sweep_b + nnz * (4 * n + 8) + 4 * rank * sum(dims), "flops": sweep_f + n * nnz * rank}
    if kind == "ttm":
        return {"bytes": n * nnz * 8 + 4 * rank * sum(dims) + n * nnz * 4 * rank // 4, "flops": 2 * n * nnz * rank}
    return {"bytes": sweep_b, "flops": sweep_f}


def tolerance(case):
    """About four times the largest difference from FP64 (BF16 iterations: from
    a repeated run, whose FP32 atomics add in another order) over the listed
    and some hundred drawn cases."""
    kind = case["kind"]
    if kind == "mttkrp" and (case["rank"] > 128 or len(_case_dims(case)) > 4):
        # rows of a power-law mode are sums of up to a million FP32 atomics
        return {"rel": 1e-3 if case["zipf"] else 5e-5}
    if kind in ("mttkrp", "first", "host"):
        return {"rel": 4e-6}
    if kind == "als":
        return {"rel": 8e-5 if case["precision"] == "fp32" else 1e-2}
    if kind == "batch":
        return {"rel": 6e-5 if case["precision"] == "fp32" else 3e-2}
    return {"rel": 2e-6 if kind == "gradient" else 8e-6}


def _mttkrp64(dims, inds, vals, mats, mode, rank):
    out = torch.zeros((dims[mode], mats[0].shape[1]), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 28) // mats[0].shape[1])
    for z in range(0, vals.numel(), step):
        p = vals[z:z + step].double()[:, None].expand(-1, mats[0].shape[1])
        for k, a in enumerate(mats):
            if k != mode:
                p = p * a.double()[inds[k][z:z + step].long()]
        out.index_add_(0, inds[mode][z:z + step].long(), p)
    out[:, rank:] = 0
    return out


def _als64(dims, inds, vals, mats, rank, iters):
    """CPD-ALS in FP64: normal equations, 2-norm weights in the first iteration
    and max(column maximum, 1) after it, unit columns at the end."""
    a = [m.double()[:, :rank] for m in mats]
    gram = [x.T @ x for x in a]
    norm2 = vals.double().square().sum()
    fits = []
    for it in range(iters):
        for m in range(len(dims)):
            mt = _mttkrp64(dims, inds, vals, a, m, rank)
            v = torch.ones((rank, rank), dtype=torch.float64, device="cuda")
            for k in range(len(dims)):
                if k != m:
                    v = v * gram[k]
            x = torch.linalg.solve(v, mt.T).T
            lam = x.norm(dim=0) if it == 0 else x.amax(0).clamp(min=1.0)
            a[m] = x / lam
            gram[m] = a[m].T @ a[m]
        v = torch.ones_like(gram[0])
        for gm in gram:
            v = v * gm
        model = torch.abs(lam @ v @ lam)
        rest = norm2 + model - 2 * ((a[-1] * mt) @ lam).sum()
        fits.append(float(1 - torch.sqrt(rest.clamp(min=0)) / torch.sqrt(norm2)))
    for m in range(len(dims)):
        nr = a[m].norm(dim=0)
        a[m] = a[m] / nr
        lam = lam * nr
    pad = [torch.nn.functional.pad(x, (0, _stride(rank) - rank)) for x in a]
    return pad, lam, np.array(fits)


def exact(case, seed):
    kind = case["kind"]
    if case.get("precision") == "bf16":
        return None  # the rounding of the factors between iterations is part of the result
    s = _inputs(case, seed)
    if kind == "batch":
        flat, lams, fits = torch.zeros(s["flat"].shape, dtype=torch.float64, device="cuda"), [], []
        views = _batch_views(s["flat"], s["tensors"], s["ranks"])
        outs = _batch_views(flat, s["tensors"], s["ranks"])
        for (dims, inds, vals), r, fs, out in zip(s["tensors"], s["ranks"], views, outs):
            a, lam, f = _als64(dims, inds, vals, fs, r, case["iters"])
            for o, x in zip(out, a):
                o.copy_(x)
            lams.append(lam)
            fits.append(f)
        return [flat, torch.cat(lams), np.stack(fits)]
    dims, inds, vals, mats, rank = s["dims"], s["inds"], s["vals"], s["mats"], case["rank"]
    if kind in ("mttkrp", "host", "first"):
        out = [_mttkrp64(dims, inds, vals, mats, m, rank) for m in range(len(dims))]
        if kind == "host":
            return [o.cpu().numpy() for o in out]
        return out + [None, None] if kind == "first" else out
    if kind == "als":
        a, lam, fits = _als64(dims, inds, vals, mats, rank, case["iters"])
        return [*a, lam, fits]
    if kind == "gradient":
        res = torch.empty(vals.shape, dtype=torch.float64, device="cuda")
        step = (1 << 27) // rank
        for z in range(0, vals.numel(), step):
            p = mats[0].double()[inds[0][z:z + step].long()]
            for a, ix in zip(mats[1:], inds[1:]):
                p = p * a.double()[ix[z:z + step].long()]
            res[z:z + step] = p.sum(1) - vals[z:z + step].double()
        grads = [_mttkrp64(dims, inds, res, mats, m, rank) for m in range(len(dims))]
        return [0.5 * res.square().sum(), *grads]
    out = []
    for m, u in enumerate(mats):  # ttm: fibers in the order of their other coordinates
        rest = [k for k in range(len(dims)) if k != m]
        key = torch.zeros(vals.shape, dtype=torch.int64, device="cuda")
        for k in rest:
            key = key * dims[k] + inds[k].long()
        _, at = torch.unique(key, return_inverse=True)
        y = torch.zeros((int(at.max()) + 1, _stride(rank)), dtype=torch.float64, device="cuda")
        y[:, :rank].index_add_(0, at, vals.double()[:, None] * u.double()[inds[m].long()])
        out += [None] * len(rest) + [y]
    return out
