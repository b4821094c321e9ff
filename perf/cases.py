"""The work a user of n4b200 has it do, as cases that can be timed and checked.

A case is a dict of plain values; ``prepare`` makes what a program holds before
the call (volumes, masks, parameters, a recorded batch graph), ``run`` is one
pass through the package's public entry points, ``exact`` is the same result in
64 bits from plain torch, written here and independent of the package.

Kinds of cases
  n4        one volume through ``N4`` (CUDA tensors in, corrected volume and lattice out)
  batch     ``N4Batch`` over volumes of uneven sizes
  graph     ``N4BatchGraph`` over volumes of one size with the learned warm start, replayed
  fit       ``FitBspline3D`` of a masked field
  evaluate  ``EvaluateBspline3D`` of a lattice on every voxel
  sharpen   ``sharpenImage`` of a masked log image
  step      the component calls of one N4 iteration, as a program that drives the loop itself makes them
  train     one training step of the warm-start encoder

Volumes are the seeded phantoms of the package's workloads: nested ellipsoids
under a B-spline bias with Rician noise, the outer ellipsoid (about 38 % of the
field of view) as the mask.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-n4_b200"))

import n4b200  # noqa: E402
from n4b200 import _lib  # noqa: E402
from n4b200.encoder import Encoder, init_params  # noqa: E402
from n4b200.warmstart import load_encoder, phantoms_gpu  # noqa: E402

DEV = "cuda"


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one iteration driven from outside on the smallest ordinary volume: launches and host time count
        dict(name="step_64x64x48", kind="step", fx=64, fy=64, fz=48, nc=7),
        # a small volume, every level to a fixed count, as the CUDA program this one stands in for runs
        dict(name="n4_64x64x48", kind="n4", fx=64, fy=64, fz=48, shrink=1, levels=3, iters=12, thr=0.0, u8=False,
             bias=False, grid=4, sigma=0.03, std=0.15),
        # the ordinary clinical volume, shrunk by 4 and run to convergence
        dict(name="n4_256x256x176", kind="n4", fx=256, fy=256, fz=176, shrink=4, levels=4, iters=50, thr=0.001,
             u8=False, bias=False, grid=6, sigma=0.02, std=0.25),
        # the largest single volume (0.5 mm), shrunk by 2 and run to convergence
        dict(name="n4_512x512x320", kind="n4", fx=512, fy=512, fz=320, shrink=2, levels=4, iters=50, thr=0.001,
             u8=False, bias=False, grid=8, sigma=0.02, std=0.25),
        # a template-sized volume with odd axes at full resolution, byte mask, bias field asked for as well
        dict(name="n4_181x217x181", kind="n4", fx=181, fy=217, fz=181, shrink=1, levels=4, iters=5, thr=0.0, u8=True,
             bias=True, grid=6, sigma=0.02, std=0.25),
        # serving one size: a recorded batch with the learned warm start, replayed on refilled buffers; the
        # cluster shape is the one the autotuner picks for this size
        dict(name="graph_32x256x256x176", kind="graph", n=32, fx=256, fy=256, fz=176, shrink=4, levels=4, iters=50,
             thr=0.001, u8=False, grid=6, sigma=0.02, std=0.25, ctas=6),
        # a study of uneven volumes in one call, byte masks
        dict(name="batch_24_uneven", kind="batch", n=24, shrink=4, levels=4, iters=6, thr=0.0, u8=True, grid=4,
             sigma=0.03, std=0.15, dims_seed=4),
        # the fit alone on the fitting grid of the largest volume
        dict(name="fit_256x256x160", kind="fit", fx=256, fy=256, fz=160, nc=11, mask=True),
        # the fit on odd axes, whose rows no vector load can take
        dict(name="fit_181x217x181", kind="fit", fx=181, fy=217, fz=181, nc=7, mask=True),
        # the dense field of the largest volume
        dict(name="evaluate_512x512x320", kind="evaluate", fx=512, fy=512, fz=320, nc=11),
        # sharpening alone on the largest fitting grid
        dict(name="sharpen_256x256x160", kind="sharpen", fx=256, fy=256, fz=160, bins=200),
        # training the warm start: forward, backward and Adam on a batch of 64
        dict(name="train_64", kind="train", n=64),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _axes(rng, lo, hi, multiple=1):
    """Three axes whose product is spread evenly over its logarithm in [lo, hi], odd ones among them."""
    side = _log_uniform(rng, lo, hi) ** (1.0 / 3.0)
    out = []
    for _ in range(3):
        a = max(16, int(side * rng.uniform(0.8, 1.25)))
        out.append(max(multiple * 8, a // multiple * multiple))
    return out


def draw(rng):
    kind = rng.choice(["n4", "n4", "n4", "batch", "graph", "fit", "fit", "evaluate", "sharpen", "step", "train"])
    if kind == "n4":
        shrink = rng.choice([1, 1, 2, 4])
        top = min(60e6, 8e6 * shrink ** 3)
        fx, fy, fz = _axes(rng, 32 * 32 * 24 * shrink ** 3, top, shrink)
        levels = rng.randint(2, 4)
        return dict(kind=kind, fx=fx, fy=fy, fz=fz, shrink=shrink, levels=levels, iters=rng.randint(2, 6), thr=0.0,
                    u8=rng.random() < 0.5, bias=rng.random() < 0.3, grid=rng.choice([4, 6]), sigma=0.02, std=0.2)
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(3, 16), shrink=4, levels=rng.randint(3, 4), iters=rng.randint(3, 6),
                    thr=0.0, u8=rng.random() < 0.5, grid=4, sigma=0.03, std=0.15, dims_seed=rng.randint(0, 10 ** 6))
    if kind == "graph":
        fx, fy, fz = (8 * rng.randint(16, 32) for _ in range(3))
        return dict(kind=kind, n=rng.randint(4, 20), fx=fx, fy=fy, fz=min(fz, 200), shrink=4, levels=4, iters=50,
                    thr=0.001, u8=rng.random() < 0.5, grid=6, sigma=0.02, std=0.25, ctas=8)
    if kind == "train":
        return dict(kind=kind, n=rng.choice([8, 16, 24, 32, 48, 56]))
    top = 60e6 if kind == "evaluate" else 10e6
    fx, fy, fz = _axes(rng, 32 * 32 * 24, top if kind != "step" else 2e6)
    case = dict(kind=kind, fx=fx, fy=fy, fz=fz)
    if kind in ("fit", "evaluate", "step"):
        case["nc"] = rng.choice([4, 5, 7, 11])
    if kind == "fit":
        case["mask"] = rng.random() < 0.7
    if kind == "sharpen":
        case["bins"] = rng.choice([64, 128, 200, 256])
    return case


def _batch_dims(case):
    """Axes of an uneven batch: each a multiple of 8 in 96..288, as scanners give them."""
    rng = np.random.default_rng(case["dims_seed"])
    return [tuple(int(v) for v in rng.choice(np.arange(96, 289, 8), size=3)) for _ in range(case["n"])]


# ---------------------------------------------------------------- inputs
def _param(case, **kw):
    return n4b200.N4Param(NumberOfFittingLevels=case["levels"], MaximumNumberOfIterations=case["iters"],
                          ConvergenceThreshold=case["thr"], low_value=0.0, ShrinkFactor=case["shrink"], **kw)


def _phantom(case, shape, seed):
    im, mask = phantoms_gpu(1, shape, seed, sigma=case.get("sigma", 0.02), grid=case.get("grid", 6),
                            coeff_std=case.get("std", 0.25), device=DEV)
    im, mask = im[0], mask[0]
    return im, (mask.to(torch.uint8) if case.get("u8") else mask)


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "batch":
        st["volumes"] = [_phantom(case, d, 1000 * seed + i) for i, d in enumerate(_batch_dims(case))]
        st["param"] = _param(case)
        return st
    if kind == "train":
        g = _generator(seed)
        # pooled log intensities (0 outside the mask) and first-level log-bias lattices
        x = torch.randn((case["n"], 32, 32, 24), device=DEV, generator=g) * 0.3 - 0.7
        st["x"] = (x * (torch.rand(x.shape, device=DEV, generator=g) < 0.4)).to(torch.bfloat16)
        st["y"] = torch.randn((case["n"], 64), device=DEV, generator=g) * 0.2
        st["encoder"] = Encoder(max_batch=case["n"], seed=seed % 1000)
        return st
    shape = (case["fx"], case["fy"], case["fz"])
    if kind == "n4":
        st["im"], st["mask"] = _phantom(case, shape, seed)
        st["param"] = _param(case)
    elif kind == "graph":
        vols = [_phantom(case, shape, 1000 * seed + i) for i in range(case["n"])]
        param = _param(case, flags=n4b200.cluster_size_flag(case["ctas"]) | _lib.FLAG_CTA_512)
        st["ctx"], st["encoder"] = n4b200.Context(0), load_encoder(max_batch=case["n"])
        st["graph"] = n4b200.N4BatchGraph(vols, param, ctx=st["ctx"], encoder=st["encoder"])
    elif kind == "evaluate":
        st["lattice"] = torch.randn((case["nc"],) * 3, device=DEV, generator=_generator(seed)) * 0.1
    else:
        im, st["mask"] = _phantom(case, shape, seed)
        st["logim"] = torch.log(im.clamp_min(1e-3))
        if kind == "fit":
            # the residual of an iteration: a smooth part and noise
            g = _generator(seed)
            st["field"] = (st["logim"] + 0.6) * 0.05 + torch.randn(shape, device=DEV, generator=g) * 0.02
            st["mask"] = st["mask"] if case["mask"] else None
        elif kind == "step":
            g = _generator(seed)
            coeffs = torch.randn((2, 4, 4, 4), device=DEV, generator=g) * torch.tensor([0.2, 0.01], device=DEV).view(2, 1, 1, 1)
            st["before"] = n4b200.EvaluateBspline3D(coeffs[0], (4, 4, 4), shape)
            st["now"] = st["before"] + n4b200.EvaluateBspline3D(coeffs[1], (4, 4, 4), shape)
    return st


# ---------------------------------------------------------------- one pass
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "n4":
        r = n4b200.N4(st["im"], st["mask"], st["param"], return_bias=case["bias"])
        return [r.im_normalized, r.lattice] + ([r.bias_field] if case["bias"] else [])
    if kind == "batch":
        return [[r.im_normalized, r.lattice] for r in n4b200.N4Batch(st["volumes"], st["param"])]
    if kind == "graph":
        st["graph"].launch()
        return [[r.im_normalized, r.lattice] for r in st["graph"].sync()]
    if kind == "train":
        loss = st["encoder"].train_step(st["x"], st["y"], 1e-3)
        return [np.float32(loss), st["encoder"].grads()]
    if kind == "fit":
        return n4b200.FitBspline3D(st["field"], st["mask"], (case["nc"],) * 3)
    if kind == "evaluate":
        return n4b200.EvaluateBspline3D(st["lattice"], (case["nc"],) * 3, (case["fx"], case["fy"], case["fz"]))
    if kind == "sharpen":
        return n4b200.sharpenImage(st["logim"], st["mask"], case["bins"], 0.01, 0.15)
    # step: the last update's convergence, then sharpen, fit, evaluate, and the refined lattice of the next level
    nc = (case["nc"],) * 3
    cv = n4b200.CalculateConvergenceMeasurement(st["before"], st["now"], st["mask"])
    logu = st["logim"] - st["now"]
    residual = logu - n4b200.sharpenImage(logu, st["mask"], 200, 0.01, 0.15)
    lattice = n4b200.FitBspline3D(residual, st["mask"], nc)
    field = n4b200.EvaluateBspline3D(lattice, nc, (case["fx"], case["fy"], case["fz"]))
    return [cv, lattice, field, n4b200.UpsampleLattice3D(lattice)]


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "train":
        # layer outputs x taps, a multiply and an add, forward and twice that backward
        macs = 16 * 16 * 12 * 16 * 27 + 8 * 8 * 6 * 32 * 16 * 27 + 4 * 4 * 3 * 64 * 32 * 27 + 8 * 64 * 64 * 27 + 512 * 64
        return {"bytes": case["n"] * (32 * 32 * 24 * 2 + 64 * 4) + 213056 * 4 * 7, "flops": 6 * case["n"] * macs}
    if kind == "batch":
        voxels = sum(a * b * c for a, b, c in _batch_dims(case))
    else:
        voxels = case["fx"] * case["fy"] * case["fz"] * case.get("n", 1)
    if kind in ("n4", "batch", "graph"):
        io = 4 + (1 if case["u8"] else 4) + 4 + (4 if case.get("bias") else 0)
        # per masked fitting voxel and iteration: evaluate and update (8), convergence term (8), bin coordinate
        # twice (2 x 4), residual (2), four weighted sums (8); about 10 iterations a level where it runs to convergence
        its = case["levels"] * (case["iters"] if case["thr"] == 0.0 else 10)
        return {"bytes": voxels * io, "flops": 0.38 * voxels / case["shrink"] ** 3 * 34 * its}
    if kind == "evaluate":
        return {"bytes": 4 * voxels, "flops": 7 * voxels}
    if kind == "fit":
        return {"bytes": (8 if case["mask"] else 4) * voxels, "flops": 16 * voxels}
    if kind == "sharpen":
        return {"bytes": 12 * voxels, "flops": 20 * voxels}
    return {"bytes": (4 * 3 + 4 + 4) * voxels, "flops": 60 * voxels}


# ---------------------------------------------------------------- 64 bits, plain torch
def _weights(n, nc):
    """Dense [n, nc] cubic B-spline weights of one axis."""
    spans = nc - 3
    span = np.float64(n) / np.float64(spans)
    u = np.arange(n, dtype=np.float64) + 0.5
    s = np.minimum(np.floor(u / span).astype(np.int64), spans - 1)
    t = (u - s * span) / span
    w = np.stack([(1 - t) ** 3 / 6, (3 * t ** 3 - 6 * t ** 2 + 4) / 6, (-3 * t ** 3 + 3 * t ** 2 + 3 * t + 1) / 6,
                  t ** 3 / 6], axis=1)
    m = np.zeros((n, nc))
    m[np.repeat(np.arange(n), 4), (s[:, None] + np.arange(4)).ravel()] = w.ravel()
    return torch.tensor(m, device=DEV)


def _contract(f, wx, wy, wz):
    t = (f.reshape(-1, f.shape[2]) @ wz).reshape(f.shape[0], f.shape[1], -1)
    t = torch.einsum("xyc,yb->xbc", t, wy)
    return torch.einsum("xbc,xa->abc", t, wx)


def _fit(f, m, nc, eps=1e-3):
    """Sum of w^3 r / sum(w^2) over sum of w^2, voxel weights w = wx wy wz."""
    ws = [_weights(n, c) for n, c in zip(f.shape, nc)]
    ps = [w ** 3 / (w ** 2).sum(1, keepdim=True) for w in ws]
    zero = torch.zeros((), dtype=torch.float64, device=DEV)
    return _contract(torch.where(m, f, zero), *ps) / (_contract(m.double(), *[w ** 2 for w in ws]) + eps)


def _evaluate(lat, shape):
    wx, wy, wz = (_weights(n, c) for n, c in zip(shape, lat.shape))
    t = torch.einsum("abc,xa->xbc", lat, wx)
    t = torch.einsum("xbc,yb->xyc", t, wy)
    return (t.reshape(-1, t.shape[2]) @ wz.T).reshape(shape)


def _refine(lat):
    for axis in range(3):
        a = lat.movedim(axis, 0)
        n = a.shape[0] - 3
        pad = torch.cat([a[:1], a, a[-1:]])
        out = torch.zeros((2 * n + 3,) + a.shape[1:], dtype=torch.float64, device=DEV)
        out[1::2] = pad[1:n + 2] / 8 + 6 * pad[2:n + 3] / 8 + pad[3:n + 4] / 8
        out[0::2] = (a[0:n + 2] + a[1:n + 3]) / 2
        lat = out.movedim(0, axis)
    return lat.contiguous()


def _sharpen(x, bins=200, noise=0.01, fwhm=0.15):
    """The sharpened values of the masked values x."""
    lo, hi = x.min(), x.max()
    slope = (hi - lo) / (bins - 1)
    c = (x - lo) / slope
    k = torch.floor(c).long()
    f = c - k
    top = k >= bins - 1
    w0 = torch.where(top & (f != 0), torch.zeros_like(f), 1 - f)
    w1 = torch.where(top, torch.zeros_like(f), f)
    hist = torch.zeros(bins + 2, dtype=torch.float64, device=DEV)
    hist += torch.bincount(k.clamp(0, bins), w0, bins + 2) + torch.bincount((k + 1).clamp(0, bins + 1), w1, bins + 2)
    pad = int(2.0 ** (math.ceil(math.log(bins) / math.log(2.0)) + 1) + 0.5)
    off = int(0.5 * (pad - bins))
    v = torch.zeros(pad, dtype=torch.float64, device=DEV)
    v[off:off + bins] = hist[:bins]
    scaled = fwhm / slope
    i = torch.arange(pad, dtype=torch.float64, device=DEV)
    i = torch.minimum(i, pad - i)
    g = 2.0 * math.sqrt(math.log(2.0) / math.pi) / scaled * torch.exp(-i * i * 4.0 * math.log(2.0) / (scaled * scaled))
    gf, vf = torch.fft.fft(g), torch.fft.fft(v)
    u = torch.fft.ifft(vf * (gf.conj() / (gf.conj() * gf + noise)).real).real.clamp_min(0.0)
    centers = lo + (torch.arange(pad, dtype=torch.float64, device=DEV) - off) * slope
    nu = torch.fft.ifft(torch.fft.fft(centers * u) * gf).real
    de = torch.fft.ifft(torch.fft.fft(u) * gf).real
    e = torch.where(de != 0, nu / torch.where(de != 0, de, torch.ones_like(de)), torch.zeros_like(de))[off:off + bins]
    kl = k.clamp(0, bins - 2)
    return torch.where(top, e[-1], e[kl] + (e[kl + 1] - e[kl]) * (c - kl))


def _n4(im, mask, case):
    """Corrected volume, lattice and bias field of fixed iteration counts."""
    s = case["shrink"]
    im = im.double()
    on = (mask != 0) & (im > 0.0)
    im = torch.where(im > 0.0, im, torch.zeros_like(im))
    small, m = im, on
    if s > 1:
        x, y, z = (d // s for d in im.shape)
        cnt = on.double().reshape(x, s, y, s, z, s).sum((1, 3, 5))
        small = (im * on).reshape(x, s, y, s, z, s).sum((1, 3, 5)) / cnt.clamp_min(1.0)
        m = (2 * cnt > s ** 3) & (small > 0.0)
    logim = torch.where(m, torch.log(small.clamp_min(1e-300)), torch.zeros_like(small))
    lat = torch.zeros((4, 4, 4), dtype=torch.float64, device=DEV)
    for level in range(case["levels"]):
        if level:
            lat = _refine(lat)
        for _ in range(case["iters"]):
            logu = logim - _evaluate(lat, logim.shape)
            r = torch.zeros_like(logu)
            r[m] = logu[m] - _sharpen(logu[m])
            lat = lat + _fit(r, m, lat.shape)
    b = torch.exp(_evaluate(lat, im.shape))
    return im / b, lat, b


def _train(st):
    from torch.nn import functional as F
    ch = [1, 16, 32, 64, 64]
    flat = torch.tensor(init_params(st["seed"] % 1000), device=DEV).double().requires_grad_(True)
    at, parts = 0, []
    for l in range(4):
        n = ch[l + 1] * ch[l] * 27
        parts += [flat[at:at + n].reshape(ch[l + 1], ch[l], 3, 3, 3), flat[at + n:at + n + ch[l + 1]]]
        at += n + ch[l + 1]
    a = st["x"].double()[:, None]
    for l in range(4):
        a = F.relu(F.conv3d(a, parts[2 * l], parts[2 * l + 1], stride=2, padding=1))
    out = a.reshape(a.shape[0], -1) @ flat[at:at + 64 * 512].reshape(64, 512).T + flat[at + 64 * 512:]
    loss = ((out - st["y"].double()) ** 2).mean()
    loss.backward()
    return [loss.detach(), flat.grad]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("n4", "batch", "graph") and case["thr"] != 0.0:
        # run to convergence, a volume stops where one value falls below the threshold: 64-bit arithmetic can stop an
        # iteration earlier or later than 32-bit logs do, and then has no value for the run's own count
        return None
    if kind == "evaluate":
        return _evaluate(prepare(case, seed)["lattice"].double(), (case["fx"], case["fy"], case["fz"]))
    if kind == "train":
        return _train(dict(prepare(case, seed), seed=seed))
    st = prepare(case, seed)
    if kind == "n4":
        return list(_n4(st["im"], st["mask"], case))[:3 if case["bias"] else 2]
    if kind == "batch":
        return [list(_n4(im, mask, case))[:2] for im, mask in st["volumes"]]
    if kind == "fit":
        m = st["mask"] != 0 if case["mask"] else torch.ones_like(st["field"], dtype=torch.bool)
        return _fit(st["field"].double(), m, (case["nc"],) * 3)
    m = st["mask"] != 0
    if kind == "sharpen":
        x = st["logim"].double()
        out = torch.zeros_like(x)
        out[m] = _sharpen(x[m], case["bins"])
        return out
    d = torch.exp(st["before"].double() - st["now"].double())[m]
    cv = float(d.std(unbiased=False) / d.mean())
    logu = (st["logim"] - st["now"]).double()
    r = torch.zeros_like(logu)
    r[m] = logu[m] - _sharpen(logu[m])
    lat = _fit(r, m, (case["nc"],) * 3)
    return [cv, lat, _evaluate(lat, logu.shape), _refine(lat)]
