"""The work that users of this framework have it do, as cases that can be timed.

Every case is one call, or one training step, through the public Python entry
points over libdtsgb: the class mirror of the reference's API (host arrays in,
host arrays out), the batched solves on device buffers, and the autograd
functions.  Parameters are those of the framework's drivers (cli.py) and
benchmark workloads (bench.py, workloads.py); inputs are synthetic images of
the same roles: polygon guides with noise, piecewise-planar depths, sparse or
dense confidences.

A case is a dict of plain values; "kind" selects the path:

  dts     Batch.upload_device + solve_dts + download_device
  hfbs    Batch.upload_device + solve_hfbs + download_device
  chroma  HFBS class on device buffers, one solve per chroma channel
  ragged  one Batch of images of uneven size, DTS and HFBS of each
  single  EdgeAwareOptimize with a DomainTransformSolver (host arrays)
  filter  DomainTransformFilter.Filter (host arrays)
  stereo  DomainTransformStereo, the calls of the stereo driver (host arrays)
  dts_grad, hfbs_grad, soft_grad   forward + backward of the autograd functions
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import domain_transform_solver_gb300 as D
from domain_transform_solver_gb300 import autograd as A

DEV = "cuda"


# ---- the cases ------------------------------------------------------------------
def listed():
    return [
        # a thumbnail or preview frame refined while a user drags a slider: the
        # smallest call, where launches and host work count
        dict(name="dts_preview_160x120", kind="dts", n=1, w=160, h=120, sigma=8.0, sigma_z=8.0,
             loss=1, over=-1.0, iters=10, bf16=False),
        # the reference's own call: one 640x480 depth map, 8x upsampled, host to host
        dict(name="dts_single_640x480", kind="single", w=640, h=480),
        # depth super-resolution by 16: the same scene size as the driver's
        # datasets and its widest windows (sigma_z = 8 * 16 / 1.8)
        dict(name="dts_depth_x16_1376x1088", kind="dts", n=1, w=1376, h=1088, sigma=128.0,
             sigma_z=71.11111, loss=1, over=-1.0, iters=10, bf16=False),
        # colorization of a camera photo by DTS: Charbonnier loss, wide windows,
        # strokes overwritten
        dict(name="dts_strokes_3264x2448", kind="dts", n=1, w=3264, h=2448, sigma=64.0,
             sigma_z=30.0, loss=2, over=0.85, iters=10, bf16=False),
        # depth super-resolution by HFBS with 64-pixel cells: a small grid
        dict(name="hfbs_depth_1376x1088", kind="hfbs", n=1, w=1376, h=1088, sigma=64.0,
             sigma_l=16.0, steps=140, bf16=False),
        # colorization of a camera photo by HFBS with the default grid (8-pixel
        # cells, 64 luma levels, 140 steps), both chroma channels
        dict(name="hfbs_chroma_3264x2448", kind="chroma", w=3264, h=2448, sigma=8.0, sigma_l=4.0,
             steps=140),
        # a dataset solved in one go: 64 images of uneven size, BF16 storage, DTS
        # and HFBS of each (the benchmark's default workload)
        dict(name="ragged_64_bf16", kind="ragged", n=64, wmin=256, wmax=1920, hmin=256, hmax=1080,
             layout=1003, bf16=True),
        # one training step through the DTS layer: batch 16 of 1024x768
        dict(name="dts_train_16x1024x768", kind="dts_grad", n=16, w=1024, h=768, iters=10),
        # one training step through the HFBS layer: two 640x480 channels
        dict(name="hfbs_train_2x640x480", kind="hfbs_grad", n=2, w=640, h=480, steps=64),
        # one training step that also learns the edge weights (soft windows)
        dict(name="soft_train_4x1024x768", kind="soft_grad", n=4, w=1024, h=768, iters=10),
        # edge-aware smoothing of a video frame, host to host
        dict(name="filter_1280x720", kind="filter", w=1280, h=720, iters=3),
        # disparity refinement as the stereo driver does it, host to host
        dict(name="stereo_720x540", kind="stereo", w=720, h=540),
    ]


def _size(rng: random.Random, lo: int, hi: int, most: int):
    """Width and height, each spread over the logarithm of [lo, hi], of at most
    `most` pixels; odd and ragged ones as likely as round ones."""
    while True:
        w = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        h = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if rng.random() < 0.3:
            w = max(lo, w // 32 * 32)
        if w * h <= most:
            return w, h


def draw(rng: random.Random):
    kind = rng.choice(["dts", "dts", "dts", "strokes", "hfbs", "hfbs", "chroma", "ragged", "single",
                       "dts_grad", "hfbs_grad", "soft_grad", "filter", "stereo"])
    if kind == "dts":  # previews up to depth super-resolution by 2, 4, 8, 16
        up = rng.choice([1, 2, 4, 8, 16])
        w, h = _size(rng, 48, 1536, 1376 * 1088)
        n = rng.choice([1, 1, 1, 2, 3, 4])
        return dict(kind="dts", n=n if n * w * h <= 1376 * 1088 else 1, w=w, h=h, sigma=8.0 * up,
                    sigma_z=8.0 if up == 1 else 8.0 * up / 1.8, loss=1, over=-1.0, iters=10,
                    bf16=rng.random() < 0.4)
    if kind == "strokes":
        w, h = _size(rng, 320, 3280, 3264 * 2448)
        return dict(kind="dts", n=1, w=w, h=h, sigma=64.0, sigma_z=30.0, loss=2, over=0.85, iters=10,
                    bf16=rng.random() < 0.3)
    if kind == "hfbs":
        w, h = _size(rng, 96, 1536, 1376 * 1088)
        return dict(kind="hfbs", n=1, w=w, h=h, sigma=8.0 * rng.choice([2, 4, 8, 16]), sigma_l=16.0,
                    steps=140, bf16=rng.random() < 0.3)
    if kind == "chroma":
        w, h = _size(rng, 240, 3280, 3264 * 2448)
        return dict(kind="chroma", w=w, h=h, sigma=8.0, sigma_l=rng.choice([4.0, 4.0, 8.0, 16.0]),
                    steps=rng.choice([64, 140]))
    if kind == "ragged":
        a, b = rng.randrange(64, 512), rng.randrange(64, 512)
        return dict(kind="ragged", n=rng.randrange(3, 33), wmin=a, wmax=a + rng.randrange(1, 1400),
                    hmin=b, hmax=b + rng.randrange(1, 560), layout=rng.randrange(1 << 20),
                    bf16=rng.random() < 0.7)
    if kind == "single":
        w, h = _size(rng, 128, 1536, 1376 * 1088)
        return dict(kind="single", w=w, h=h)
    if kind == "dts_grad":
        w, h = _size(rng, 96, 1280, 1024 * 768)
        return dict(kind="dts_grad", n=rng.randrange(1, 17), w=w, h=h, iters=rng.choice([5, 10]))
    if kind == "hfbs_grad":
        w, h = _size(rng, 96, 1280, 1024 * 768)
        return dict(kind="hfbs_grad", n=rng.randrange(1, 4), w=w, h=h, steps=rng.choice([32, 64]))
    if kind == "soft_grad":
        w, h = _size(rng, 96, 1280, 1024 * 768)
        return dict(kind="soft_grad", n=rng.randrange(1, 5), w=w, h=h, iters=rng.choice([5, 10]))
    if kind == "filter":
        w, h = _size(rng, 128, 1920, 1920 * 1080)
        return dict(kind="filter", w=w, h=h, iters=rng.choice([1, 3]))
    w, h = _size(rng, 160, 768, 768 * 768)
    return dict(kind="stereo", w=w, h=h)


def _ragged_sizes(case):
    rng = random.Random(case["layout"])
    return [(rng.randint(case["wmin"], case["wmax"]), rng.randint(case["hmin"], case["hmax"]))
            for _ in range(case["n"])]


# ---- parameters -----------------------------------------------------------------
def _dts_params(case):
    if case["kind"] == "dts":
        f = dict(sigma_x=case["sigma"], sigma_y=case["sigma"],
                 sigma_r=0.25 if case["loss"] == 2 else 0.1)
        o = dict(num_iterations=case["iters"], loss=case["loss"], lambda_=0.99,
                 sigma_z=case["sigma_z"], step_size=0.99)
    else:
        f = dict(sigma_x=8.0, sigma_y=8.0, sigma_r=0.1)
        o = dict(num_iterations=case.get("iters", 10), loss=1, lambda_=0.99, sigma_z=8.0,
                 step_size=0.99)
    return f, o


def _hfbs_params(case):
    return dict(sigma_x=case.get("sigma", 8.0), sigma_y=case.get("sigma", 8.0),
                sigma_l=case.get("sigma_l", 16.0), lambda_=8.0, alpha=1.0, beta=0.9,
                bistoch_iter_max=20, optim_iter_max=case.get("steps", 64), neg_exp_beta=0.9)


_STEREO_FILTER = dict(sigma_x=8.0, sigma_y=8.0, sigma_r=0.1)
_STEREO_OPT = dict(num_iterations=1, loss=2, lambda_=0.99, sigma_z=30.0, step_size=0.99,
                   photo_consis_lambda=0.01, DT_lambda=0.0)
_CONF = dict(sigma_x=8.0, sigma_y=8.0, sigma_r=0.2, sigmas=[16.0, 0.0])
_STEREO_OFFSET, _STEREO_CLEAR = 0.0, 20
_FILTER = dict(sigma_x=8.0, sigma_y=8.0, sigma_r=0.2)


# ---- synthetic inputs ---------------------------------------------------------------
def _labels(rs: np.random.RandomState, w, h, n_poly):
    """(h, w) int64 labels of n_poly random convex polygons over a background."""
    lab = torch.zeros((h, w), dtype=torch.int64, device=DEV)
    for i in range(1, n_poly + 1):
        r = rs.uniform(0.05, 0.35) * min(w, h)
        cx, cy = rs.uniform(0, w), rs.uniform(0, h)
        x0, x1 = max(int(cx - r), 0), min(int(cx + r) + 1, w)
        y0, y1 = max(int(cy - r), 0), min(int(cy + r) + 1, h)
        a = rs.uniform(0, 2 * math.pi, rs.randint(2, 6))
        d = rs.uniform(0.3, 0.9, len(a)) * r
        if x1 <= x0 or y1 <= y0:
            continue
        xx = torch.arange(x0, x1, device=DEV, dtype=torch.float32) - float(cx)
        yy = torch.arange(y0, y1, device=DEV, dtype=torch.float32)[:, None] - float(cy)
        m = None
        for t, q in zip(a, d):
            k = xx * math.cos(t) + yy * math.sin(t) <= float(q)
            m = k if m is None else m & k
        lab[y0:y1, x0:x1] = torch.where(m, i, lab[y0:y1, x0:x1])
    return lab


def _edge_weights(imgs, f):
    """dH, dV of each image, as a program that learns them computes them itself."""
    return [[x.float() for x in _weights(_ycbcr(g), f)] for g, _, _ in imgs]


class _Scene:
    """A polygon scene: labels, and the seeded generators of its planes and noise."""

    def __init__(self, seed, w, h, n_poly=40):
        self.rs = np.random.RandomState((int(seed) * 2654435761 + w * 40503 + h) % (1 << 32))
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(int(self.rs.randint(1 << 30)))
        self.w, self.h, self.n = w, h, n_poly
        self.lab = _labels(self.rs, w, h, n_poly)

    def per_label(self, lo, hi):
        return torch.from_numpy(self.rs.uniform(lo, hi, self.n + 1).astype(np.float32)).to(DEV)

    def noise(self, scale):
        return scale * torch.randn((self.h, self.w), device=DEV, generator=self.gen)

    def rand(self):
        return torch.rand((self.h, self.w), device=DEV, generator=self.gen)

    def planes(self, lo, hi):
        span = (hi - lo) / max(self.w, self.h)
        a, b, c = self.per_label(lo, hi), self.per_label(-span, span), self.per_label(-span, span)
        xx = torch.arange(self.w, device=DEV, dtype=torch.float32) - self.w / 2
        yy = torch.arange(self.h, device=DEV, dtype=torch.float32)[:, None] - self.h / 2
        return (a[self.lab] + b[self.lab] * xx + c[self.lab] * yy).clamp_(lo, hi)

    def rgba(self, sigma=3.0):
        """RGB colours per polygon plus N(0, sigma) noise, alpha 255."""
        out = torch.full((self.h, self.w, 4), 255, dtype=torch.uint8, device=DEV)
        for k in range(3):
            v = torch.floor(self.per_label(0, 256))[self.lab] + self.noise(sigma)
            out[..., k] = v.round_().clamp_(0, 255).to(torch.uint8)
        return out

    def grey(self):
        """A smoothly shaded grey guide, the same value in R, G, B."""
        xx = torch.arange(self.w, device=DEV, dtype=torch.float32) - self.w / 2
        yy = torch.arange(self.h, device=DEV, dtype=torch.float32)[:, None] - self.h / 2
        v = self.per_label(30, 225)[self.lab]
        v = v + self.per_label(-0.15, 0.15)[self.lab] * xx + self.per_label(-0.15, 0.15)[self.lab] * yy
        v = v.round_().clamp_(0, 255).to(torch.uint8)
        return torch.stack([v, v, v, torch.full_like(v, 255)], dim=2).contiguous()


def _sparse_depth(sc, stride=None, frac=None):
    """Depths in [0.5, 10] plus N(0, 0.01) at the samples, 0 elsewhere, and the confidence (1 there)."""
    conf = torch.zeros((sc.h, sc.w), device=DEV)
    if stride:
        conf[::stride, ::stride] = 1.0
    else:
        conf = (sc.rand() < frac).float()
    return (sc.planes(0.5, 10.0) + sc.noise(0.01)) * conf, conf


def _dense_depth(sc):
    """An interpolated depth in [0, 1] and a bump confidence in (0, 1]."""
    t = (sc.planes(0.05, 0.95) + sc.noise(0.002)).clamp_(0, 1)
    return t, 0.02 + 0.98 * sc.rand()


def _strokes(sc):
    """A chroma plane in [0, 255] (128 outside the strokes) and the stroke mask."""
    mask = (torch.floor(sc.per_label(0, 3))[sc.lab] == 0) & (sc.rand() < 0.5)
    return torch.where(mask, torch.floor(sc.per_label(60, 196))[sc.lab], 128.0), mask.float()


def _chroma(sc, frac=0.02):
    """U and V in [-0.5, 0.5] at a random 2% of the pixels, confidence 1 there."""
    mask = (sc.rand() < frac).float()
    return [sc.per_label(-0.5, 0.5)[sc.lab] * mask for _ in range(2)], mask


def _images(case, seed):
    """The case's instances on the GPU: rgba, target(s), confidence."""
    kind = case["kind"]
    if kind == "ragged":
        out = []
        for i, (w, h) in enumerate(_ragged_sizes(case)):
            sc = _Scene(seed * 1000 + i, w, h)
            out.append((sc.rgba(), *_sparse_depth(sc, frac=0.05)))
        return out
    out = []
    for i in range(case.get("n", 1)):
        w, h = case["w"], case["h"]
        if kind in ("chroma", "hfbs_grad"):
            sc = _Scene(seed * 1000 + i, w, h, 30)
            g = sc.grey()
            uv, c = _chroma(sc)
            out.append((g, uv if kind == "chroma" else uv[0], c))
            continue
        sc = _Scene(seed * 1000 + i, w, h)
        if kind == "dts" and case["loss"] == 2:
            out.append((sc.grey(), *_strokes(sc)))
        elif kind == "dts" and case["sigma"] > 8.0:
            out.append((sc.rgba(), *_dense_depth(sc)))
        elif kind == "hfbs":
            t, c = _dense_depth(sc)
            out.append((sc.rgba(), (t - 0.5) * 128.0, c))
        elif kind == "filter":
            out.append((sc.rgba(), sc.planes(0.0, 255.0) + sc.noise(8.0), None))
        elif kind == "stereo":
            disp = sc.planes(4.0, 60.0)
            g = sc.rgba()
            t = disp + sc.noise(0.5)
            xs = (torch.arange(w, device=DEV) + disp.round().long()) % w
            right = torch.gather(g, 1, xs[..., None].expand(-1, -1, 4)).contiguous()
            out.append((g, t, right))
        else:
            out.append((sc.rgba(), *_sparse_depth(sc, stride=8)))
    return out


def _grad_seed(case, seed, shape):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + 13)
    return torch.randn(shape, device=DEV, generator=gen)


# ---- what a program has in hand -----------------------------------------------------
class _State:
    pass


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def prepare(case, seed):
    s = _State()
    kind = s.kind = case["kind"]
    imgs = _images(case, seed)
    if kind in ("dts", "hfbs", "ragged"):
        s.sizes = [(t.shape[1], t.shape[0]) for _, t, _ in imgs]
        s.imgs = [(g.contiguous(), t.contiguous(), c.contiguous()) for g, t, c in imgs]
        s.batch = D.Batch(s.sizes, flags=D.FLAG_BF16_STORAGE if case["bf16"] else 0)
        s.stream = torch.cuda.Stream()
        s.batch.set_stream(s.stream.cuda_stream)
        f, o = _dts_params(case)
        s.filt, s.opt = D.DomainFilterParams(**f), D.DomainOptimizeParams(**o)
        s.over = case.get("over", -1.0)
        s.grid = D.HFBSGridParams(**_hfbs_params(case))
        # results side by side in one buffer, image after image
        offs = np.cumsum([0] + [w * h for w, h in s.sizes])
        s.ins = [[x.data_ptr() for x in part] for part in zip(*s.imgs)]
        s.outs = {}
        for which in (0, 1) if kind == "ragged" else (0,) if kind == "dts" else (1,):
            buf = torch.empty(int(offs[-1]), device=DEV)
            s.outs[which] = (buf, [buf.data_ptr() + 4 * int(a) for a in offs[:-1]])
        return s
    if kind == "chroma":
        s.rgba, s.targets, s.conf = imgs[0]
        w, h = case["w"], case["h"]
        p = _hfbs_params(case)
        gx, gy, gl = _grid_dims(w, h, p)
        s.hfbs = D.HFBS(D.ImageDim(w, h), gx + 1, gy + 1, gl + 1)
        s.hfbs.SetFilterParams(D.HFBSGridParams(**p))
        s.stream = torch.cuda.Stream()
        s.hfbs.SetStream(s.stream.cuda_stream)
        s.outs = [torch.empty((h, w), device=DEV) for _ in range(2)]
        return s
    if kind in ("single", "filter", "stereo"):
        dim = D.ImageDim(case["w"], case["h"])
        g, t, c = imgs[0]
        s.rgba, s.target = _host(g), _host(t)
        s.other = None if c is None else _host(c)
        s.dim = dim
        if kind == "single":
            f, o = _dts_params(case)
            s.options = D.DtsOptions(filter_options=D.DomainFilterParams(**f),
                                     optim_options=D.DomainOptimizeParams(**o), image_dims=dim)
            s.solver = D.DomainTransformSolver(dim)
        elif kind == "filter":
            s.solver = D.DomainTransformFilter(dim)
            s.iters = case["iters"]
        else:
            s.solver = D.DomainTransformStereo(dim)
        return s
    # training steps: stacked images, inputs that want gradients, an upstream gradient
    s.rgba = torch.stack([g for g, _, _ in imgs])
    s.target = torch.stack([t for _, t, _ in imgs]).requires_grad_(True)
    s.conf = torch.stack([c for _, _, c in imgs]).requires_grad_(True)
    s.grad = _grad_seed(case, seed, s.target.shape)
    f, o = _dts_params(case)
    s.filt, s.opt = D.DomainFilterParams(**f), D.DomainOptimizeParams(**o)
    s.grid = D.HFBSGridParams(**_hfbs_params(case))
    if kind == "soft_grad":
        s.dh, s.dv = (torch.stack(x).requires_grad_(True) for x in zip(*_edge_weights(imgs, f)))
    return s


# ---- one pass -----------------------------------------------------------------------
def run(s):
    k = s.kind
    if k in ("dts", "hfbs", "ragged"):
        cur = torch.cuda.current_stream()
        s.stream.wait_stream(cur)
        s.batch.upload_device(D.COLOR_SPACE.YCbCr, *s.ins)
        if k != "hfbs":
            s.batch.solve_dts(s.filt, s.opt, s.over)
        if k != "dts":
            s.batch.solve_hfbs(s.grid)
        for which, (_, ptrs) in s.outs.items():
            s.batch.download_device(which, ptrs)
        cur.wait_stream(s.stream)
        return [buf for buf, _ in s.outs.values()]
    if k == "chroma":
        cur = torch.cuda.current_stream()
        s.stream.wait_stream(cur)
        for t, o in zip(s.targets, s.outs):
            s.hfbs.InitFrameDevice(D.COLOR_SPACE.RGB, s.rgba.data_ptr(), t.data_ptr(),
                                   s.conf.data_ptr())
            s.hfbs.Optimize()
            s.hfbs.DownloadDevice(D.ImageType.OPTIMIZED_QUANTITY, o.data_ptr())
        cur.wait_stream(s.stream)
        return s.outs
    if k == "single":
        return D.EdgeAwareOptimize(s.rgba, s.target, s.other, s.options, s.solver)[0]
    if k == "filter":
        s.solver.SetImageDim(s.dim)
        s.solver.InitFrame(D.COLOR_SPACE.RGB, s.rgba)
        return s.solver.Filter(D.DomainFilterParams(**_FILTER), s.target, s.iters)
    if k == "stereo":
        v = s.solver
        v.SetImageDim(s.dim)
        v.ClearAll()
        v.InitFrame(D.COLOR_SPACE.RGB, s.rgba, s.target, None)
        v.InitRightFrame(_STEREO_OFFSET, D.COLOR_SPACE.RGB, s.other)
        v.ComputeConfidence(D.DomainFilterParamsVec1(**_CONF), _STEREO_CLEAR)
        v.ComputeColorSpaceDifferential(D.DomainFilterParams(**_STEREO_FILTER))
        v.IntegrateColorDifferentials()
        v.ProcessRightFrame()
        v.Optimize(D.DomainOptimizeParams(**_STEREO_OPT), -1.0)
        return v.Download(D.ImageType.OPTIMIZED_QUANTITY)
    if k == "dts_grad":
        v = A.dts_solve(s.rgba, s.target, s.conf, s.filt, s.opt)
        return [v.detach(), *torch.autograd.grad(v, (s.target, s.conf), s.grad)]
    if k == "hfbs_grad":
        v = A.hfbs_solve(s.rgba, s.target, s.conf, s.grid)
        return [v.detach(), *torch.autograd.grad(v, (s.target, s.conf), s.grad)]
    v = A.soft_dts_solve(s.dh, s.dv, s.target, s.conf, s.opt, 1.0)
    return [v.detach(), *torch.autograd.grad(v, (s.dh, s.dv, s.target, s.conf), s.grad)]


def work(case):
    """Inputs read once, results written once, and the solver's own arithmetic:
    about 30 operations per pixel and DTS iteration (two window means and the
    update), 20 per voxel and heavy-ball or normalisation step; three times that
    with a backward."""
    kind = case["kind"]
    px = sum(w * h for w, h in _ragged_sizes(case)) if kind == "ragged" else \
        case.get("n", 1) * case["w"] * case["h"]
    sizes = _ragged_sizes(case) if kind == "ragged" else \
        [(case["w"], case["h"])] * (2 if kind == "chroma" else case.get("n", 1))
    flops = 0.0
    if kind not in ("hfbs", "chroma", "hfbs_grad"):
        its = {"stereo": 4, "filter": case.get("iters", 3)}.get(kind, case.get("iters", 10))
        flops += 30.0 * px * its
    if kind in ("hfbs", "chroma", "ragged", "hfbs_grad"):
        p = _hfbs_params(case)
        vx = sum(math.prod(_grid_dims(w, h, p)) for w, h in sizes)
        flops += 20.0 * vx * (p["bistoch_iter_max"] + p["optim_iter_max"])
    per_px = {"ragged": 20, "chroma": 4 + 4 + 8 + 8, "filter": 12, "stereo": 16, "dts_grad": 28,
              "hfbs_grad": 28, "soft_grad": 40}.get(kind, 16)
    if kind.endswith("_grad"):
        flops *= 3.0
    return {"bytes": float(per_px * px), "flops": flops}


# ---- the same in 64 bits, in plain torch ------------------------------------------------
F64 = torch.float64


def _f32(x):
    return float(np.float32(x))


def _fma(a, b, c):
    """a * b + c with one rounding (a: a number; b, c: tensors), by Dekker's and Knuth's error-free
    product and sum."""
    def split(x):
        t = 134217729.0 * x
        hi = t - (t - x)
        return hi, x - hi
    p = a * b
    ah, al = split(a)
    bh, bl = split(b)
    e = ((ah * bh - p) + ah * bl + al * bh) + al * bl
    s = p + c
    z = s - p
    return s + (((p - (s - z)) + (c - z)) + e)


def _ycbcr(rgba):
    """The reference's colour conversion: double arithmetic with multiply-adds, truncated."""
    r, g, b = (rgba[..., k].to(F64) for k in range(3))
    one = torch.ones_like(r)
    y = _fma(0.114, b, _fma(0.299, r, 0.587 * g))
    cb = _fma(0.5, b, _fma(-0.331264, g, _fma(-0.168736, r, 128.0 * one)))
    cr = _fma(-0.081312, b, _fma(-0.418688, g, _fma(0.5, r, 128.0 * one)))
    return torch.stack([torch.trunc(v) for v in (y, cb, cr)] + [rgba[..., 3].to(F64)], -1)


def _weights(guide, f):
    """dH, dV of a guide (h, w, 4) of whole numbers in 64 bits."""
    out = []
    for axis, s in ((1, f["sigma_x"]), (0, f["sigma_y"])):
        r = float(np.float32(s) / np.float32(f["sigma_r"]))
        prev = torch.zeros_like(guide)
        prev.narrow(axis, 1, guide.shape[axis] - 1).copy_(guide.narrow(axis, 0, guide.shape[axis] - 1))
        ssd = ((guide - prev) ** 2).sum(-1)
        out.append(torch.sqrt(ssd * _f32(0.0000153787) * r * r + 1.0))
    return out


def _windows(e, axis, sigma, limit):
    """The window of each pixel along `axis` (0: y, 1: x): index of the prefix sum before its first
    pixel and after its last, and its number of pixels."""
    n = e.shape[axis]
    ct = torch.cumsum(e, axis)
    dl = torch.ones(e.shape, dtype=torch.int64, device=e.device)
    du = torch.zeros_like(dl)
    for k in range(min(int(sigma) + 1, n - 1), 0, -1):
        far = (ct.narrow(axis, k, n - k) - ct.narrow(axis, 0, n - k)) > sigma
        a = dl.narrow(axis, k, n - k)
        a.copy_(torch.where(far, k, a))
        m = min(limit, n) - k
        if m > 0:
            b = du.narrow(axis, 0, m)
            b.copy_(torch.where(far.narrow(axis, 0, m), k - 1, b))
    # no pixel beyond sigma: the window keeps the pixel itself (dl = 1, du = 0); du of a pixel whose
    # first neighbour is already beyond is 0 as well
    shape = [1, 1]
    shape[axis] = n
    p = torch.arange(n, device=e.device).view(shape)
    return p - dl + 1, p + du + 1, (dl + du).to(F64)


def _box(v, win, axis):
    lo, hi, n = win
    zero = torch.zeros_like(v.narrow(axis, 0, 1))
    s = torch.cat([zero, torch.cumsum(v, axis)], axis)
    return (torch.gather(s, axis, hi) - torch.gather(s, axis, lo)) / n


def _dts64(guide, t, c, f, o, over=-1.0, photo=None):
    dh, dv = _weights(guide, f)
    sz, h, w = _f32(o["sigma_z"]), *t.shape
    wx, wy = _windows(dh, 1, sz, w), _windows(dv, 0, sz, min(w, h))
    lam, st = _f32(o["lambda_"]), _f32(o["step_size"])
    fixed = (c > over) if 0 < over < 1 else None
    cn = c / wx[2]
    v = t
    for _ in range(o["num_iterations"]):
        if fixed is not None:
            v = torch.where(fixed, t, v)
        d = v - t
        g = cn * d if o["loss"] == 1 else 0.5 * cn * d / torch.sqrt(d * d + _f32(1e-6))
        if photo is not None:
            g = g + 0.5 * photo(v)
        v = v - st * (lam * (v - _box(v, wx, 1)) + g)
        if fixed is not None:
            v = torch.where(fixed, t, v)
        v = v - st * lam * (v - _box(v, wy, 0))
    return v


def _filter64(guide, chans, f, iters):
    dh, dv = _weights(guide, f)
    h, w = chans[0].shape
    for it in range(iters):
        m = np.float32(1 if it == 0 else 3 * 2.0 ** (iters - it - 1) / math.sqrt(4.0 ** iters - 1))
        wx = _windows(dh, 1, float(np.float32(f["sigma_x"]) * m), w)
        wy = _windows(dv, 0, float(np.float32(f["sigma_y"]) * m), min(w, h))
        chans = [_box(_box(v, wx, 1), wy, 0) for v in chans]
    return chans


def _stereo64(g, t, right):
    left, rt, tt = g.to(F64), right.to(F64), t.to(F64)
    h, w = t.shape
    m1, m2 = _filter64(left, [tt, tt * tt], _CONF, 3)
    var = m2 - m1 * m1
    conf = torch.where(var < 0, 0.0, torch.exp(-var * (0.5 / _CONF["sigmas"][0] ** 2)))
    conf[:, : _STEREO_CLEAR + 1] = 0.0
    sxr = np.float32(_STEREO_FILTER["sigma_r"]) / np.float32(_STEREO_FILTER["sigma_x"])
    dh_r = _weights(rt, _STEREO_FILTER)[0]

    def photo(v):
        x = torch.arange(w, device=v.device, dtype=torch.float32)
        xr = (_STEREO_OFFSET + x) - v.float()
        ok = (xr >= 0) & (xr < w)
        xi = torch.where(ok, xr, 0.0).long()
        sad = (left - torch.gather(rt, 1, xi[..., None].expand(-1, -1, 4))).abs().sum(-1)
        gr = torch.gather(dh_r, 1, xi)
        val = _f32(_STEREO_OPT["photo_consis_lambda"]) * 2 * sad * _f32(0.00392156863) * \
            ((gr * gr - 1) * float(sxr * sxr))
        return torch.where(ok, val, 0.0)
    return _dts64(left, tt, conf, _STEREO_FILTER, _STEREO_OPT, photo=photo)


def _grid_dims(w, h, p):
    return (int(math.ceil(np.float32(w) / np.float32(p["sigma_x"]))),
            int(math.ceil(np.float32(h) / np.float32(p["sigma_y"]))),
            int(math.ceil(255.0 / float(np.float32(p["sigma_l"])))))


def _hfbs64(luma, t, c, p, faces=True):
    """HFBS of one image; faces: the normalisation reads the reference's pad faces (an allocation
    larger than the grid)."""
    h, w = t.shape
    gx, gy, gl = _grid_dims(w, h, p)
    dev = t.device

    def axis(n, s):
        q = torch.arange(n, device=dev, dtype=torch.float32) / np.float32(s)
        return q.to(F64), torch.floor(q).long()
    fx, bx = axis(w, p["sigma_x"])
    fy, by = axis(h, p["sigma_y"])
    fl, bl = axis(256, p["sigma_l"])
    fz, bz = fl[luma], bl[luma]
    # bins over (gl + 1) levels: the last one holds the luma overflow
    at = (bz * gy + by[:, None]) * gx + bx

    def splat(v):
        out = torch.zeros((gl + 1) * gy * gx, dtype=F64, device=dev)
        return out.index_add(0, at.reshape(-1), v.reshape(-1)).view(gl + 1, gy, gx)
    cnt_all = splat(torch.ones_like(t))
    cnt, csum, b = cnt_all[:gl], splat(c)[:gl], splat(c * t)[:gl]

    def nb6(a, pad=(0.0, 0.0, 0.0)):
        s = torch.zeros_like(a)
        for ax, value in ((2, pad[0]), (1, pad[1]), (0, pad[2])):
            n = a.shape[ax]
            shape = list(a.shape)
            shape[ax] = 1
            z, e = a.new_zeros(shape), a.new_full(shape, value)
            s = s + torch.cat([z, a.narrow(ax, 0, n - 1)], ax) + torch.cat([a.narrow(ax, 1, n - 1), e], ax)
        return s
    eps = _f32(0.00001)
    norm = torch.ones_like(cnt)
    for it in range(p["bistoch_iter_max"]):
        pad = [1.0 if faces and g % 8 and it % 2 == 0 else 0.0 for g in (gx, gy, gl)]
        norm = torch.sqrt(norm * (cnt + eps) / (2 * norm + nb6(norm, pad) + eps))
    lam = _f32(p["lambda_"])
    inv = 1.0 / torch.clamp(lam * (cnt - 2 * norm * norm) + csum, min=1e-3)
    beta = _f32(p["neg_exp_beta"])

    def blur(a):
        for ax in (2, 1, 0):
            i = torch.arange(a.shape[ax], device=dev, dtype=F64)
            k = beta ** (i[:, None] - i[None, :]).abs()
            a = torch.movedim(torch.tensordot(torch.movedim(a, ax, -1), k, dims=1), -1, ax)
        return a
    z = blur(b) / (blur(csum) + 1e-7)
    hb = torch.zeros_like(z)
    al, be = _f32(p["alpha"]), _f32(p["beta"])
    for _ in range(p["optim_iter_max"]):
        g = z - (b + lam * norm * nb6(z * norm)) * inv
        hb = be * hb + torch.where(g.abs() > 1.345, torch.sign(g), g)
        z = z - al * hb
    # count-weighted trilinear slice; zeros past the grid, counts but no z in the overflow level
    cw = torch.nn.functional.pad(cnt_all, (0, 1, 0, 1, 0, 1))
    zw = torch.nn.functional.pad(z, (0, 1, 0, 1, 0, 2)) * cw
    num = den = 0.0
    wz = (fz - torch.floor(fz))
    wx, wy = fx - torch.floor(fx), (fy - torch.floor(fy))[:, None]
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                k = ((bz + dz) * (gy + 1) + by[:, None] + dy) * (gx + 1) + bx + dx
                wt = (wx if dx else 1 - wx) * (wy if dy else 1 - wy) * (wz if dz else 1 - wz)
                num = num + zw.reshape(-1)[k] * wt
                den = den + cw.reshape(-1)[k] * wt
    return num / den


def _soft64(dh, dv, t, c, o, tau=1.0):
    """The soft-window solve: along a line, w_pq = clamp((sigma - D_pq) / tau + 1/2, 0, 1)."""
    sig, reach = _f32(o["sigma_z"]), int(math.ceil(o["sigma_z"] + tau / 2)) + 1
    lam, st = _f32(o["lambda_"]), _f32(o["step_size"])
    axes = []
    for e, ax in ((dh, 1), (dv, 0)):
        ct, n = torch.cumsum(e, ax), e.shape[ax]
        ws = []
        for k in range(1, min(reach, n - 1) + 1):
            d = ct.narrow(ax, k, n - k) - ct.narrow(ax, 0, n - k)
            ws.append(torch.clamp((sig - d) / tau + 0.5, 0.0, 1.0))
        axes.append((ax, n, ws))

    def both(v, ax, n, ws, own):
        """own weight times v plus every pair's weight times the other end's v."""
        s = own * v
        for k, wk in enumerate(ws, 1):
            pad = [0, 0, k, 0] if ax == 0 else [k, 0, 0, 0]
            rev = [0, 0, 0, k] if ax == 0 else [0, k, 0, 0]
            s = s + torch.nn.functional.pad(wk * v.narrow(ax, 0, n - k), pad)
            s = s + torch.nn.functional.pad(wk * v.narrow(ax, k, n - k), rev)
        return s
    own = min(max(sig / tau + 0.5, 0.0), 1.0)
    ns = [both(torch.ones_like(t), *a, own) for a in axes]
    v = t
    for _ in range(o["num_iterations"]):
        v = v - st * (lam * (v - both(v, *axes[0], own) / ns[0]) + c / ns[0] * (v - t))
        v = v - st * lam * (v - both(v, *axes[1], own) / ns[1])
    return v


def exact(case, seed):
    kind = case["kind"]
    imgs = _images(case, seed)
    f, o = _dts_params(case)
    p = _hfbs_params(case)
    if kind in ("dts", "hfbs", "ragged"):
        res = []
        for which in (0, 1) if kind == "ragged" else (0,) if kind == "dts" else (1,):
            parts = []
            for g, t, c in imgs:
                if case["bf16"]:
                    t, c = t.bfloat16(), c.bfloat16()
                guide, t, c = _ycbcr(g), t.to(F64), c.to(F64)
                v = _dts64(guide, t, c, f, o, case.get("over", -1.0)) if which == 0 else \
                    _hfbs64(guide[..., 0].long(), t, c, p)
                parts.append(v.reshape(-1))
            res.append(torch.cat(parts))
        return res
    if kind == "chroma":
        g, uv, c = imgs[0]
        return [_hfbs64(g[..., 0].long(), t.to(F64), c.to(F64), p) for t in uv]
    if kind == "single":
        g, t, c = imgs[0]
        return _dts64(_ycbcr(g), t.to(F64), c.to(F64), f, o)
    if kind == "filter":
        return _filter64(imgs[0][0].to(F64), [imgs[0][1].to(F64)], _FILTER, case["iters"])[0]
    if kind == "stereo":
        return _stereo64(*imgs[0])
    grad = _grad_seed(case, seed, (len(imgs), case["h"], case["w"])).to(F64)
    if kind == "soft_grad":
        dhv = _edge_weights(imgs, f)
    rows = []
    for i, (g, t, c) in enumerate(imgs):
        t, c = (x.to(F64).requires_grad_(True) for x in (t, c))
        if kind == "dts_grad":
            wrt = (t, c)
            v = _dts64(_ycbcr(g), t, c, f, o)
        elif kind == "hfbs_grad":
            wrt = (t, c)
            v = _hfbs64(_ycbcr(g)[..., 0].long(), t, c, p, faces=False)
        else:
            dh, dv = (x.to(F64).requires_grad_(True) for x in dhv[i])
            wrt = (dh, dv, t, c)
            v = _soft64(dh, dv, t, c, o)
        rows.append([v.detach(), *torch.autograd.grad(v, wrt, grad[i])])
    return [torch.stack(col) for col in zip(*rows)]
