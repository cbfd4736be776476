"""The paths that a launch picks by size, type or alignment, each at the sizes
where it can go wrong."""
import numpy as np
import pytest

import parity as P

pytestmark = pytest.mark.gpu


# ---- splat: a CTA per cell from 256 pixels a cell on ---------------------------
@pytest.mark.parametrize("w,h,sx,sy,sl,guide", [
    (97, 53, 16.0, 16.0, 16.0, "noise"),      # 256-pixel cells, runs of one pixel
    (255, 130, 51.0, 5.0, 16.0, "noise"),     # 255 pixels: a thread per cell
    (200, 170, 32.0, 32.0, 5.0, "noise"),     # one chunk exactly; luma bin 51 overflows
    (200, 170, 33.0, 31.5, 4.0, "steps"),     # ragged cells
    (150, 140, 128.0, 100.0, 16.0, "flat"),   # one run through every chunk
    (300, 41, 300.0, 41.0, 1.0, "noise"),     # one cell, 255 luma bins (and an overflow bin)
])
@pytest.mark.parametrize("bf16", [0, 1])
def test_splat_sums_of_large_cells(gpu_ready, w, h, sx, sy, sl, guide, bf16):
    """Counts are exact; a sum of n float products is within n * 2^-23 of
    their absolute sum (n - 1 additions and one product, each 2^-24)."""
    D = gpu_ready
    rng = np.random.default_rng(w + h)
    y, x = np.mgrid[0:h, 0:w]
    luma = {"noise": rng.integers(0, 256, (h, w)), "flat": np.full((h, w), 200),
            "steps": (x // 7 + y // 3) * 11 % 256}[guide].astype(np.uint8)
    rgba = np.repeat(luma[..., None], 4, axis=2)
    t = rng.normal(0, 10, (h, w)).astype(np.float32)
    c = rng.random((h, w)).astype(np.float32)
    b = D.Batch([(w, h)], flags=D.FLAG_BF16_STORAGE if bf16 else 0)
    b.upload(D.COLOR_SPACE.RGB, [rgba], [t], [c])
    b.solve_hfbs(D.HFBSGridParams(sigma_x=sx, sigma_y=sy, sigma_l=sl, bistoch_iter_max=1,
                                  optim_iter_max=1))
    if bf16:
        t, c = P.bf16_round(t), P.bf16_round(c)
    f = np.float32
    dims = (int(np.ceil(f(w) / f(sx))), int(np.ceil(f(h) / f(sy))), int(np.ceil(255.0 / sl)))
    bx = np.floor(x.astype(f) / f(sx)).astype(int)
    by = np.floor(y.astype(f) / f(sy)).astype(int)
    bl = np.floor(luma.astype(f) / f(sl)).astype(int)
    at = ((bl * dims[1] + by) * dims[0] + bx).ravel()

    def bins(v):
        full = np.bincount(at, weights=v.astype(np.float64).ravel(),
                           minlength=(dims[2] + 1) * dims[1] * dims[0])
        return full[:dims[2] * dims[1] * dims[0]].reshape(dims[2], dims[1], dims[0])
    n = bins(np.ones((h, w)))
    assert np.array_equal(b.debug_grid(0, 1, dims), n.astype(f))
    ct = c.astype(np.float64) * t
    for which, v in ((2, c.astype(np.float64)), (3, ct)):
        err = np.abs(b.debug_grid(0, which, dims) - bins(v))
        assert (err <= n * 2.0 ** -23 * bins(np.abs(v))).all(), which


# ---- overwrite: held by the iteration itself ----------------------------------
@pytest.mark.parametrize("w,h,sz", [(70, 45, 8.0), (33, 140, 30.0), (400, 300, 71.0),
                                    (900, 700, 12.0)])
@pytest.mark.parametrize("loss,flags", [(1, 0), (2, 0), (1, 1)])
def test_overwritten_pixels_hold_the_target(gpu_ready, oracle_mod, w, h, sz, loss, flags):
    """Against the FP64 oracle on the GPU's windows, within the parity bar;
    one iteration alone leaves its last Y half-step on them."""
    from domain_transform_solver_gb300 import workloads as W
    from test_gpu_dts import _run_dts
    D, O = gpu_ready, oracle_mod
    inst = W.depth_sr_instance(90 + w, w, h, n_poly=9, sample_frac=0.2)
    inst.target[:] += (inst.confidence == 0) * np.float32(2.0)
    t, c = inst.target, inst.confidence
    if flags:
        t, c = P.bf16_round(t), P.bf16_round(c)
    for n in (1, 4):
        opt = dict(W.CFG0_OPT, num_iterations=n, loss=loss, sigma_z=sz)
        v, s = _run_dts(D, inst, 1, W.CFG0_FILTER, opt, 0.85, flags)
        szf = float(np.float32(sz))
        win = {(a, szf): s.DebugBounds(a, szf) for a in (0, 1)}
        ref, _ = O.dts_solve(inst.rgba, t, c, 1, W.CFG0_FILTER, opt, 0.85, overrides=win)
        assert np.abs(v - ref).max() <= P.TOL_REL * P.target_range(t), n


# ---- device copies: vectors or single pixels -----------------------------------
@pytest.mark.parametrize("sizes", [[(64, 40)], [(65, 40)], [(1, 1), (3, 9), (512, 8)],
                                   [(2048, 1700), (513, 9)]])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("flags", [0, 1])
def test_device_copies_of_any_alignment(gpu_ready, sizes, shift, flags):
    """Images at 16-byte boundaries and one element past them, of widths that
    are and are not multiples of four: what comes back after no iterations is
    the target, bit for bit."""
    torch = pytest.importorskip("torch")
    D = gpu_ready
    rng = np.random.default_rng(7)
    dev = torch.device("cuda:0")
    ts = [rng.normal(0, 5, (h, w)).astype(np.float32) for w, h in sizes]
    rg = [rng.integers(0, 256, (h, w, 4)).astype(np.uint8) for w, h in sizes]

    def put(a):
        flat = torch.from_numpy(np.ascontiguousarray(a).view(np.float32).reshape(-1))
        buf = torch.zeros(flat.numel() + 4, device=dev)
        buf[shift:shift + flat.numel()] = flat
        return buf
    tb, gb = [put(t) for t in ts], [put(g) for g in rg]
    ob = [torch.full((w * h + 4,), -1.0, device=dev) for w, h in sizes]
    torch.cuda.synchronize()
    b = D.Batch(sizes, flags=flags)
    b.upload_device(D.COLOR_SPACE.YCbCr, [x.data_ptr() + 4 * shift for x in gb],
                    [x.data_ptr() + 4 * shift for x in tb], None)
    b.solve_dts(D.DomainFilterParams(8.0, 8.0, 0.1), D.DomainOptimizeParams(num_iterations=0))
    b.download_device(0, [x.data_ptr() + 4 * shift for x in ob])
    host = b.download(0)
    for t, o, hv in zip(ts, ob, host):
        want = P.bf16_round(t) if flags else t
        assert np.array_equal(hv, want)
        got = o.cpu().numpy()
        assert np.array_equal(got[shift:shift + t.size].reshape(t.shape), want)
        assert (got[:shift] == -1).all() and (got[shift + t.size:] == -1).all()


# ---- HFBS: clusters for grids that stay on chip, marches for the others --------
@pytest.mark.parametrize("gx,gy,sl,steps,bistoch", [
    (24, 5, 16.0, 5, 7),     # clusters of one row a CTA, of fewer CTAs than 16
    (25, 1, 16.0, 6, 2),     # one row: one CTA
    (1, 9, 255.0, 8, 20),    # one column, one level
    (22, 17, 16.0, 9, 3),    # 16 CTAs, nine of them with rows
    (49, 12, 15.0, 3, 1),    # 17 levels: five groups, the last with one
    (128, 64, 16.0, 4, 6),   # the most a cluster holds: 131072 voxels
    (129, 64, 16.0, 5, 7),   # one column past it: marches, a last pass of one step
    (240, 33, 17.0, 7, 3),   # ten strips exactly, 15 levels
    (71, 30, 4.0, 9, 5),     # 64 levels, the most a march takes
    (30, 7, 3.95, 9, 5),     # 65 levels: one step per launch
    (73, 150, 8.0, 4, 4),    # 32 levels, several blocks along y
])
def test_grid_solvers_match_the_oracle(gpu_ready, oracle_mod, gx, gy, sl, steps, bistoch):
    """Normalisation and solution of grids at the edges of the clusters' slabs
    and the marches' strips, levels and passes, against the FP64 oracle at the
    parity bar (targets small enough that the Huber clamp stays out)."""
    D, O = gpu_ready, oracle_mod
    rng = np.random.default_rng(gx * 100 + gy)
    w, h = 8 * gx - 3 if gx > 1 else 8, 8 * gy - 5
    luma = rng.integers(0, 256, (h, w)).astype(np.uint8)
    rgba = np.repeat(luma[..., None], 4, axis=2)
    t = rng.uniform(-0.5, 0.5, (h, w)).astype(np.float32)
    c = (rng.random((h, w)) < 0.3).astype(np.float32)
    gl = int(np.ceil(255.0 / float(np.float32(sl))))
    params = dict(sigma_x=8.0, sigma_y=8.0, sigma_l=sl, lambda_=8.0, alpha=1.0, beta=0.9,
                  bistoch_iter_max=bistoch, optim_iter_max=steps, neg_exp_beta=0.9)
    dims = (gx + 1, gy + 1, gl + 1)
    s = D.HFBS(D.ImageDim(w, h), *dims)
    s.SetFilterParams(D.HFBSGridParams(**params))
    s.InitFrame(D.COLOR_SPACE.RGB, rgba, t, c)
    s.Optimize()
    assert s.GridDims() == (gx, gy, gl)
    ref, o, st = O.hfbs_solve(rgba, t, c, 0, params, max_grid=dims)
    assert st == 0
    norm = o.grid("splat_norm")
    assert np.abs(s.DebugGrid(3) - norm).max() <= 1e-5 * max(1.0, float(np.abs(norm).max()))
    assert np.abs(s.DebugGrid(7) - o.grid("z_final")).max() <= P.TOL_REL * P.target_range(t)
    out = s.Download(D.ImageType.OPTIMIZED_QUANTITY)
    fin = np.isfinite(ref)
    assert np.abs(out[fin] - ref[fin]).max() <= P.TOL_REL * P.target_range(t)


# ---- DTS passes ---------------------------------------------------------------
@pytest.mark.parametrize("w,h,sz", [
    (236, 40, 8.0),     # a row of one X segment exactly (two rounds)
    (237, 33, 8.0),     # one column past it; a second Y tile of one row
    (365, 200, 16.5),   # three rounds; the widest halo of 8 rows a warp
    (493, 1100, 17.0),  # four rounds, one column past; 16 rows a warp
    (900, 600, 56.0), (900, 600, 57.0),     # 16 | 32 rows a warp
    (780, 720, 61.0),   # halos of more than one round
    (777, 700, 127.9), (777, 700, 128.0),   # 12 | 16 warps a tile
    (700, 760, 201.0),  # 20 warps
    (60, 50, 253.9),    # the widest halo, wider than the image
    (5000, 3, 30.0), (3, 5000, 30.0),
])
def test_passes_match_the_oracle(gpu_ready, oracle_mod, w, h, sz):
    """Segment, tile and halo edges of both passes, alone and in a batch of two
    (other launch shapes, the same bits), against the FP64 oracle on the GPU's
    windows, within the parity bar."""
    from domain_transform_solver_gb300 import workloads as W
    from test_gpu_dts import _run_dts
    D, O = gpu_ready, oracle_mod
    inst = W.depth_sr_instance(17 + w, w, h, n_poly=7, sample_frac=0.2)
    other = W.depth_sr_instance(18 + w, 700, 800, n_poly=7, sample_frac=0.2)
    opt = dict(W.CFG0_OPT, num_iterations=3, sigma_z=sz)
    v, s = _run_dts(D, inst, 1, W.CFG0_FILTER, opt)
    szf = float(np.float32(sz))
    win = {(a, szf): s.DebugBounds(a, szf) for a in (0, 1)}
    ref, _ = O.dts_solve(inst.rgba, inst.target, inst.confidence, 1, W.CFG0_FILTER, opt,
                         overrides=win)
    assert np.abs(v - ref).max() <= P.TOL_REL * P.target_range(inst.target)
    b = D.Batch([(w, h), (700, 800)])
    b.upload(D.COLOR_SPACE.YCbCr, [inst.rgba, other.rgba], [inst.target, other.target],
             [inst.confidence, other.confidence])
    b.solve_dts(D.DomainFilterParams(**W.CFG0_FILTER), D.DomainOptimizeParams(**opt))
    assert np.array_equal(b.download(0)[0], v)


# ---- HFBS adjoint: one cluster per grid where every step's iterate is kept -----
@pytest.mark.parametrize("w,h,sx,sy,sl,steps", [
    (200, 8, 8.0, 8.0, 16.0, 9),       # one row: a cluster of one
    (90, 70, 8.0, 8.0, 29.0, 12),      # nine levels, rows that do not divide
    (97, 141, 8.0, 8.0, 63.0, 1),      # five levels, one step
    (640, 480, 8.0, 8.0, 16.0, 6),     # two items a thread, every thread used
    (512, 512, 8.0, 8.0, 16.0, 5),     # the largest cube of 16 levels
    (648, 488, 8.0, 8.0, 16.0, 5),     # just above: a launch per step
])
def test_adjoint_in_clusters_is_the_adjoint_by_steps(gpu_ready, w, h, sx, sy, sl, steps):
    """Recomputed segments take a launch per step; both round alike."""
    D = gpu_ready
    rng = np.random.default_rng(w * 3 + h)
    rgba = rng.integers(0, 256, (2, h, w, 4)).astype(np.uint8)
    t = rng.normal(0, 2, (2, h, w)).astype(np.float32)
    c = rng.random((2, h, w)).astype(np.float32)
    gout = rng.standard_normal((2, h, w)).astype(np.float32)
    f = np.float32
    dims = (int(np.ceil(f(w) / f(sx))), int(np.ceil(f(h) / f(sy))), int(np.ceil(255.0 / sl)))
    got = []
    for segment in (1, 3):
        s = [D.HFBS(D.ImageDim(w, h), *dims) for _ in range(2)]
        for i in range(2):
            s[i].SetFilterParams(D.HFBSGridParams(sigma_x=sx, sigma_y=sy, sigma_l=sl,
                                                  optim_iter_max=steps))
            s[i].EnableGrad(True, segment)
            s[i].InitFrame(D.COLOR_SPACE.RGB, rgba[i], t[i], c[i])
            s[i].Optimize()
            got.append(s[i].Backward(gout[i]))
    for i in range(2):
        assert np.abs(got[i][0]).max() > 0
        assert np.array_equal(got[i][0], got[2 + i][0])
        assert np.array_equal(got[i][1], got[2 + i][1])


# ---- window bounds: a pass along rows and a pass down columns ------------------
@pytest.mark.parametrize("w,h,sigma", [
    (1, 1, 8.0), (3, 200, 8.0), (200, 3, 8.0), (40, 300, 71.0),  # lines shorter than a window
    (130, 70, 8.0), (333, 257, 0.5), (109, 110, 15.9),           # one tile more or less
    (493, 450, 8.0), (1030, 520, 8.0),                           # segments of 3 and 4 rounds
    (700, 90, 64.0), (90, 700, 130.0), (1200, 460, 253.0),       # wide halos, 32 rows a warp
])
@pytest.mark.parametrize("fix_y", [0, 1])
def test_window_bounds_are_the_searches_of_the_fixed_point_weights(gpu_ready, w, h, sigma, fix_y):
    """The linear search over the fixed-point weights, bit for bit."""
    D = gpu_ready
    rng = np.random.default_rng(w + 7 * h)
    y, x = np.mgrid[0:h, 0:w]
    rgba = (rng.integers(0, 40, (h, w, 4)) + ((x // 9 + y // 5) % 3 * 60)[..., None]).astype(np.uint8)
    rgba[..., 3] = 255
    s = D.DomainTransformSolver(D.ImageDim(w, h), D.FLAG_FIX_Y_LIMIT if fix_y else 0)
    s.InitFrame(D.COLOR_SPACE.RGB, rgba, np.zeros((h, w), np.float32), None)
    fp = D.DomainFilterParams(sigma_x=8.0, sigma_y=6.0, sigma_r=0.3)
    s.ComputeColorSpaceDifferential(fp)
    f = np.float32
    r = int(np.floor(f(sigma))) + 1
    F = 30 - int(np.ceil(np.log2(r * float(f(sigma) + f(1)))))
    T = int(np.floor(float(f(sigma)) * 2.0 ** F))
    for axis, sig in ((0, fp.sigma_x), (1, fp.sigma_y)):
        g = rgba.astype(np.int64) if axis == 0 else rgba.astype(np.int64).transpose(1, 0, 2)
        n, lines = g.shape[1], g.shape[0]
        ratio = f(sig) / f(fp.sigma_r)
        d = ((g[:, 1:] - g[:, :-1]) ** 2).sum(-1).astype(f)
        t = (d * f(0.0000153787)) * ratio
        wt = np.sqrt((t.astype(np.float64) * float(ratio) + 1.0).astype(f))
        q = np.rint(np.minimum(wt, f(sigma) + f(1)) * f(2.0 ** F)).astype(np.int64)
        S = np.concatenate([np.zeros((lines, 1), np.int64), np.cumsum(q, axis=1)], axis=1)
        lim = n if axis == 0 else (n if fix_y else min(w, h))
        pos = np.arange(n)[None, :]
        lower = np.broadcast_to(pos - 1, (lines, n)).copy()
        upper = np.broadcast_to(pos, (lines, n)).copy()
        for k in range(min(r, n - 1), 0, -1):  # the nearest pixel beyond sigma wins
            far = S[:, k:] - S[:, :-k] > T
            lower[:, k:][far] = np.broadcast_to(pos[:, k:] - k, far.shape)[far]
            stop = far & (pos[:, k:] < lim)
            upper[:, :-k][stop] = np.broadcast_to(pos[:, :-k] + k - 1, far.shape)[stop]
        got = s.DebugBounds(axis, sigma)
        want = (lower, upper) if axis == 0 else (lower.T, upper.T)
        assert np.array_equal(got[0], want[0]), axis
        assert np.array_equal(got[1], want[1]), axis


# ---- caller pointers by value: 128 instances a launch --------------------------
@pytest.mark.parametrize("n", [128, 129, 300])
def test_more_images_than_a_launch_has_pointers_for(gpu_ready, n):
    import torch
    D = gpu_ready
    rng = np.random.default_rng(n)
    sizes = [(int(w), int(h)) for w, h in rng.integers(1, 24, (n, 2))]
    g = [rng.integers(0, 256, (h, w, 4)).astype(np.uint8) for w, h in sizes]
    t = [rng.normal(0, 1, (h, w)).astype(np.float32) for w, h in sizes]
    c = [rng.random((h, w)).astype(np.float32) for w, h in sizes]
    host, dev = D.Batch(sizes), D.Batch(sizes)
    dev.set_stream(torch.cuda.Stream().cuda_stream)
    to = [[torch.from_numpy(a).cuda() for a in x] for x in (g, t, c)]
    out = [torch.full((h, w), -1.0, device="cuda") for w, h in sizes]
    torch.cuda.synchronize()
    fp, op = D.DomainFilterParams(), D.DomainOptimizeParams(num_iterations=2, loss=1, sigma_z=4.0)
    host.upload(D.COLOR_SPACE.YCbCr, g, t, c)
    host.solve_dts(fp, op)
    dev.upload_device(D.COLOR_SPACE.YCbCr, *[[a.data_ptr() for a in x] for x in to])
    dev.solve_dts(fp, op)
    dev.download_device(0, [o.data_ptr() for o in out])
    torch.cuda.synchronize()
    for a, o in zip(host.download(0), out):
        assert np.array_equal(a, o.cpu().numpy())


# ---- DTS adjoint: a Y^T pass and an X^T pass -----------------------------------
@pytest.mark.parametrize("w,h,sz", [
    (1, 1, 8.0), (3, 130, 8.0), (129, 33, 0.5), (365, 200, 8.0),  # segments of 2 and 3 rounds
    (1030, 520, 8.0),                                             # of 4, 128 staged rows
    (300, 120, 40.0), (700, 300, 76.9),                           # wide halos, 32 rows a warp
])
@pytest.mark.parametrize("bf16", [0, 1])
def test_adjoint_passes_match_the_oracle(gpu_ready, oracle_mod, w, h, sz, bf16):
    """The bar of the adjoint's tests (1e-4 of the largest gradient), alone and
    in a batch with the same bits."""
    import test_gpu_adjoint as A
    D = gpu_ready
    rng = np.random.default_rng(w + h)
    flags = D.FLAG_BF16_STORAGE if bf16 else 0
    data = []
    for ww, hh in ((w, h), (37, 21)):
        y, x = np.mgrid[0:hh, 0:ww]
        rgba = (rng.integers(0, 9, (hh, ww, 4)) + ((x // 23 + y // 17) % 3 * 70)[..., None])
        t, c, g = (rng.standard_normal((hh, ww)).astype(np.float32),
                   rng.random((hh, ww)).astype(np.float32),
                   rng.standard_normal((hh, ww)).astype(np.float32))
        if bf16:
            t, c = P.bf16_round(t), P.bf16_round(c)
        data.append((rgba.astype(np.uint8), t, c, g))
    opt = dict(num_iterations=3, loss=1, lambda_=0.9, sigma_z=sz, step_size=0.8)
    got = []
    for d in (data[:1], data):
        b = A._batch(D, d, opt, flags=flags)
        gt, gc = b.backward([g for _, _, _, g in d])
        got.append((gt[0], gc[0]))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    rgba, t, c, g = data[0]
    o = A._oracle(oracle_mod, rgba, t, c, A._gpu_windows(D, rgba, t, c, sz, flags))
    rt, rc = o.backward(3, 1, 0.9, sz, 0.8, g)
    A._check_grad(got[0][0], rt, 1)
    if rc.any():  # windows of one pixel leave v at t: dL/dc is zero, its float form rounding
        A._check_grad(got[0][1], rc, 1)


def test_adjoint_of_wider_windows_is_refused(gpu_ready):
    import test_gpu_adjoint as A
    D = gpu_ready
    data = [(np.zeros((9, 9, 4), np.uint8), *(np.ones((9, 9), np.float32) for _ in range(3)))]
    opt = dict(num_iterations=2, loss=1, lambda_=0.9, sigma_z=77.0, step_size=0.8)
    with pytest.raises(D.DtsgbError):
        A._batch(D, data, opt).backward([data[0][3]])


# ---- HFBS blur: lines of up to 32 levels in registers --------------------------
@pytest.mark.parametrize("sl", [255.0, 17.0, 16.0, 15.0, 8.0, 7.9])  # 1, 15, 16, 17, 32, 33 levels
@pytest.mark.parametrize("w,h", [(40, 90), (700, 600)])  # both fields in a warp or one
def test_blur_is_the_recursion_along_each_axis(gpu_ready, sl, w, h):
    """Sums of positive terms, two roundings a step and direction: relative
    error at most 4 * 2^-24 a step of the three sweeps."""
    D = gpu_ready
    rng = np.random.default_rng(int(sl) + w)
    rgba = rng.integers(0, 256, (h, w, 4)).astype(np.uint8)
    c = rng.random((h, w)).astype(np.float32)
    f = np.float32
    dims = (int(np.ceil(f(w) / f(4))), int(np.ceil(f(h) / f(4))), int(np.ceil(255.0 / sl)))
    s = D.HFBS(D.ImageDim(w, h), *dims)
    s.SetFilterParams(D.HFBSGridParams(sigma_x=4.0, sigma_y=4.0, sigma_l=sl, bistoch_iter_max=1,
                                       optim_iter_max=1, neg_exp_beta=0.9))
    s.InitFrame(D.COLOR_SPACE.RGB, rgba, np.ones((h, w), np.float32), c)
    s.Optimize()
    ref = s.DebugGrid(1).astype(np.float64)
    beta = float(f(0.9))
    for axis in (2, 1, 0):
        a = np.moveaxis(ref, axis, 0)
        fwd, bwd = a.copy(), np.zeros_like(a)
        for i in range(1, len(a)):
            fwd[i] += beta * fwd[i - 1]
        for i in range(len(a) - 2, -1, -1):
            bwd[i] = beta * (bwd[i + 1] + a[i + 1])
        ref = np.moveaxis(fwd + bwd, 0, axis)
    got = s.DebugGrid(5)
    assert (np.abs(got - ref) <= sum(dims) * 2.0 ** -22 * ref).all()


# ---- host images whose rows do not fill the pitch ------------------------------
@pytest.mark.parametrize("w,h", [(1001, 300), (1002, 262), (720, 540), (999, 262), (1024, 256)])
@pytest.mark.parametrize("bf16", [0, 1])
def test_host_images_of_a_megabyte_arrive_whole(gpu_ready, w, h, bf16):
    D = gpu_ready
    rng = np.random.default_rng(w + h)
    rgba = rng.integers(0, 256, (h, w, 4)).astype(np.uint8)
    t, c = rng.random((2, h, w)).astype(np.float32)
    s = D.DomainTransformSolver(D.ImageDim(w + 7, h + 3), D.FLAG_BF16_STORAGE if bf16 else 0)
    s.SetImageDim(D.ImageDim(w, h))
    s.ClearAll()
    s.InitFrame(D.COLOR_SPACE.RGB, rgba, t, c)
    r = P.bf16_round if bf16 else lambda a: a
    assert np.array_equal(s.Download(D.ImageType.TARGET), r(t))
    assert np.array_equal(s.Download(D.ImageType.CONFIDENCE), r(c))
    assert np.array_equal(s.Download(D.ImageType.COLOR_IMAGE), rgba)


# ---- a first solve under a capture: no block tables, an instance a launch -------
def test_first_solve_of_a_batch_under_a_capture(gpu_ready):
    import torch
    D = gpu_ready
    rng = np.random.default_rng(5)
    sizes = [(90, 60), (33, 140), (401, 77)]
    g = [rng.integers(0, 256, (h, w, 4)).astype(np.uint8) for w, h in sizes]
    t = [rng.normal(0, 1, (h, w)).astype(np.float32) for w, h in sizes]
    c = [rng.random((h, w)).astype(np.float32) for w, h in sizes]
    fp, op = D.DomainFilterParams(), D.DomainOptimizeParams(num_iterations=3, loss=1, sigma_z=8.0)
    ref = D.Batch(sizes)
    ref.upload(D.COLOR_SPACE.YCbCr, g, t, c)
    ref.solve_dts(fp, op)
    want = ref.download(0)
    b = D.Batch(sizes, use_graphs=False)
    stream = torch.cuda.Stream()
    b.set_stream(stream.cuda_stream)
    keep = [[torch.from_numpy(a).cuda() for a in x] for x in (g, t, c)]
    out = [torch.full((h, w), -1.0, device="cuda") for w, h in sizes]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        b.upload_device(D.COLOR_SPACE.YCbCr, *[[a.data_ptr() for a in x] for x in keep])
        b.solve_dts(fp, op)
        b.download_device(0, [o.data_ptr() for o in out])
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    for a, o in zip(want, out):
        assert np.array_equal(a, o.cpu().numpy())


# ---- block tables of a batch: per halo, for the batch's life --------------------
def _batch_on_a_stream(D, sizes, seed=5):
    """A batch without graphs of its own on a stream, its inputs on host and device."""
    import torch
    rng = np.random.default_rng(seed)
    host = ([rng.integers(0, 256, (h, w, 4)).astype(np.uint8) for w, h in sizes],
            [rng.normal(0, 1, (h, w)).astype(np.float32) for w, h in sizes],
            [rng.random((h, w)).astype(np.float32) for w, h in sizes])
    b = D.Batch(sizes, use_graphs=False)
    stream = torch.cuda.Stream()
    b.set_stream(stream.cuda_stream)
    dev = [[torch.from_numpy(a).cuda() for a in x] for x in host]
    torch.cuda.synchronize()
    return b, stream, host, dev


def _dts_op(D, sigma_z, n=3):
    return D.DomainOptimizeParams(num_iterations=n, loss=1, sigma_z=sigma_z)


@pytest.mark.parametrize("grad", [0, 1])
def test_a_callers_graph_outlives_solves_at_other_sigmas(gpu_ready, grad):
    """Captured after a solve at its own sigma, replayed after solves at more
    sigmas than the batch sets memory aside for: the same bits."""
    import torch
    D = gpu_ready
    sizes = [(90, 60), (33, 140), (401, 77)]
    b, stream, host, dev = _batch_on_a_stream(D, sizes)
    fp = D.DomainFilterParams(sigma_x=8.0, sigma_y=8.0, sigma_r=4.0)
    ptrs = [[a.data_ptr() for a in x] for x in dev]
    out = [[torch.full((h, w), -1.0, device="cuda") for w, h in sizes] for _ in range(3)]
    optr = [[o.data_ptr() for o in x] for x in out]
    b.enable_grad(bool(grad), 2)

    def work(sigma):
        b.upload_device(D.COLOR_SPACE.YCbCr, *ptrs)
        b.solve_dts(fp, _dts_op(D, sigma))
        b.download_device(0, optr[0])
        if grad:
            b.backward_device(ptrs[2], optr[1], optr[2])
    work(8.0)
    torch.cuda.synchronize()
    want = [o.cpu().numpy() for x in out for o in x]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        work(8.0)
    for sigma in (30.0, *np.linspace(1.5, 75.5, 38)):
        work(float(sigma))
    torch.cuda.synchronize()
    other = [o.cpu().numpy() for x in out for o in x]
    assert not np.array_equal(other[0], want[0])
    torch.cuda.empty_cache()
    graph.replay()
    torch.cuda.synchronize()
    for a, o in zip(want, (o for x in out for o in x)):
        assert np.array_equal(a, o.cpu().numpy())


def test_a_solve_at_a_new_sigma_waits_for_nothing(gpu_ready):
    """The first solve of a batch, and one at another sigma, behind work that
    takes a while on the batch's stream."""
    import torch
    D = gpu_ready
    sizes = [(90, 60), (33, 140), (401, 77)]
    fp = D.DomainFilterParams()
    for warm in (1, 0):  # (a kernel's first launch in the process may wait)
        b, stream, host, dev = _batch_on_a_stream(D, sizes)
        b.upload(D.COLOR_SPACE.YCbCr, *host)
        for sigma in (8.0, 30.0, 64.0, 8.0):
            if not warm:
                with torch.cuda.stream(stream):
                    torch.cuda._sleep(500_000_000)  # a quarter of a second
                    done = stream.record_event()
            b.solve_dts(fp, _dts_op(D, sigma))
            if not warm:
                assert not done.query(), sigma
            torch.cuda.synchronize()


@pytest.mark.parametrize("sizes", [[(400, 300)], [(90, 60), (333, 140)], [(700, 900)]])
def test_windows_wider_than_a_pass_stages_are_held_to_it(gpu_ready, oracle_mod, sizes):
    """A caller's graph that has kept its bounds finds another sigma's in the
    plane: the passes use those windows as far as their own sigma reaches (the
    FP64 oracle with the windows cut there, parity bar), and the adjoint stays
    in its tiles."""
    import torch
    D, O = gpu_ready, oracle_mod
    b, stream, host, dev = _batch_on_a_stream(D, sizes)
    rng = np.random.default_rng(3)
    for g, d in zip(host[0], dev[0]):  # flat blocks: windows as wide as sigma allows
        g[:] = np.kron(rng.integers(0, 256, (g.shape[0] // 50 + 1, g.shape[1] // 70 + 1, 1)),
                       np.ones((50, 70, 1)))[:g.shape[0], :g.shape[1]].astype(np.uint8)
        d.copy_(torch.from_numpy(g))
    torch.cuda.synchronize()
    fp = D.DomainFilterParams(sigma_x=8.0, sigma_y=8.0, sigma_r=4.0)
    ptrs = [[a.data_ptr() for a in x] for x in dev]
    out = [torch.full((h, w), -1.0, device="cuda") for w, h in sizes]
    gt, gc = ([torch.full((h, w), -1.0, device="cuda") for w, h in sizes] for _ in range(2))
    b.enable_grad(True, 2)
    b.upload_device(D.COLOR_SPACE.RGB, *ptrs)

    def solve(sigma):
        b.solve_dts(fp, _dts_op(D, sigma))
        b.download_device(0, [o.data_ptr() for o in out])
        b.backward_device(ptrs[2], [o.data_ptr() for o in gt], [o.data_ptr() for o in gc])
    solve(8.0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        solve(8.0)  # (the guide is unchanged: no bounds pass in it)
    solve(40.0)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    for (w, h), g, t, c, o in zip(sizes, *host, out):
        s = D.DomainTransformSolver(D.ImageDim(w, h))
        s.InitFrame(D.COLOR_SPACE.RGB, g, t, c)
        s.ComputeColorSpaceDifferential(fp)
        win = {}
        for axis in (0, 1):
            lo, hi = s.DebugBounds(axis, 40.0)
            pos = np.arange(w)[None, :] if axis == 0 else np.arange(h)[:, None]
            assert (hi - pos).max() > 8 and (pos - lo).max() > 9
            win[(axis, 8.0)] = np.maximum(lo, pos - 9), np.minimum(hi, pos + 8)
        ref, _ = O.dts_solve(g, t, c, 0, dict(sigma_x=8.0, sigma_y=8.0, sigma_r=4.0),
                             dict(num_iterations=3, loss=1, lambda_=1.0, sigma_z=8.0,
                                  step_size=0.99), overrides=win)
        assert np.abs(o.cpu().numpy() - ref).max() <= P.TOL_REL * P.target_range(t)
    assert all(torch.isfinite(x).all() for x in gt + gc)


# ---- shared memory beyond 48 KB: threads whose launches of a kernel differ -------
@pytest.mark.parametrize("kind,sizes", [
    ("hfbs", [(512, 512, 16.0), (100, 80, 16.0), (60, 50, 16.0)]),      # clusters
    ("hfbs", [(1200, 1000, 4.0), (1200, 1000, 17.0), (1200, 1000, 8.0)]),  # marches
    ("hfbs", [(512, 512, 2.0), (60, 50, 1.0), (512, 512, 3.0)]),        # splats of many levels
    ("dts", [(900, 700, 60.0), (900, 700, 100.0), (900, 700, 253.0)]),  # Y passes
])
def test_threads_with_launches_of_other_sizes(gpu_ready, kind, sizes):
    """A solver in each thread; every result is the one it has alone."""
    import threading
    D = gpu_ready
    solvers, runs = [], []
    for w, h, s in sizes:
        rng = np.random.default_rng(w)
        frame = (rng.integers(0, 256, (h, w, 4)).astype(np.uint8),
                 rng.normal(0, 1, (h, w)).astype(np.float32), rng.random((h, w)).astype(np.float32))
        if kind == "hfbs":
            v = D.HFBS(D.ImageDim(w, h), -(-w // 8), -(-h // 8), int(np.ceil(255 / s)))
            v.SetFilterParams(D.HFBSGridParams(sigma_x=8.0, sigma_y=8.0, sigma_l=s,
                                               bistoch_iter_max=2, optim_iter_max=2))
            v.InitFrame(D.COLOR_SPACE.RGB, *frame)
            runs.append(v.Optimize)
        else:
            v = D.DomainTransformSolver(D.ImageDim(w, h))
            v.InitFrame(D.COLOR_SPACE.RGB, *frame)
            v.ComputeColorSpaceDifferential(D.DomainFilterParams())
            runs.append(lambda v=v, s=s: v.Optimize(_dts_op(D, s, 10)))
        solvers.append(v)
    want, errors = [], []
    for v, run in zip(solvers, runs):
        run()
        want.append(v.Download(D.ImageType.OPTIMIZED_QUANTITY))

    def loop(run):
        try:
            for _ in range(300):
                run()
        except D.DtsgbError as e:
            errors.append(e)
    threads = [threading.Thread(target=loop, args=(r,)) for r in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for v, a in zip(solvers, want):
        assert np.array_equal(v.Download(D.ImageType.OPTIMIZED_QUANTITY), a, equal_nan=True)


# ---- splat: both forms add the same products in the same order ------------------
@pytest.mark.parametrize("w,h,sx,sy", [(102, 60, 51.0, 5.0),    # 255 pixels: a thread per cell
                                       (96, 48, 16.0, 16.0)])   # 256: a CTA per cell
@pytest.mark.parametrize("bf16", [0, 1])
def test_splat_sums_bit_for_bit(gpu_ready, w, h, sx, sy, bf16):
    """Rounded products added in row-major order of a cell's runs, each run
    first: in float32 on the host."""
    D = gpu_ready
    rng = np.random.default_rng(w + bf16)
    luma = np.repeat(rng.integers(0, 256, (h, (w + 3) // 4)), 4, axis=1)[:, :w].astype(np.uint8)
    t = rng.normal(0, 10, (h, w)).astype(np.float32)
    c = rng.random((h, w)).astype(np.float32)
    b = D.Batch([(w, h)], flags=D.FLAG_BF16_STORAGE if bf16 else 0)
    b.upload(D.COLOR_SPACE.RGB, [np.repeat(luma[..., None], 4, axis=2)], [t], [c])
    b.solve_hfbs(D.HFBSGridParams(sigma_x=sx, sigma_y=sy, sigma_l=64.0, bistoch_iter_max=1,
                                  optim_iter_max=1))
    if bf16:
        t, c = P.bf16_round(t), P.bf16_round(c)
    ct = c * t
    gx, gy, gl = round(w / sx), round(h / sy), 4
    want = np.zeros((2, gl, gy, gx), np.float32)
    for y in range(gy):
        for x in range(gx):
            at = np.s_[int(y * sy):int((y + 1) * sy), int(x * sx):int((x + 1) * sx)]
            bins = (luma[at] // 64).ravel()
            starts = np.flatnonzero(np.r_[True, bins[1:] != bins[:-1]])
            for a, e in zip(starts, np.r_[starts[1:], bins.size]):
                for k, v in enumerate((c[at].ravel(), ct[at].ravel())):
                    want[k, bins[a], y, x] += np.add.accumulate(v[a:e])[-1]
    for k in (0, 1):
        assert np.array_equal(b.debug_grid(0, 2 + k, (gx, gy, gl)), want[k])


# ---- knobs that no solve depends on --------------------------------------------
def test_a_solve_stays_differentiable_when_the_dts_knobs_change(gpu_ready):
    import test_gpu_adjoint as A
    D = gpu_ready
    rng = np.random.default_rng(8)
    data = [(rng.integers(0, 256, (40, 60, 4)).astype(np.uint8),
             *(rng.standard_normal((40, 60)).astype(np.float32) for _ in range(3)))]
    b = A._batch(D, data, dict(num_iterations=3, loss=1, lambda_=0.9, sigma_z=8.0, step_size=0.8))
    want = b.backward([data[0][3]])
    for knob, values in ((D.TUNE_DTS_TILE, (64, 32)), (D.TUNE_BOUNDS_SEGMENT, (4, 16))):
        for v in values:
            b.set_tuning(knob, v)
            got = b.backward([data[0][3]])
            assert all(np.array_equal(x[0], y[0]) for x, y in zip(got, want))


# ---- guide state that only a replay computes ------------------------------------
@pytest.mark.parametrize("solver", ["dts", "hfbs"])
def test_a_captured_solve_leaves_no_guide_state_behind(gpu_ready, solver):
    """Solved at one set of parameters, captured at another and not replayed,
    then solved at the captured one: that solve computes its own windows or
    normalisation."""
    import torch
    D = gpu_ready
    sizes = [(90, 60), (333, 140)]
    b, stream, host, dev = _batch_on_a_stream(D, sizes)
    ref = D.Batch(sizes)

    def solve(batch, k):
        if solver == "dts":
            batch.solve_dts(D.DomainFilterParams(sigma_x=8.0, sigma_y=8.0, sigma_r=4.0),
                            _dts_op(D, (30.0, 8.0)[k]))
        else:
            batch.solve_hfbs(D.HFBSGridParams(sigma_x=8.0, sigma_y=8.0, sigma_l=16.0,
                                              bistoch_iter_max=(2, 20)[k], optim_iter_max=4))
    for batch in (b, ref):
        batch.upload(D.COLOR_SPACE.YCbCr, *host)
    solve(b, 0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        solve(b, 1)
    solve(b, 1)
    solve(ref, 1)
    which = 0 if solver == "dts" else 1
    for x, y in zip(b.download(which), ref.download(which)):
        assert np.array_equal(x, y, equal_nan=True)


# ---- DTS adjoint: large gradients among small ones in a row ---------------------
@pytest.mark.parametrize("h,sz", [(60, 8.0), (60, 30.5), (60, 70.0),  # 2 and 4 rounds a segment
                                  (200, 8.0), (600, 8.0)])            # 3 and 4
def test_small_gradients_beside_large_ones_keep_their_bits(gpu_ready, oracle_mod, h, sz):
    """A gradient of 1e7 in each row, out of reach of the columns compared: the
    adjoint's bar there, relative to the largest of them (1e-4; a sum's
    conversions are within (2h + 1)^2 / 2 * 2^-30 of its largest term)."""
    import test_gpu_adjoint as A
    D = gpu_ready
    w, n = 900, 2
    rng = np.random.default_rng(int(sz))
    y, x = np.mgrid[0:h, 0:w]
    rgba = (rng.integers(0, 9, (h, w, 4)) + ((x // 23 + y // 17) % 3 * 70)[..., None]).astype(np.uint8)
    t, c, g = (rng.standard_normal((h, w)).astype(np.float32),
               rng.random((h, w)).astype(np.float32),
               rng.standard_normal((h, w)).astype(np.float32))
    reach = n * (int(sz) + 1) + int(sz) + 64
    clear = slice(20 + reach, w)
    g[:, 20] = 1e7
    opt = dict(num_iterations=n, loss=1, lambda_=0.9, sigma_z=sz, step_size=0.8)
    b = A._batch(D, [(rgba, t, c, g)], opt)
    gt, gc = b.backward([g])
    o = A._oracle(oracle_mod, rgba, t, c, A._gpu_windows(D, rgba, t, c, sz, 0))
    rt, rc = o.backward(n, 1, 0.9, sz, 0.8, g)
    for got, ref in ((gt[0], rt), (gc[0], rc)):
        got, ref = got[:, clear], ref[:, clear]
        assert 0.1 < np.abs(ref).max() < 100
        assert np.abs(got - ref).max() <= 1e-4 * np.abs(ref).max()
