"""The work that users have this framework do, as measurable cases.

A case is one call of a public entry point of ``tcoh_b200`` on a seeded
synthetic stack (``tcoh_b200.synthetic``: Voronoi regions of distributed
scatterers, exponential coherence decay, 0.5 % NULL or zero samples, samples
rounded to digital numbers, so that equal amplitudes occur):

* ``device``     Backend.run_device: prepared strips resident on the GPU;
* ``host``       Backend.run: the module's ocl_run path, page-locked host
                 buffers in and out;
* ``raw``        Backend.run_raw_device: I/Q planes on the GPU, the strip
                 preparation (and, with geometry, the flat-earth and
                 topographic phase removal) on the device;
* ``adjoint``    Backend.adjoint_raw: temporal coherence and its gradient
                 with respect to a height error and a phase screen;
* ``static``     run_device_static: the form without device allocation;
* ``module``     temporal_coherence: the module's whole strip loop over a
                 stack in host memory, context included.

``exact`` restates the path in 64-bit torch. The selection of homogeneous
pixels is defined by single-precision statistics, which it follows operation
by operation; everything after the selection is double precision.
"""

import math

import numpy as np
import torch

import tcoh_b200
import tcoh_b200.scene as scene
import tcoh_b200.synthetic as synthetic

DEFAULTS = dict(entry="device", wa=21, wr=7, test="ks", alpha=0.05, min_shp=20, estimator="evd",
                bias=False, pairs="none", geometry=False, spacing=12.0, g0_max=0.99, nregions=32)
GRID_STEP = 16  # lines and samples between the nodes of the phase grid


def listed():
    def case(name, n, rows, cols, **kw):
        return dict(DEFAULTS, name=name, n=n, rows=rows, cols=cols, **kw)

    return [
        # A test crop: what a user tries the options on; launches and their
        # latency are all of it.
        case("crop n10", 10, 48, 40, min_shp=10, g0_max=0.95, nregions=8),
        # A small image of a short stack, the first of the published
        # configurations.
        case("image n10", 10, 512, 512, min_shp=10, g0_max=0.95, nregions=8),
        # The module's default options (KS, EVD, 21 x 7) on a 30-date subset.
        case("defaults n30", 30, 250, 1000),
        # The configuration of the headline metric: an eighth of its
        # 4096 x 4096 strip.
        case("metric n30", 30, 512, 4096, test="ad", estimator="emi", bias=True),
        # The same through host buffers, in the strip that the module's
        # default memory= budget gives at 4096 columns: the drop-in call.
        case("module strip n30", 30, 188, 4096, entry="host", test="ad", estimator="emi",
             bias=True),
        # An odd number of dates, a small window, a ragged region, EMI
        # without bias correction, consecutive pair coherences.
        case("ragged n17", 17, 203, 331, wa=9, wr=5, test="ad", estimator="emi",
             pairs="consecutive", nregions=8),
        # Interferometric use: phase removed on the device from orbits and
        # an elevation map, all 435 pair coherences written.
        case("geometry pairs n30", 30, 96, 2048, entry="raw", test="tlog", pairs="all",
             geometry=True),
        # Between the two sizes of link kernels: 45 dates.
        case("ragged n45", 45, 61, 517, test="ad", bias=True, spacing=6.0),
        # The long stack with six-day dates, EVD and EMI.
        case("long n60 evd", 60, 96, 2048, entry="raw", spacing=6.0),
        case("long n60 emi", 60, 40, 1024, entry="raw", estimator="emi", spacing=6.0),
        # One step of a height-error and atmosphere inversion.
        case("adjoint n30", 30, 160, 512, entry="adjoint", test="tlog", geometry=True),
        # The whole call on a stack in host memory, with the defaults.
        case("whole call n30", 30, 200, 300, entry="module"),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    entry = rng.choice(["device"] * 8 + ["host"] * 2 + ["raw"] * 4 + ["adjoint"] * 3 +
                       ["static"] + ["module"] * 2)
    n = log_int(6, 32 if entry == "adjoint" else 64)
    c = dict(DEFAULTS, entry=entry, n=n)
    fitting = [w for w in ((21, 7), (21, 7), (21, 7), (9, 5), (7, 5), (11, 11))
               if w[0] * w[1] >= max(20, n)]
    c["wa"], c["wr"] = rng.choice(fitting)
    c["test"] = rng.choice(["ks", "ad", "tlog"])
    c["alpha"] = rng.choice([0.05, 0.05, 0.01])
    c["min_shp"] = rng.choice([10, 20])
    c["estimator"] = rng.choice(["evd", "emi"])
    c["bias"] = rng.random() < 0.4
    if entry != "adjoint":
        c["pairs"] = rng.choice(["none", "none", "consecutive", "all"])
    if entry in ("raw", "adjoint"):
        c["geometry"] = rng.random() < 0.5
    c["spacing"] = rng.choice([6.0, 12.0])
    c["g0_max"] = rng.choice([0.95, 0.99])
    c["nregions"] = rng.choice([8, 32])
    # the pixels that about a sixth of the largest listed case's work buys,
    # less for host-bound entry points and where every pair plane is kept
    most = 120e9 / (link_flops(c) + gram_flops(c))
    most = min(most, {"device": 6e5, "host": 3e5, "raw": 3e5, "adjoint": 8e4, "static": 1e5,
                      "module": 6e4}[entry])
    if n > 32 and c["estimator"] == "emi":
        most = min(most, 5e4)
    if c["pairs"] == "all":
        most = min(most, 4e8 / (4.0 * n * (n - 1) / 2))
    pixels = log_int(1500, max(2000, most))
    aspect = math.exp(rng.uniform(math.log(0.1), math.log(1.5)))
    c["rows"] = max(8, int(math.sqrt(pixels * aspect)))
    c["cols"] = max(16, pixels // c["rows"])
    return c


# ---------------------------------------------------------------------------
# Inputs.

def settings_of(c):
    return tcoh_b200.make_settings(c["n"], window=(c["wa"], c["wr"]), shp_test=c["test"],
                                   alpha=c["alpha"], min_shp=c["min_shp"],
                                   estimator=c["estimator"], bias=c["bias"],
                                   pairs=c["pairs"] != "none", pairs_all=c["pairs"] == "all")


def grid_phase(grid, levels, h, row0):
    """Phases (N, rows, cols) of the grid (float64 tensor [gr][gc][levels][N])
    at heights h of region rows row0 ..: bilinear in position, quadratic in
    height; rows outside the grid take its first or last row."""
    rows, cols = h.shape
    dev = h.device
    rr = (torch.arange(rows, device=dev) + row0).clamp(0, (grid.shape[0] - 1) * GRID_STEP - 1)
    cc = torch.arange(cols, device=dev)
    gr, gc = rr // GRID_STEP, cc // GRID_STEP
    fr = ((rr - gr * GRID_STEP).double() / GRID_STEP)[:, None, None]
    fc = ((cc - gc * GRID_STEP).double() / GRID_STEP)[None, :, None]
    if len(levels) == 3:
        a, b, d = levels
        weights = [(h - b) * (h - d) / ((a - b) * (a - d)), (h - a) * (h - d) / ((b - a) * (b - d)),
                   (h - a) * (h - b) / ((d - a) * (d - b))]
    else:
        weights = [torch.ones_like(h)]
    out = 0.0
    for k, wk in enumerate(weights):
        g = grid[:, :, k]
        v = ((1 - fr) * ((1 - fc) * g[gr][:, gc] + fc * g[gr][:, gc + 1]) +
             fr * ((1 - fc) * g[gr + 1][:, gc] + fc * g[gr + 1][:, gc + 1]))
        out = out + wk[:, :, None] * v
    return out.permute(2, 0, 1)


def acquisition(c, seed):
    """Geometry, its phase grid and heights of a case with geometry."""
    rows, cols = c["rows"], c["cols"]
    geo, orbits = scene.acquisition(c["n"], rows, cols, seed=seed + 1)
    heights = scene.fbm_heights(rows, cols, hurst=0.8, hmax=2000.0, seed=seed + 2)
    g = tcoh_b200.make_geometry(heights=heights, h0=0.0, **geo)
    grid = tcoh_b200.geometry_grid(g, orbits)
    levels = [g.hmin, 0.5 * (g.hmin + g.hmax), g.hmax][:grid.shape[2]]
    return dict(geometry=g, grid=grid, levels=levels, heights=heights)


def inputs(c, seed):
    """The stack of a case on the GPU, and its acquisition if it has one."""
    n, rows, cols = c["n"], c["rows"], c["cols"]
    stack = synthetic.generate(n, rows, cols, nregions=c["nregions"], g0_max=c["g0_max"],
                               spacing=c["spacing"], seed=seed, device=torch.device("cuda"))
    acq = None
    if c["geometry"]:
        acq = acquisition(c, seed)
        grid, h = torch.from_numpy(acq["grid"]).cuda(), torch.from_numpy(acq["heights"]).cuda()
        for r in range(0, rows, 64):
            phi = grid_phase(grid, acq["levels"], h[r:r + 64], r)
            stack[:, r:r + 64] *= torch.polar(torch.ones_like(phi), -phi).to(torch.complex64)
    return stack, acq


def raw_planes(c, stack):
    """I/Q planes (N, padded rows, cols), NULL outside the region."""
    ha = c["wa"] // 2
    re = torch.full((c["n"], c["rows"] + 2 * ha, c["cols"]), float("nan"), device=stack.device)
    im = torch.full_like(re, float("nan"))
    re[:, ha:ha + c["rows"]] = stack.real
    im[:, ha:ha + c["rows"]] = stack.imag
    return re, im


def padded_heights(c, acq):
    e = np.full((c["rows"] + 2 * (c["wa"] // 2), c["cols"]), np.nan)
    e[c["wa"] // 2:c["wa"] // 2 + c["rows"]] = acq["heights"]
    return e


def strip(c, stack):
    """Padded strip: samples (P, W, N, 2), sorted amplitudes (P, W, N) and
    validity (P, W)."""
    n, rows, cols = stack.shape
    ha, hr = c["wa"] // 2, c["wr"] // 2
    re, im = stack.real, stack.imag
    ok = ~(torch.isnan(re) | torch.isnan(im) | ((re == 0) & (im == 0))).any(dim=0)
    zero = torch.zeros((), device=stack.device)
    re, im = torch.where(ok[None], re, zero), torch.where(ok[None], im, zero)
    inner = (slice(ha, ha + rows), slice(hr, hr + cols))
    slc = torch.zeros((rows + 2 * ha, cols + 2 * hr, n, 2), device=stack.device)
    amp = torch.zeros((rows + 2 * ha, cols + 2 * hr, n), device=stack.device)
    valid = torch.zeros((rows + 2 * ha, cols + 2 * hr), dtype=torch.uint8, device=stack.device)
    slc[inner][..., 0] = re.permute(1, 2, 0)
    slc[inner][..., 1] = im.permute(1, 2, 0)
    amp[inner] = torch.sqrt(re * re + im * im).sort(dim=0)[0].permute(1, 2, 0)
    valid[inner] = ok.to(torch.uint8)
    return slc, amp, valid


def perturbation(c, seed):
    """A smooth height error (15 m RMS) and a phase screen (0 - 2 rad)."""
    rng = np.random.default_rng(seed + 3)
    prow, cols = c["rows"] + 2 * (c["wa"] // 2), c["cols"]
    dh = scene.smooth(rng.normal(0.0, 15.0, (prow, cols)), 9)
    dh *= 15.0 / dh.std()
    psi = np.stack([scene.fbm_heights(prow, cols, hurst=0.8, hmax=2.0, seed=seed + 10 + k)
                    for k in range(c["n"])]).astype(np.float32)
    return dh, psi


def pinned(a):
    """A page-locked host copy, as numpy."""
    t = torch.as_tensor(a)
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy()


def prepare(case, seed):
    c = case
    n, rows, cols, entry = c["n"], c["rows"], c["cols"], c["entry"]
    stack, acq = inputs(c, seed)
    s = settings_of(c)
    state = dict(case=c, settings=s)
    if entry == "module":
        state["stack"] = stack.cpu().numpy()
        return state
    if entry != "static":
        state["backend"] = tcoh_b200.Backend(s, cols + c["wr"] - 1, device=0)
        if acq:
            state["backend"].set_geometry(acq["geometry"], acq["grid"])
    if entry in ("device", "host", "static"):
        state["strip"] = strip(c, stack)
        if entry == "host":
            state["strip"] = [pinned(a) for a in state["strip"]]
    else:
        state["planes"] = raw_planes(c, stack)
        elev = padded_heights(c, acq) if acq else None
        state["elev"] = torch.from_numpy(elev).cuda() if acq else None
        if entry == "adjoint":
            state["planes"] = [pinned(a) for a in state["planes"]]
            state["elev"] = pinned(elev) if acq else None
            dh, psi = perturbation(c, seed)
            state["dh"], state["psi"] = pinned(dh) if acq else None, pinned(psi)
    prow = rows + c["wa"] - 1
    shapes = {"coh": ((rows, cols), torch.float32), "count": ((rows, cols), torch.int32)}
    if s.npairs:
        shapes["pairs"] = ((s.npairs, rows, cols), torch.float32)
    if entry == "adjoint":
        shapes["grad_dh"] = ((prow, cols), torch.float32)
        shapes["grad_psi"] = ((n, prow, cols), torch.float32)
    on_host = entry in ("host", "adjoint")
    out = {k: torch.zeros(shape, dtype=dtype, device="cpu" if on_host else "cuda",
                          pin_memory=on_host) for k, (shape, dtype) in shapes.items()}
    state["out"] = {k: v.numpy() for k, v in out.items()} if on_host else out
    return state


def run(state):
    c, out = state["case"], state.get("out")
    rows, cols, entry, ha = c["rows"], c["cols"], c["entry"], c["wa"] // 2
    if entry == "device":
        state["backend"].run_device(*state["strip"], rows, cols, out["coh"], out["count"],
                                    out.get("pairs"), stream=torch.cuda.current_stream())
        return out
    if entry == "static":
        tcoh_b200.run_device_static(state["settings"], cols + c["wr"] - 1, *state["strip"], rows,
                                    cols, out["coh"], out["count"], out.get("pairs"),
                                    stream=torch.cuda.current_stream())
        return out
    if entry == "raw":
        state["backend"].run_raw_device(*state["planes"], state["elev"], -ha, rows, rows, cols,
                                        out["coh"], out["count"], out.get("pairs"),
                                        stream=torch.cuda.current_stream())
        return out
    if entry == "host":
        return state["backend"].run(*state["strip"], rows, cols, out=out)
    if entry == "adjoint":
        return state["backend"].adjoint_raw(*state["planes"], state["elev"], state["dh"],
                                            state["psi"], -ha, rows, rows, cols, out=out)
    r = tcoh_b200.temporal_coherence(state["stack"], window=(c["wa"], c["wr"]),
                                     shp_test=c["test"], alpha=c["alpha"], min_shp=c["min_shp"],
                                     estimator=c["estimator"], bias_correction=c["bias"],
                                     pairs=c["pairs"] != "none",
                                     pairs_mode="all" if c["pairs"] == "all" else "consecutive")
    return {k: r[k] for k in ("coh", "count", "pairs") if k in r}


# ---------------------------------------------------------------------------
# Work of one pass.

def gram_flops(c):
    """Masked Gram per pixel, with seven candidates in ten selected."""
    n = c["n"]
    return 8.0 * 0.7 * c["wa"] * c["wr"] * n * (n + 1) / 2


def link_flops(c):
    """Normalisation, eigenvector (and inverse), goodness of fit per pixel."""
    n = c["n"]
    f = 15.0 * n * (n - 1) + 16.0 * n ** 3 / 3 + 8.0 * n * n + 320.0 * n
    return f + (n ** 3 + 2.0 * n * n if c["estimator"] == "emi" else 0.0)


def shp_flops(c):
    n, area = c["n"], c["wa"] * c["wr"]
    return area * {"ks": 2.0 * n, "ad": 7.0 * (2 * n - 1), "tlog": 6.0}[c["test"]]


def work(case):
    c = case
    n, rows, cols = c["n"], c["rows"], c["cols"]
    pixels, prow = rows * cols, rows + c["wa"] - 1
    npairs = {"none": 0, "consecutive": n - 1, "all": n * (n - 1) // 2}[c["pairs"]]
    out = pixels * 4 * (2 + npairs)
    per_pixel = shp_flops(c) + gram_flops(c) + link_flops(c)
    if c["entry"] in ("device", "host", "static"):
        inp = prow * (cols + c["wr"] - 1) * (12 * n + 1)
    elif c["entry"] == "module":
        inp = pixels * 8 * n
    else:
        inp = prow * cols * (8 * n + (8 if c["geometry"] else 0))
    if c["entry"] == "adjoint":
        inp += prow * cols * (4 * n + (8 if c["geometry"] else 0))
        out += prow * cols * 4 * (n + 1)
        per_pixel += gram_flops(c) + link_flops(c)  # the backward of both
    return {"bytes": float(inp + out), "flops": float(pixels * per_pixel)}


# ---------------------------------------------------------------------------
# The result in 64 bits.

def tlog_stats(amp, n):
    """Mean and variance of the log amplitudes, float32, summed in order."""
    logs = torch.log(amp.double()).float()
    mean = torch.zeros_like(logs[..., 0])
    for k in range(n):
        mean = mean + logs[..., k]
    mean = mean / torch.full_like(mean, n)
    var = torch.zeros_like(mean)
    for k in range(n):
        d = logs[..., k] - mean
        var = var + d * d
    return mean, var / torch.full_like(var, n - 1)


def homogeneous(s, a, b):
    """KS or AD decision of centre series a against candidates b (B, N), both
    sorted; equal values take the centre's first."""
    n = s.ndates
    before_a = torch.searchsorted(b, a)  # b's below each a
    before_b = torch.searchsorted(a, b, right=True)  # a's not above each b
    i = torch.arange(n, device=a.device)
    if s.test == 0:
        d = torch.maximum((i + 1 - before_a).abs().amax(1), (before_b - i - 1).abs().amax(1))
        return d <= s.ks_max
    step = torch.zeros((a.shape[0], 2 * n), dtype=torch.int32, device=a.device)
    step.scatter_(1, before_a + i, 1)
    m = step.cumsum(1)[:, :-1].to(torch.int32)
    j = torch.arange(1, 2 * n, device=a.device, dtype=torch.int32)
    num = (2 * n * m - j * n).float()
    q = num * num / (j * (2 * n - j)).float()
    t = torch.zeros_like(q[:, 0])
    for k in range(2 * n - 1):
        t = t + q[:, k]
    f = [float(np.float32("%.9e" % v)) for v in (s.ad_norm, s.ad_sigma, s.ad_crit)]
    one = torch.ones_like(t)
    return (t * (one * f[0]) - 1.0) / (one * f[1]) <= one * f[2]


def selection(c, s, amp, valid, r0, r1):
    """SHP mask (B, window) of output rows r0 .. r1 - 1, and the centres'
    validity."""
    wa, wr, cols, n = c["wa"], c["wr"], c["cols"], c["n"]
    ha, hr = wa // 2, wr // 2

    def at(x, dy, dx):
        return x[r0 + dy:r1 + dy, dx:dx + cols].reshape((r1 - r0) * cols, *x.shape[2:])

    centre, ok = at(amp, ha, hr).contiguous(), at(valid, ha, hr).bool()
    if s.test == 2:
        mean, var = tlog_stats(torch.where(amp > 0, amp, torch.ones_like(amp)), n)
        crit = torch.full((1,), float(np.float32("%.9e" % s.tlog_crit)), device=amp.device)
    keep = torch.empty((centre.shape[0], wa * wr), dtype=torch.bool, device=amp.device)
    for dy in range(wa):
        for dx in range(wr):
            if s.test == 2:
                se = torch.sqrt((at(var, ha, hr) + at(var, dy, dx)) /
                                torch.full_like(crit, float(n)))
                t = (at(mean, ha, hr) - at(mean, dy, dx)).abs() / se
                h = ~(se > 0) | (t <= crit)
            else:
                h = homogeneous(s, centre, at(amp, dy, dx).contiguous())
            keep[:, dy * wr + dx] = h & at(valid, dy, dx).bool() & ok
    return keep, ok


def coherence_matrix(keep, samples, bias):
    """T (B, N, N) of the kept samples (B, window, N), complex128."""
    x = samples * keep[:, :, None]
    cov = x.transpose(1, 2) @ x.conj()
    looks = keep.sum(1).double()
    d = torch.sqrt(cov.diagonal(dim1=1, dim2=2).real)
    dd = d[:, :, None] * d[:, None, :]
    t = torch.where(dd > 0, cov / torch.where(dd > 0, dd, 1.0), 0.0)
    if bias:
        m2 = t.real ** 2 + t.imag ** 2
        lk = looks[:, None, None]
        m2c = (lk * m2 - 1.0) / torch.where(lk > 1, lk - 1.0, 1.0)
        up = (m2 > 0) & (m2c > 0)
        f = torch.where(up, torch.sqrt(torch.where(up, m2c, 1.0) / torch.where(up, m2, 1.0)), 0.0)
        t = torch.where(lk > 1, t * f, t)
    eye = torch.eye(t.shape[1], dtype=torch.float64, device=t.device)
    return t * (1.0 - eye) + eye


def goodness(t, estimator):
    """Temporal coherence (B) of the matrices t, batches that the batched
    eigensolver takes at a time."""
    return torch.cat([goodness_batch(p, estimator) for p in t.split(8192)])


def dominant(h):
    """Eigenvector (B, N) of the largest eigenvalue of each Hermitian matrix.
    Above 32 dates, where the library solves one matrix at a time, by
    repeated squaring of the matrix shifted to be positive."""
    n = h.shape[1]
    if n <= 32:
        return torch.linalg.eigh(h)[1][:, :, -1]
    norm = torch.linalg.matrix_norm(h)[:, None, None]
    h = h / norm + torch.eye(n, dtype=h.dtype, device=h.device)
    for _ in range(36):
        h = h @ h
        h = h / torch.linalg.matrix_norm(h)[:, None, None]
    best = h.diagonal(dim1=1, dim2=2).real.argmax(1)
    return h.gather(2, best[:, None, None].expand(-1, n, 1))[:, :, 0]


def goodness_batch(t, estimator):
    n = t.shape[1]
    if estimator == "emi":
        m = t.abs()
        inv = torch.linalg.inv_ex(m)[0]
        poor = ~(n * inv.abs().amax((1, 2)) < 1e8)
        if poor.any():
            w, v = torch.linalg.eigh(m[poor])
            w = torch.where(w.abs() >= 1e-9, 1.0 / w, 0.0)
            inv[poor] = (v * w[:, None, :]) @ v.transpose(1, 2)
        u = dominant(-0.5 * (inv + inv.transpose(1, 2)) * t)
    else:
        u = dominant(t)
    mag = u.abs().detach()
    floor = 1e-3 * mag.amax(1, keepdim=True)
    ref = torch.where(mag[:, n // 2] <= floor[:, 0], mag.argmax(1), n // 2)
    rel = u * u.gather(1, ref[:, None]).conj()
    big = mag > floor
    e = torch.where(big, rel / torch.where(big, rel, 1.0).abs(), 1.0)
    some = (t != 0).detach()
    w = torch.where(some, t / torch.where(some, t, 1.0).abs(), 1.0)
    i, j = torch.triu_indices(n, n, 1, device=t.device)
    return (w[:, i, j] * e[:, i].conj() * e[:, j]).sum(1).abs() / (0.5 * n * (n - 1))


def linked(t):
    """Whether the non-zero entries of each matrix connect all dates."""
    reach = (t != 0).double()
    for _ in range(t.shape[1].bit_length()):
        reach = (reach @ reach > 0).double()
    return reach[:, 0].min(1)[0] > 0


def windows(c, x, r0, r1):
    """Samples (B, window, N) of the windows of output rows r0 .. r1 - 1."""
    v = x[r0:r1 + c["wa"] - 1].unfold(0, c["wa"], 1).unfold(1, c["wr"], 1)
    return v.permute(0, 1, 3, 4, 2).reshape((r1 - r0) * c["cols"], c["wa"] * c["wr"], c["n"])


def exact(case, seed):
    c = case
    n, rows, cols, entry = c["n"], c["rows"], c["cols"], c["entry"]
    adjoint = entry == "adjoint"
    # more is over about 20 seconds of batched eigenvectors or their backward
    if rows * cols * n ** 3 > (4.0e9 if adjoint else 6.0e10):
        return None
    stack, acq = inputs(c, seed)
    s = settings_of(c)
    slc, amp, valid = strip(c, stack)
    x = torch.complex(slc[..., 0].double(), slc[..., 1].double())
    ha, hr = c["wa"] // 2, c["wr"] // 2
    prow = rows + 2 * ha
    theta = dh = psi = None
    if acq or adjoint:
        theta = torch.zeros((n, prow, cols), dtype=torch.float64, device=x.device)
        h = None
        if acq:
            h = torch.from_numpy(padded_heights(c, acq)).cuda().nan_to_num()
        if adjoint:
            dh, psi = (torch.from_numpy(a.astype(np.float64)).cuda() for a in perturbation(c, seed))
            psi.requires_grad_()
            dh.requires_grad_()
            theta = theta + psi
            h = h + dh if acq else None
        if acq:
            theta = theta + grid_phase(torch.from_numpy(acq["grid"]).cuda(), acq["levels"], h, -ha)
    rotation = theta
    if adjoint:  # the chain up to the samples once, after the windows
        rotation = theta.detach().clone().requires_grad_()
    coh = torch.full((rows * cols,), float("nan"), dtype=torch.float64, device=x.device)
    pairs = None
    if s.npairs:
        pairs = torch.full((s.npairs, rows * cols), float("nan"), dtype=torch.float64,
                           device=x.device)
        i, j = (torch.triu_indices(n, n, 1, device=x.device) if s.pairs_all else
                torch.stack([torch.arange(n - 1), torch.arange(1, n)]).to(x.device))
    per = max(1, int((0.5e9 if adjoint else 1.5e9) / (cols * c["wa"] * c["wr"] * n * 16)))
    for r0 in range(0, rows, per):
        r1 = min(rows, r0 + per)
        keep, ok = selection(c, s, amp, valid, r0, r1)
        use = ok & (keep.sum(1) >= s.min_looks)
        if not use.any():
            continue
        with torch.set_grad_enabled(adjoint):
            a = x[r0:r1 + 2 * ha]
            if rotation is not None:
                phi = rotation[:, r0:r1 + 2 * ha].permute(1, 2, 0)
                a = a * torch.nn.functional.pad(torch.polar(torch.ones_like(phi), phi),
                                                (0, 0, hr, hr))
            t = coherence_matrix(keep[use], windows(c, a, 0, r1 - r0)[use], c["bias"])
            at = use.nonzero()[:, 0] + r0 * cols
            if pairs is not None:
                pairs[:, at] = t[:, i, j].abs().T
            if c["bias"]:
                link = linked(t.detach())
                t, at = t[link], at[link]
            if not len(at):
                continue
            g = goodness(t, c["estimator"])
            coh[at] = g.detach()
            if adjoint:
                g.sum().backward()
    out = {"coh": coh.reshape(rows, cols), "count": None}
    if pairs is not None:
        out["pairs"] = pairs.reshape(-1, rows, cols)
    if adjoint:
        theta.backward(rotation.grad)
        out["grad_psi"] = psi.grad
        out["grad_dh"] = dh.grad if acq else torch.zeros_like(dh)
    return out
