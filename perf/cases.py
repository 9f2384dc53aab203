"""The imaging work this library is timed on.

Each case is one call (or one call sequence) a program makes through the public
entry points: imaging a dataset with a plan, the three plan stages one by one,
a batch of snapshots, a burst of served requests, or the reference's own call
sequence on host arrays.  Observations are seeded Earth-rotation tracks of the
array layouts in ``rick_b200.synth`` with a few point sources, receiver noise,
unequal weights and some flagged (NaN) samples, made on the GPU.

The mixed form computes in FP32 and is used for its speed where FP32 accuracy is
enough; programs that ask for it keep FP32 images, so those cases end with the
conversion.  The plain form's images stay FP64.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import rick_b200 as R
from rick_b200 import synth

C_LIGHT = 299_792_458.0
PI = 3.14159265359  # the truncated pi of the imaging definition


def _image(name, call, precision, layout, n_ant, extent_m, lat, dec, hours, rows, nchan, npol,
           f_lo, f_hi, grid, planes, kernel, support, w_first=0, w_count=0):
    return dict(name=name, call=call, precision=precision, layout=layout, n_ant=n_ant,
                extent_m=extent_m, lat=lat, dec=dec, hours=hours, rows=rows, nchan=nchan,
                npol=npol, f_lo=f_lo, f_hi=f_hi, grid=grid, planes=planes, kernel=kernel,
                support=support, w_first=w_first, w_count=w_count)


def listed():
    return [
        # A quick look at one short scan on a small grid: the call is all
        # launches and host work.
        _image("quicklook_fp64", "image", "fp64", "compact", 43, 500.0, -23.0, -20.0, 0.004, 5418,
               1, 2, 99.5e9, 100.5e9, 128, 4, "gauss", 7),
        # One compact-array snapshot in the mixed form (the size of a snapshot
        # survey's ordinary job; odd row count).
        _image("snapshot_mixed", "image", "mixed", "compact", 43, 500.0, -23.0, -35.0, 0.15,
               243_811, 2, 2, 99.5e9, 100.5e9, 1024, 8, "kaiser_bessel", 7),
        # The small plain FP64 image: a 40-antenna disc array, 1 h.
        _image("disc_fp64", "image", "fp64", "disc", 40, 3000.0, 45.0, 45.0, 1.0, 279_800, 8, 2,
               120e6, 128e6, 512, 8, "gauss", 7),
        # A grid whose axes are not powers of two, with sample counts per row
        # that are not multiples of four (3 polarisation products kept).
        _image("ragged_fp64", "image", "fp64", "disc", 40, 12000.0, 45.0, 30.0, 2.0, 400_003, 5, 3,
               120e6, 128e6, 1500, 12, "kaiser_bessel", 7),
        # Grid, transform and correct as separate calls (a program that looks at
        # or changes the cube in between).
        _image("stages_fp64", "stages", "fp64", "yarms", 27, 10000.0, 34.1, 40.0, 2.0, 300_001, 8,
               2, 1.0e9, 1.2e9, 2048, 8, "kaiser_bessel", 7),
        # The LOFAR-like large single image, FP64 and mixed.
        _image("lofar_fp64", "image", "fp64", "lograd", 60, 40000.0, 52.9, 50.0, 4.0, 5_096_600,
               64, 4, 130e6, 142e6, 4096, 32, "kaiser_bessel", 7),
        _image("lofar_mixed", "image", "mixed", "lograd", 60, 40000.0, 52.9, 50.0, 4.0, 5_096_600,
               64, 4, 130e6, 142e6, 4096, 32, "kaiser_bessel", 7),
        # The JVLA-like wide field: one w-plane shard of the 64-plane job (what
        # each of four GPUs does) in FP64, and a 32-plane job in the mixed form.
        _image("wide_shard_fp64", "image", "fp64", "yarms", 27, 21000.0, 34.1, 10.0, 6.0,
               3_789_800, 16, 2, 1.0e9, 1.5e9, 8192, 64, "gauss_hi", 9, 24, 16),
        _image("wide_mixed", "image", "mixed", "yarms", 27, 21000.0, 34.1, 10.0, 6.0, 3_789_800,
               16, 2, 1.0e9, 1.5e9, 8192, 32, "gauss_hi", 9),
        # Snapshots of uneven sizes (256^2 to 2048^2, 4 to 16 planes) in one
        # CUDA graph.
        dict(name="batch_mixed", call="batch", precision="mixed", jobs=64, mix=4242,
             vis_lo=1e4, vis_hi=1e7),
        # A burst of requests to a running server: submitted at once, waited for.
        dict(name="served_mixed", call="served", precision="mixed", jobs=24, mix=977,
             vis_lo=1e4, vis_hi=2e6),
        # The reference's call sequence on host arrays (wstack, FFT, phase
        # correction), as its own host code makes it.
        _image("dropin_fp64", "dropin", "fp64", "disc", 40, 6000.0, 45.0, 45.0, 0.25, 70_200, 8,
               2, 120e6, 128e6, 512, 8, "kaiser_bessel", 7),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["image", "stages", "batch", "served", "dropin"], [12, 2, 2, 1, 1])[0]
    if kind in ("batch", "served"):
        return dict(call=kind, precision=rng.choice(["mixed", "mixed", "fp64"]) if kind == "batch"
                    else "mixed", jobs=rng.randint(5, 48), mix=rng.randrange(1 << 20),
                    vis_lo=1e4, vis_hi=4e6)
    precision = rng.choice(["fp64", "mixed"]) if kind != "dropin" else "fp64"
    if kind == "dropin":
        grid, cells = _log_int(rng, 64, 1024), 4e6
    elif rng.random() < 0.7:  # power-of-two axes
        grid, cells = 1 << rng.randint(6, 13), 5.4e8
    else:
        grid, cells = _log_int(rng, 48, 3000), 5e7
    planes = _log_int(rng, 1, max(1, min(64, int(cells / grid ** 2))))
    nchan, npol = _log_int(rng, 1, 64), rng.choice([1, 2, 2, 4, 4])
    most = min(5e6, 1.2e9 / (nchan * npol)) if kind != "dropin" else 2e5
    rows = _log_int(rng, 1e3, most)
    layout = rng.choice(["compact", "disc", "lograd", "yarms"])
    n_ant = rng.randint(20, 60) if layout != "yarms" else 27
    f_lo = rng.choice([120e6, 1.0e9])
    w_first = w_count = 0
    if kind == "image" and planes >= 4 and rng.random() < 0.15:
        w_count = planes // rng.choice([2, 4])
        w_first = rng.randint(0, planes - w_count)
    # an array large enough for its grid: the imaged field stays inside the horizon
    extent = grid * C_LIGHT / f_lo * math.exp(rng.uniform(math.log(4), math.log(40)))
    c = _image("", kind, precision, layout, n_ant, extent, rng.uniform(-40, 55),
               rng.uniform(-30, 60), rng.uniform(0.05, 6.0), rows, nchan, npol, f_lo, f_lo * 1.1,
               grid, planes,
               rng.choice(["kaiser_bessel", "kaiser_bessel", "gauss", "gauss_hi"]),
               rng.choice([3, 5, 7, 7, 7, 9, 9, 11, 15]), w_first, w_count)
    del c["name"]
    return c


# ---- observations -------------------------------------------------------------

def _observation(c, seed):
    """Rows of one dataset on the GPU: (uu, vv, ww, weights, vis_re, vis_im), and
    the resolution and w range its meta file would carry."""
    rng = np.random.default_rng(seed)
    cfg = synth.ObsConfig("perf", c["layout"], c["n_ant"], c["extent_m"], c["lat"], c["dec"], 1.0,
                          1.0, c["nchan"], c["f_lo"], c["f_hi"], c["npol"], 4, "lognormal", 1.0,
                          0.3, c["grid"], c["planes"], c["kernel"], c["support"])
    enu = synth.antenna_enu(cfg, rng)
    lat, dec = math.radians(c["lat"]), math.radians(c["dec"])
    x = -math.sin(lat) * enu[:, 1]
    y = enu[:, 0]
    z = math.cos(lat) * enu[:, 1]
    a1, a2 = np.triu_indices(c["n_ant"], k=1)
    dev = torch.device("cuda")
    lam0 = C_LIGHT / (0.5 * (c["f_lo"] + c["f_hi"]))
    bx, by, bz = (torch.tensor((q[a2] - q[a1]) / lam0, device=dev) for q in (x, y, z))
    n, nchan, npol = c["rows"], c["nchan"], c["npol"]
    nt = -(-n // len(a1))
    h = (torch.arange(nt, dtype=torch.float64, device=dev) + 0.5) / nt - 0.5
    h = h * (c["hours"] * 3600.0 * 2 * math.pi / 86164.0905)
    sh, ch = torch.sin(h)[:, None], torch.cos(h)[:, None]
    sd, cd = math.sin(dec), math.cos(dec)
    u = (sh * bx + ch * by).reshape(-1)[:n].contiguous()
    v = (-sd * ch * bx + sd * sh * by + cd * bz).reshape(-1)[:n].contiguous()
    w = (cd * ch * bx - cd * sh * by + sd * bz).reshape(-1)[:n].contiguous()
    umax, vmax = float(u.abs().max()), float(v.abs().max())
    wmin, wmax = float(w.min()), float(w.max())
    maxg = max(umax, vmax)
    ming = min(float(u.min()), float(v.min()))
    src = 0.3 / maxg * c["grid"] * (rng.random((2, 4)) - 0.5)  # inside the imaged field
    src = np.clip(src, -0.3, 0.3)
    flux = rng.lognormal(0.0, 1.0, 4)
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    scale = torch.tensor((c["f_lo"] + (c["f_hi"] - c["f_lo"]) * (np.arange(nchan) + 0.5) / nchan) /
                         (0.5 * (c["f_lo"] + c["f_hi"])), device=dev)
    stokes_i = torch.tensor([1.0, 0.0, 0.0, 1.0][:npol] if npol == 4 else [1.0] * npol, device=dev)
    re = torch.empty((n, nchan, npol), dtype=torch.float32, device=dev)
    im = torch.empty_like(re)
    step = max(1, (1 << 24) // (nchan * npol))
    for r0 in range(0, n, step):
        r1 = min(n, r0 + step)
        vr = torch.zeros((r1 - r0, nchan), dtype=torch.float32, device=dev)
        vi = torch.zeros_like(vr)
        for s in range(4):
            l, m = float(src[0, s]), float(src[1, s])
            ph = l * u[r0:r1] + m * v[r0:r1] + (math.sqrt(1 - l * l - m * m) - 1) * w[r0:r1]
            ph = ph[:, None] * scale
            ph = ((ph - torch.floor(ph)) * (-2 * math.pi)).float()
            vr += float(flux[s]) * torch.cos(ph)
            vi += float(flux[s]) * torch.sin(ph)
        shape = (r1 - r0, nchan, npol)
        re[r0:r1] = vr[:, :, None] * stokes_i
        im[r0:r1] = vi[:, :, None] * stokes_i
        re[r0:r1] += 0.3 * torch.randn(shape, generator=gen, device=dev)
        im[r0:r1] += 0.3 * torch.randn(shape, generator=gen, device=dev)
        flagged = torch.rand(shape, generator=gen, device=dev) < 0.002
        re[r0:r1].masked_fill_(flagged, float("nan"))
    wt = torch.rand(n * npol, generator=gen, device=dev) + 0.5
    rows = ((u + maxg) / (2 * maxg), (v + maxg) / (2 * maxg), (w - wmin) / (wmax - wmin), wt,
            re.reshape(-1), im.reshape(-1))
    return rows, 1.0 / max(abs(ming), maxg), wmin, wmax


def _snapshots(c):
    """The jobs of a batch or burst: their sizes follow from the case alone."""
    rng = random.Random(c["mix"])
    for _ in range(c["jobs"]):
        nchan = rng.randint(1, 4)
        rows = max(903, int(math.exp(rng.uniform(math.log(c["vis_lo"]), math.log(c["vis_hi"]))) /
                            (2 * nchan)))
        yield _image("", "image", c["precision"], "compact", 43, 500.0, -23.0,
                     rng.uniform(-60.0, 20.0), max(rows / 903 * 2.0 / 3600.0, 0.001), rows, nchan, 2,
                     99.5e9, 100.5e9, rng.choice([256, 512, 1024, 2048]), rng.randint(4, 16),
                     "kaiser_bessel", 7)


def _geometry(c):
    return R.Geometry(c["grid"], c["grid"], c["planes"], c["support"], c["kernel"],
                      c["precision"])


def prepare(case, seed):
    c = case
    if c["call"] in ("batch", "served"):
        sizes = list(_snapshots(c))
        images = torch.empty(sum(2 * j["grid"] ** 2 for j in sizes), dtype=torch.float64,
                             device="cuda")
        jobs, at = [], 0
        for k, j in enumerate(sizes):
            rows, res, wmin, wmax = _observation(j, seed * 1000 + k)
            plane = j["grid"] ** 2
            jobs.append(R.Job(_geometry(j), j["rows"], j["nchan"], j["npol"], rows, res, wmin, wmax,
                              images[at: at + plane], images[at + plane: at + 2 * plane]))
            at += 2 * plane
        torch.cuda.synchronize()
        s = dict(case=c, jobs=jobs, images=images)
        if c["call"] == "batch":
            s["batch"] = R.Batch(jobs, c["precision"])
        else:
            s["server"] = R.Server(c["precision"], hbm_budget=24 * 10**9, max_batch_jobs=64,
                                   streams=3)
        return s
    rows, res, wmin, wmax = _observation(c, seed)
    s = dict(case=c, res=res, wmin=wmin, wmax=wmax)
    n, plane = c["rows"], c["grid"] ** 2
    if c["call"] == "dropin":
        s["rows"] = [t.cpu().numpy() for t in rows]
        s["grid"] = np.zeros(2 * c["planes"] * plane)
        s["gridss"] = np.zeros(2 * c["planes"] * plane)
        s["image"] = np.zeros((2, plane))
        return s
    planes = (c["w_first"], c["w_count"]) if c["w_count"] else None
    s["rows"] = rows
    s["image"] = torch.empty((2, c["grid"], c["grid"]), dtype=torch.float64, device="cuda")
    s["plan"] = R.Plan(_geometry(c), n, c["nchan"], c["npol"], planes=planes)
    torch.cuda.synchronize()
    return s


def run(state):
    s, c = state, state["case"]
    st = torch.cuda.current_stream()
    if c["call"] == "image":
        s["plan"].image(c["rows"], s["rows"], s["res"], s["wmin"], s["wmax"], s["image"][0],
                        s["image"][1], stream=st)
    elif c["call"] == "stages":
        s["plan"].grid(c["rows"], s["rows"], R.ROWS_SECTOR0, stream=st)
        s["plan"].fft(stream=st)
        s["plan"].phase(s["res"], s["wmin"], s["wmax"], s["image"][0], s["image"][1], stream=st)
    elif c["call"] == "batch":
        s["batch"].run(stream=st)
    elif c["call"] == "served":
        tickets = [s["server"].submit(j) for j in s["jobs"]]
        for t in tickets:
            s["server"].wait(t)
    else:
        n, g, nw = c["rows"], c["grid"], c["planes"]
        uu, vv, ww, wt, re, im = s["rows"]
        R.set_kernel(c["kernel"])
        s["grid"].fill(0.0)   # wstack and phase_correction add into their outputs
        s["image"].fill(0.0)
        R.wstack(nw, n, c["nchan"], c["npol"], uu, vv, ww, re, im, wt, 1.0 / g, 1.0 / nw,
                 c["support"], g, g, s["grid"])
        R.fft_planes(s["grid"], nw, g, g, out=s["gridss"])
        R.phase_correction(s["gridss"], s["image"][0], s["image"][1], g, g, nw, g, g, s["res"],
                           s["wmin"], s["wmax"])
        return {"grid": s["grid"], "gridss": s["gridss"], "image": s["image"]}
    out = s["images"] if "images" in s else s["image"]
    return out.float() if c["precision"] == "mixed" else out


# ---- what a pass cannot do without ---------------------------------------------

def _work(c):
    vis = c["rows"] * c["nchan"] * c["npol"]
    planes = c["w_count"] or c["planes"]
    kept = c["rows"] * planes / c["planes"]
    cells = planes * c["grid"] ** 2
    vis *= planes / c["planes"]  # a shard needs the samples of its own planes only
    # each sample weighted and summed once, each footprint cell added into once,
    # one 1-D inverse transform per column and plane, the w-correction per pixel
    # and plane (rows of the planes without data need no transform)
    flops = 4 * vis + 4 * c["support"] ** 2 * kept + 5 * cells * math.log2(c["grid"]) + 8 * cells
    return 8 * vis + kept * (24 + 4 * c["npol"]), flops


def work(case):
    c = case
    if c["call"] in ("batch", "served"):
        parts = [(_work(j), j["grid"] ** 2) for j in _snapshots(c)]
    else:
        parts = [(_work(c), c["grid"] ** 2)]
    out_bytes = 8 if c["precision"] == "mixed" else 16
    total = sum(p[0][0] + out_bytes * p[1] for p in parts)
    if c["call"] == "dropin":  # the cube in and out of each call, the image in and out
        total += 4 * 16 * c["planes"] * c["grid"] ** 2
    return {"bytes": total, "flops": sum(p[0][1] for p in parts)}


# ---- the definition, in 64 bits --------------------------------------------------

def _bessel0(x):
    d, ds, total = 0.0, 1.0, 1.0
    while True:
        d += 2.0
        ds *= x * x / (d * d)
        total += ds
        if ds <= total * 1e-8:
            return total


def _table(kernel, support):
    n = 5 * support
    mid = n // 2
    tab = np.zeros(n)
    for i in range(mid + 1):
        if kernel == "gauss":
            tab[mid + i] = math.sqrt(0.5 / PI) * math.exp(-0.5 * (i / 5.0) ** 2)
        else:
            tab[mid + i] = _bessel0(8.6 * math.sqrt(1.0 - (i / mid) ** 2)) / _bessel0(8.6)
    for i in range(mid):
        tab[i] = tab[n - 1 - i]
    return torch.tensor(tab, device="cuda")


def _axis_weights(pos, support, kernel, tab):
    """Kernel factors [support, rows] of the cells around positions ``pos``."""
    half = (support - 1) // 2
    frac = pos - pos.to(torch.int64)
    out = []
    for d in range(support):
        dist = (float(d - half) + 0.5) - frac
        if kernel == "gauss_hi":
            out.append(torch.exp(-0.5 * dist * dist))
        else:
            k = (5.0 * (dist + half).abs()).to(torch.int64).clamp_(max=5 * support - 1)
            out.append(tab[k])
    return out


def _exact_planes(c, rows, each):
    """Grids plane after plane of the job and calls each(plane, complex grid)."""
    uu, vv, ww, wt, re, im = rows
    n, nchan, npol, g, sup = c["rows"], c["nchan"], c["npol"], c["grid"], c["support"]
    half = (sup - 1) // 2
    re, im, wt = re.view(n, nchan, npol), im.view(n, nchan, npol), wt.view(n, 1, npol)
    s_re = torch.empty(n, dtype=torch.float64, device="cuda")
    s_im = torch.empty_like(s_re)
    step = max(1, (1 << 25) // (nchan * npol))
    for r0 in range(0, n, step):
        r = slice(r0, min(n, r0 + step))
        ok = ~torch.isnan(re[r])
        # the product weight * sample is FP32 by definition, the sums are wide
        s_re[r] = torch.where(ok, wt[r] * re[r], 0.0).double().sum((1, 2))
        s_im[r] = torch.where(ok, wt[r] * im[r], 0.0).double().sum((1, 2))
    dx, dw = 1.0 / g, 1.0 / c["planes"]
    pu, pv, gw = uu / dx, vv / dx, (ww / dw).to(torch.int64)
    tab = None if c["kernel"] == "gauss_hi" else _table(c["kernel"], sup)
    amp = 0.5 / PI if c["kernel"] == "gauss_hi" else 1.0
    order = torch.argsort(gw)
    bounds = torch.searchsorted(gw[order], torch.arange(c["planes"] + 1, device="cuda")).tolist()
    first = c["w_first"]
    for iw in range(first, first + (c["w_count"] or c["planes"])):
        pick = order[bounds[iw]: bounds[iw + 1]]
        # one guard ring of cells takes what falls outside the grid
        ring = half + 1
        pitch = g + 2 * ring
        grid = torch.zeros((pitch * pitch, 2), dtype=torch.float64, device="cuda")
        if len(pick):
            a, b = pu[pick], pv[pick]
            wu = _axis_weights(a, sup, c["kernel"], tab)
            wv = _axis_weights(b, sup, c["kernel"], tab)
            s = torch.stack([s_re[pick], s_im[pick]], 1) * amp
            corner = (b.to(torch.int64) - half + ring) * pitch + a.to(torch.int64) - half + ring
            for e in range(sup):
                for d in range(sup):
                    grid.index_add_(0, corner + (e * pitch + d), s * (wu[d] * wv[e])[:, None])
        grid = grid.view(pitch, pitch, 2)[ring: ring + g, ring: ring + g].contiguous()
        each(iw, torch.view_as_complex(grid))


def _exact_image(c, seed, keep_cubes=False):
    rows, res, wmin, wmax = _observation(c, seed)
    g, nw = c["grid"], c["planes"]
    i = torch.arange(g, dtype=torch.float64, device="cuda")
    x = torch.where(i - g // 2 < 0, i + g // 2, i - g // 2)
    lm = torch.sin(x * res) ** 2
    root = torch.sqrt(1.0 - (lm[None, :] + lm[:, None]))
    dw = (wmax - wmin) / nw
    image = torch.zeros((g, g), dtype=torch.complex128, device="cuda")
    cubes = []

    def each(iw, grid):
        plane = torch.fft.ifft2(grid)
        if keep_cubes:
            cubes.append((grid.clone(), plane.clone()))
        if nw > 1:
            arg = (2.0 * PI * (wmin + iw * dw)) * (root - 1.0)
            plane = plane * torch.polar(root * (dw / (wmax - wmin)), arg)
        image.add_(plane)

    _exact_planes(c, rows, each)
    image = torch.stack([image.real, image.imag])
    return (image, cubes) if keep_cubes else image


def exact(case, seed):
    c = case
    if c["call"] in ("batch", "served"):
        return torch.cat([_exact_image(j, seed * 1000 + k).reshape(-1)
                          for k, j in enumerate(_snapshots(c))])
    if c["call"] == "dropin":
        image, cubes = _exact_image(c, seed, keep_cubes=True)
        cube = [torch.view_as_real(torch.stack([p[k] for p in cubes])).reshape(-1).cpu().numpy()
                for k in (0, 1)]
        return {"grid": cube[0], "gridss": cube[1],
                "image": image.reshape(2, -1).cpu().numpy()}
    return _exact_image(c, seed)
