"""Timed cases of the denoise stage: what a program that calls it does, over the range it does it.

A case is one frame of a renderer (or one call of a post-filter, one batch, one burst of served
requests) at a stated size, samples per pixel, storage and set of knobs. `listed` holds the fixed
ones, `draw` gives more of the same ranges; `prepare` makes what the program has in hand before the
call, `run` is the call, `work` the bytes and operations it cannot do without and `exact` the same
results in 64-bit arithmetic.

Scenes. "synth" is the benchmark's structure: 48 Voronoi regions, each with a constant normal and
albedo, a planar depth and a log-normal radiance (mu in [-2, 1], sigma 0.8), half of them depending
on two random dimensions, 0.1 % fireflies, every random dimension valid. "path" adds what the
committed cornell_box samples of the reference's tracer show: a quarter of the samples black (whole
regions in shadow), a tenth of a region's samples or more without some random dimension (more than
half of the pixels mix validity patterns), and a background region without a primary hit.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "rpd-statmc-denoiser_gb300"))

import rpd_gb300 as R  # noqa: E402

DEV = "cuda"

# Stage knobs. "bench": the benchmark's plain method (rpf tile 16, colour radius 5, variance radius 3).
# "defaults": RenderConfig's defaults (tile 8, colour radius 7, variance radius 1). "fine": a smaller
# colour window over a coarser sensitivity grid.
KNOBS = {
    "bench": dict(rpf_tile_size=16, color_window_radius=5, color_normal_threshold=0.6, color_depth_threshold=0.2,
                  color_compat_alpha=0.01, color_sigma_max=4.0, var_window_radius=3, var_normal_threshold=0.6,
                  var_compat_sigma=3.0, var_shrinkage_k=0.7, var_iterations=2, adaptive_spp=4,
                  adaptive_base_samples=1, adaptive_sigma_max=4.0),
    "defaults": dict(adaptive_spp=4, adaptive_base_samples=1),
    "fine": dict(rpf_tile_size=32, color_window_radius=3, var_window_radius=2, var_iterations=3, adaptive_spp=4,
                 adaptive_base_samples=0),
}
SIZES = [(256, 256), (640, 360), (1280, 720), (1920, 1080), (2048, 1152)]  # the mixed-size job stream's
SPPS = [4, 8, 16, 32, 64]
FRAME_FIELDS = ("DENOISED", "UNCERTAINTY", "VARIANCE_DENOISED", "SENSITIVITY_CONFIDENCE")


def listed():
    f = dict(kind="frame", storage="fp32", scene="synth", knobs="bench", env=False, sample_albedo=False)
    return [
        # a thumbnail: every launch is latency
        dict(f, name="frame 64x48x8", width=64, height=48, spp=8),
        # the reference's cornell_box preview, with a tracer's samples (albedo per sample)
        dict(f, name="cornell 256x256x4", width=256, height=256, spp=4, scene="path", sample_albedo=True),
        # odd sizes, a count that is no power of two, the renderer's default knobs, an environment map
        dict(f, name="ragged 1283x717x6", width=1283, height=717, spp=6, knobs="defaults", scene="path", env=True),
        # the benchmark's frame, and the same in compact storage
        dict(f, name="plain 1080p x16", width=1920, height=1080, spp=16),
        dict(f, name="compact 1080p x16", width=1920, height=1080, spp=16, storage="fp16"),
        # the largest frame of the job stream
        dict(f, name="compact 2048x1152x64", width=2048, height=1152, spp=64, storage="fp16"),
        # render()'s sequence with one adaptive pass: a tracer's samples, then counts per pixel
        dict(f, name="adaptive 1280x720 8+4", kind="adaptive", width=1280, height=720, spp=8, scene="path"),
        # the drop-in as a CPU tracer calls it: samples in page-locked host memory, image back to it
        dict(f, name="host 960x540x8", kind="host", width=960, height=540, spp=8),
        # the post-filters on a full frame
        dict(kind="atrous", name="a-trous 1080p", width=1920, height=1080, iterations=5, sigma_c=0.3, sigma_n=0.2,
             sigma_a=0.1),
        dict(kind="bilateral", name="joint bilateral 1080p", width=1920, height=1080, sigma_c=0.3, sigma_n=0.2,
             sigma_p=2.0, sigma_a=0.1),
        # an animation's uneven frames in one graph launch
        dict(kind="batch", name="batch of 6", knobs="bench", scene="synth",
             frames="256x256x4 640x360x32 1280x720x8 640x360x64 1920x1080x16 256x256x16"),
        # a burst of requests at the server, three adaptive passes each
        dict(kind="served", name="served burst of 8", storage="fp16",
             frames="256x256x4 640x360x16 1280x720x8 256x256x64 1920x1080x8 640x360x4 1280x720x16 256x256x8"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["adaptive"] * 2 + ["host", "atrous", "bilateral", "batch", "served"])
    w, h = _log_int(rng, 48, 2048), _log_int(rng, 32, 1152)
    if kind in ("atrous", "bilateral"):
        c = dict(kind=kind, width=w, height=h, sigma_c=round(rng.uniform(0.1, 1.0), 3),
                 sigma_n=round(rng.uniform(0.1, 0.5), 3), sigma_a=round(rng.uniform(0.05, 0.5), 3))
        if kind == "atrous":
            return dict(c, iterations=rng.randint(1, 6))
        return dict(c, sigma_p=rng.choice([0.7, 1.0, 1.5, 2.0, 3.0]))
    if kind in ("batch", "served"):
        frames = " ".join("%dx%dx%d" % (*rng.choice(SIZES[:4]), rng.choice(SPPS[:4])) for _ in range(rng.randint(2, 6)))
        if kind == "batch":
            return dict(kind=kind, knobs=rng.choice(sorted(KNOBS)), scene=rng.choice(["synth", "path"]), frames=frames)
        return dict(kind=kind, storage=rng.choice(["fp16", "fp32"]), frames=frames)
    c = dict(kind=kind, width=w, height=h, spp=_log_int(rng, 1, 64), knobs=rng.choice(sorted(KNOBS)),
             scene=rng.choice(["synth", "path"]), env=rng.random() < 0.3, sample_albedo=False, storage="fp32")
    if kind == "frame":
        c["storage"] = rng.choice(["fp32", "fp32", "fp16"])
    if kind == "host":
        c["spp"] = min(c["spp"], 16)
    if c["storage"] == "fp32":
        c["sample_albedo"] = rng.random() < 0.4
        while w * h * c["spp"] > 60_000_000:  # FP32 frames hold twice the bytes
            c["spp"] //= 2
    return c


# ---- scenes -----------------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFF)
    return g


def _scene(w, h, kind, g):
    """Per-region tables and each pixel's region."""
    n = 48
    rnd = lambda *s: torch.rand(*s, device=DEV, generator=g)  # noqa: E731
    cx, cy = rnd(n) * w, rnd(n) * h
    x = torch.arange(w, device=DEV, dtype=torch.float32)
    y = torch.arange(h, device=DEV, dtype=torch.float32)
    best = torch.full((h, w), math.inf, device=DEV)
    region = torch.zeros((h, w), dtype=torch.int64, device=DEV)
    for r in range(n):
        d = (x[None, :] - cx[r]) ** 2 + (y[:, None] - cy[r]) ** 2
        near = d < best
        best = torch.where(near, d, best)
        region[near] = r
    nrm = torch.stack([rnd(n) * 2 - 1, rnd(n) * 2 - 1, rnd(n) + 0.3], 1)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    tint = rnd(n, 3) + 0.2
    tint = tint / (tint @ torch.tensor([0.2126, 0.7152, 0.0722], device=DEV))[:, None]
    s = dict(normal=nrm, d0=rnd(n) * 5 + 3, gx=rnd(n) * 4 - 2, gy=rnd(n) * 4 - 2, albedo=rnd(n, 3) * 0.9 + 0.05,
             tint=tint, mu=rnd(n) * 3 - 2, dim_a=(rnd(n) * 8).long().clamp(max=7),
             dim_b=(rnd(n) * 8).long().clamp(max=7), region=region.reshape(-1), w=w, h=h, kind=kind,
             black=torch.zeros(n, device=DEV), loss=torch.zeros(n, device=DEV))
    if kind == "path":
        s["black"] = (rnd(n) * 1.1 - 0.3).clamp(0.0, 0.8)
        s["black"][::8] = 1.0  # in shadow
        s["loss"] = rnd(n) * 0.5
    return s


def _samples(s, pix, g, env, sample_albedo):
    """The FP32 planes of one sample per entry of `pix` (pixel indices, in increasing order)."""
    n = pix.numel()
    rnd = lambda: torch.rand(n, device=DEV, generator=g)  # noqa: E731
    reg = s["region"][pix]
    u = [rnd() for _ in range(8)]  # lens uv, BRDF uv, light select, light uv, Russian roulette
    pu = [rnd() for _ in range(2)]
    lum = torch.exp(s["mu"][reg] + 0.8 * torch.randn(n, device=DEV, generator=g))
    dep = (reg & 1) == 1
    ua, ub = torch.zeros(n, device=DEV), torch.zeros(n, device=DEV)
    for d in range(8):
        ua = torch.where(s["dim_a"][reg] == d, u[d], ua)
        ub = torch.where(s["dim_b"][reg] == d, u[d], ub)
    lum = torch.where(dep, lum * (1.0 + 0.5 * (ua + ub - 1.0)), lum)
    lum = torch.where(rnd() < 0.001, lum * 100.0, lum)
    flags = torch.full((n,), 0xBF, dtype=torch.uint8, device=DEV)  # every dimension but the environment
    hit = torch.ones(n, dtype=torch.bool, device=DEV)
    if s["kind"] == "path":
        lum = torch.where(rnd() < s["black"][reg], torch.zeros_like(lum), lum)
        lost = rnd() < s["loss"][reg]  # paths that end before Russian roulette
        flags = torch.where(lost, flags & 0x7F, flags)
        lost = rnd() < 0.2 * s["loss"][reg]  # paths that end at the first hit
        flags = torch.where(lost, torch.full_like(flags, 0x03), flags)
        hit = reg != 1  # background
        flags = torch.where(hit, flags, torch.full_like(flags, 0x02))
    if env:
        flags = torch.where((flags & 0x08) != 0, flags | 0x40, flags)
    x, y = (pix % s["w"]).float(), torch.div(pix, s["w"], rounding_mode="floor").float()
    depth = s["d0"][reg] + s["gx"][reg] * ((x + pu[0]) / s["w"] - 0.5) + s["gy"][reg] * ((y + pu[1]) / s["h"] - 0.5)
    zero = torch.zeros(n, device=DEV)
    p = {"radiance": [lum * s["tint"][:, c][reg] for c in range(3)],
         "normal": [torch.where(hit, s["normal"][:, c][reg], zero) for c in range(3)],
         "depth": [torch.where(hit, depth.clamp(1.0, 10.0), zero)], "pixel_u": pu, "lens_u": u[0:2], "brdf_u": u[2:4],
         "light_u": u[5:7], "flags": [flags],
         "category": [((u[4] * 4).to(torch.uint8).clamp(max=3) | torch.where(u[7] < 0.8, 16, 0).to(torch.uint8))]}
    if env:
        p["env_u"] = [rnd(), rnd()]
    if sample_albedo:
        p["albedo"] = [torch.where(hit, s["albedo"][:, c][reg], zero) for c in range(3)]
    return p


def _encode16(p, scale):
    """The compact planes of FP32 ones (rpd_sample_soa16's formats)."""
    out = {"sqrt_radiance": [v.clamp(min=0).sqrt().half().view(torch.int16) for v in p["radiance"]],
           "normal": [(v * 32767.0).round().to(torch.int16) for v in p["normal"]],
           "depth": [(v / scale).half().view(torch.int16) for v in p["depth"]],
           "pixel_albedo": [v.half().view(torch.int16) for v in p["pixel_albedo"]],
           "flags": p["flags"], "category": p["category"]}
    for name in ("pixel_u", "lens_u", "brdf_u", "light_u", "env_u"):
        if name in p:
            out[name] = [(v * 65536.0).floor().clamp(max=65535).to(torch.int32).to(torch.int16) for v in p[name]]
    return out


def _decode16(p, scale):
    u16 = lambda v: (v.to(torch.int32) & 0xFFFF).double()  # noqa: E731
    out = {"radiance": [v.view(torch.half).double().square() for v in p["sqrt_radiance"]],
           "normal": [(v.double() / 32767.0).clamp(min=-1.0) for v in p["normal"]],
           "depth": [v.view(torch.half).double() * scale for v in p["depth"]],
           "pixel_albedo": [v.view(torch.half).double() for v in p["pixel_albedo"]],
           "flags": p["flags"], "category": p["category"]}
    for name in ("pixel_u", "lens_u", "brdf_u", "light_u", "env_u"):
        if name in p:
            out[name] = [u16(v) / 65536.0 for v in p[name]]
    return out


DEPTH_SCALE = 16.0


def _passes(case, seed):
    """The frame's pushes, [(planes, counts per pixel or None)], from the seed alone."""
    w, h, spp = case["width"], case["height"], case["spp"]
    g = _generator(seed)
    s = _scene(w, h, case["scene"], g)
    pix = torch.arange(w * h, device=DEV).repeat_interleave(spp)
    passes = []
    for counts in [None] + ([_extra_counts(s, g, 4)] if case["kind"] == "adaptive" else []):
        if counts is not None:
            pix = torch.arange(w * h, device=DEV).repeat_interleave(counts.long())
        p = _samples(s, pix, g, case.get("env", False), case.get("sample_albedo", False))
        if "albedo" not in p:
            p["pixel_albedo"] = [s["albedo"][:, c][s["region"]].contiguous() for c in range(3)]
        if case.get("storage") == "fp16":
            p = _encode16(p, DEPTH_SCALE)
        passes.append((p, counts))
    return passes


def _extra_counts(s, g, spp):
    """An adaptive pass's counts: `spp` a pixel on average, most of them on noisy regions, some pixels far more."""
    n = s["region"].numel()
    weight = torch.exp(0.5 * s["mu"])[s["region"]] * (0.25 + torch.rand(n, device=DEV, generator=g))
    weight = torch.where(torch.rand(n, device=DEV, generator=g) < 0.01, weight * 8, weight)
    c = (weight * (spp / weight.mean()) + torch.rand(n, device=DEV, generator=g)).floor()
    return c.clamp(1, 8 * spp).to(torch.int32)


# ---- what a program keeps ------------------------------------------------------------------------

_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = R.Context(0, 0)
    return _ctx


class _State:
    """A program's objects, released with the state."""

    def __init__(self, case):
        self.case, self.closing, self.out = case, [], None

    def own(self, obj, method="close"):
        self.closing.append(getattr(obj, method))
        return obj

    def __del__(self):
        for close in reversed(self.closing):
            close()


def _device_planes(st, ctx, p, w, h, n, compact):
    """The planes in the stage's own device buffers."""
    dev = (R.DeviceSamples16(ctx, n, w * h, tuple(p), DEPTH_SCALE) if compact
           else R.DeviceSamples(ctx, n, w * h, tuple(p)))
    st.own(dev, "free")
    torch.cuda.synchronize()
    for name, planes in p.items():
        for buf, t in zip(dev.bufs[name], planes):
            R.check(R.lib().rpd_memcpy(ctx.handle, buf.ptr, t.data_ptr(), t.numel() * t.element_size(), 2))
    return dev


def _host_planes(st, p, w, h, n):
    """The planes in page-locked host memory, as HostSamples."""
    host = R.HostSamples.__new__(R.HostSamples)
    host.n_samples, host.n_pixels, host.planes = n, w * h, {}
    for name, planes in p.items():
        t = torch.stack(planes).cpu().numpy() if len(planes) > 1 else planes[0].cpu().numpy()
        a = st.own(R.PinnedBuffer(t.nbytes), "free").array(t.dtype, t.shape)
        a[...] = t
        host.planes[name] = a
    return host


def _config(case, w, h):
    return R.default_config(image_width=w, image_height=h, seed=1234, **KNOBS[case["knobs"]])


def _outputs(w, h, fields):
    return {f.lower(): torch.empty((h, w, 3) if f in R.RGB_FIELDS else (h, w), device=DEV) for f in fields}


def _read(job, out, fields):
    for f in fields:
        t = out[f.lower()]
        R.check(R.lib().rpd_job_read_async(job.handle, R.FIELD[f], t.data_ptr(), t.numel() * 4, R.MEM_DEVICE))


def _frames(case):
    return [tuple(int(v) for v in f.split("x")) for f in case["frames"].split()]


def _images(w, h, seed):
    """A frame as the post-filters take it: noisy radiance over a scene's normals (n / 2 + 1 / 2) and albedo."""
    g = _generator(seed)
    s = _scene(w, h, "synth", g)
    reg = s["region"]
    lum = torch.exp(s["mu"][reg] + 0.4 * torch.randn(w * h, device=DEV, generator=g))
    raw = (lum[:, None] * s["tint"][reg]).reshape(h, w, 3).contiguous()
    nrm = s["normal"][reg] + 0.05 * torch.randn(w * h, 3, device=DEV, generator=g)
    nrm = (nrm / nrm.norm(dim=1, keepdim=True) * 0.5 + 0.5).reshape(h, w, 3).contiguous()
    alb = (s["albedo"][reg] + 0.02 * torch.rand(w * h, 3, device=DEV, generator=g)).reshape(h, w, 3).contiguous()
    return raw, nrm, alb


def prepare(case, seed):
    ctx = _context()
    st = _State(case)
    kind = case["kind"]
    if kind in ("atrous", "bilateral"):
        st.images = _images(case["width"], case["height"], seed)
        st.out = [torch.empty_like(st.images[0]) for _ in range(1 if kind == "atrous" else 3)]
    elif kind == "served":
        knobs = _config(dict(knobs="bench"), 1, 1).replace(adaptive_passes=3, adaptive_spp=4, adaptive_base_samples=1)
        st.server = st.own(R.Server(ctx, knobs, max_inflight=32, storage=case["storage"]))
        st.seed = seed
        st.out = [torch.empty((h, w, 3), device=DEV) for w, h, _ in _frames(case)]
        st.to = []
        for t in st.out:  # the server's device outputs are named by their address
            b = R.DeviceBuffer.__new__(R.DeviceBuffer)
            b.ctx, b.nbytes, b.ptr = ctx, t.numel() * 4, t.data_ptr()
            st.to.append(b)
    elif kind == "batch":
        st.batch = R.Batch(ctx)
        st.jobs, st.out = [], []
        for k, (w, h, spp) in enumerate(_frames(case)):
            one = dict(kind="frame", width=w, height=h, spp=spp, scene=case["scene"], storage="fp16")
            planes, _ = _passes(one, seed + 1000 * k)[0]
            dev = _device_planes(st, ctx, planes, w, h, w * h * spp, True)
            job = st.own(R.Job(ctx, _config(case, w, h)))
            st.batch.add(job, dev, spp)
            st.jobs.append(job)
            st.out.append(_outputs(w, h, FRAME_FIELDS))
        st.own(st.batch)
    else:
        w, h = case["width"], case["height"]
        passes = _passes(case, seed)
        n = w * h * case["spp"]
        st.job = st.own(R.Job(ctx, _config(case, w, h)))
        if kind == "host":
            st.samples = _host_planes(st, passes[0][0], w, h, n)
            st.image = torch.empty((h, w, 3), pin_memory=True)  # page-locked
        else:
            st.samples = _device_planes(st, ctx, passes[0][0], w, h, n, case["storage"] == "fp16")
            st.out = _outputs(w, h, FRAME_FIELDS)
        if kind == "adaptive":
            planes, counts = passes[1]
            st.extra = _device_planes(st, ctx, planes, w, h, int(counts.sum()), False)
            st.counts = st.own(R.DeviceBuffer(ctx, 4 * w * h), "free")
            R.check(R.lib().rpd_memcpy(ctx.handle, st.counts.ptr, counts.data_ptr(), 4 * w * h, 2))
    torch.cuda.synchronize()
    return st


def run(st):
    case = st.case
    kind = case["kind"]
    lib, ctx = R.lib(), _context()
    if kind in ("atrous", "bilateral"):
        a = [t.data_ptr() for t in st.images]
        w, h, out = case["width"], case["height"], [t.data_ptr() for t in st.out]
        if kind == "atrous":
            R.check(lib.rpd_atrous_wavelet(ctx.handle, *a, w, h, case["sigma_c"], case["sigma_n"], case["sigma_a"],
                                           case["iterations"], out[0], R.MEM_DEVICE))
        else:
            R.check(lib.rpd_joint_bilateral(ctx.handle, *a, w, h, case["sigma_c"], case["sigma_n"], case["sigma_p"],
                                            case["sigma_a"], *out, R.MEM_DEVICE))
        return st.out
    if kind == "served":
        for k, (w, h, spp) in enumerate(_frames(case)):
            st.server.submit(w, h, spp, st.seed + 7919 * k, out=st.to[k], tag=k)
        st.server.drain()
        if any(c["status"] for c in st.server.poll()):
            raise RuntimeError("a request failed")
        return st.out
    if kind == "batch":
        st.batch.run()
        st.batch.sync()
        for job, out in zip(st.jobs, st.out):
            _read(job, out, FRAME_FIELDS)
        return st.out
    job, n = st.job, case["width"] * case["height"]
    job.begin_frame()
    job.push(st.samples, 0, n, case["spp"])
    job.end_pass()
    job.recompute_sensitivity()
    if kind == "adaptive":
        job.statmc_denoise()
        job.variance_denoise()
        asked = job.compute_adaptive_sample_counts()
        job.push(st.extra, 0, n, 0, counts=st.counts)  # what the tracer drew
        job.end_pass()
        job.recompute_sensitivity()
    job.statmc_denoise()
    job.variance_denoise()
    if kind == "host":
        R.check(lib.rpd_job_read(job.handle, R.FIELD["DENOISED"], st.image.data_ptr(), n * 12, R.MEM_HOST))
        return {"denoised": st.image}
    _read(job, st.out, FRAME_FIELDS)
    return {**st.out, "counts": asked} if kind == "adaptive" else st.out


# ---- the work a pass cannot do without ------------------------------------------------------------


def _frame_work(w, h, spp, knobs, compact, env=False, sample_albedo=False, out_bytes=24):
    n, npix, k = w * h * spp, w * h, KNOBS[knobs]
    dims = 10 if env else 8
    per = 2 * (7 + dims) + 2 if compact else 4 * (7 + dims + (3 if sample_albedo else 0)) + 2
    r, rv, iters = k.get("color_window_radius", 7), k.get("var_window_radius", 1), k.get("var_iterations", 2)
    pixel_albedo = 0 if sample_albedo else (6 if compact else 12)
    flops = n * (45 + 4 * 5 * 3) + npix * (75 * (2 * r + 1) ** 2 + 16 * iters * (2 * rv + 1) ** 2 + 150)
    return {"bytes": n * per + npix * (pixel_albedo + out_bytes), "flops": flops}


def work(case):
    kind = case["kind"]
    if kind in ("atrous", "bilateral"):
        n = case["width"] * case["height"]
        if kind == "atrous":
            return {"bytes": n * 48, "flops": n * case["iterations"] * 25 * 35}
        r = max(1, math.ceil(3 * case["sigma_p"]))
        return {"bytes": n * 72, "flops": n * (2 * r + 1) ** 2 * 50}
    if kind in ("batch", "served"):
        parts = [_frame_work(w, h, spp, case.get("knobs", "bench"), True, out_bytes=24 if kind == "batch" else 12)
                 for w, h, spp in _frames(case)]
        if kind == "served":  # the samples are made on the device: 12 more a pixel, none of them read from outside
            parts = [{"bytes": w * h * 12, "flops": p["flops"] + w * h * (12 * 150 + spp * 45)}
                     for (w, h, spp), p in zip(_frames(case), parts)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    w, h = case["width"], case["height"]
    p = _frame_work(w, h, case["spp"], case["knobs"], case["storage"] == "fp16", case["env"], case["sample_albedo"],
                    12 if kind == "host" else 28 if kind == "adaptive" else 24)
    if kind == "adaptive":
        again = _frame_work(w, h, 4, case["knobs"], False, case["env"], case["sample_albedo"], 0)
        p = {"bytes": p["bytes"] + again["bytes"], "flops": p["flops"] + again["flops"]}
    return p


# ---- the same results in 64 bits ------------------------------------------------------------------

_LUM = [float(np.float32(v)) for v in (0.2126, 0.7152, 0.0722)]
_T05 = [12.706, 4.303, 3.182, 2.776, 2.571, 2.447, 2.365, 2.306, 2.262, 2.228, 2.201, 2.179, 2.160, 2.145, 2.131, 2.120,
        2.110, 2.101, 2.093, 2.086, 2.080, 2.074, 2.069, 2.064, 2.060, 2.056, 2.052, 2.048, 2.045, 2.042]
_T01 = [63.657, 9.925, 5.841, 4.604, 4.032, 3.707, 3.499, 3.355, 3.250, 3.169, 3.106, 3.055, 3.012, 2.977, 2.947, 2.921,
        2.898, 2.878, 2.861, 2.845, 2.831, 2.819, 2.807, 2.797, 2.787, 2.779, 2.771, 2.763, 2.756, 2.750]


def _f(v):
    """A knob as the single-precision value it is given in."""
    return float(np.float32(v))


def _add(into, pix, spp, v):
    """into[pixel] += the pixel's samples of v (spp each, or as pix says)."""
    if spp:
        into += v.reshape(-1, spp).sum(1)
    else:
        into.index_add_(0, pix, v)


def _moments(np_, passes):
    """Per-pixel counts, sums and central squares over all passes' samples (every radiance is finite)."""
    add = _add
    zero = lambda: torch.zeros(np_, dtype=torch.float64, device=DEV)  # noqa: E731
    m = {k: zero() for k in ("n", "hits", "depth", "lum", "m2")}
    m |= {k: [zero() for _ in range(3)] for k in ("color", "sqrt", "sq", "normal", "albedo")}
    for pix, spp, p in passes:
        hit = (p["flags"][0] & 1).double()
        add(m["n"], pix, spp, torch.ones_like(hit))
        add(m["hits"], pix, spp, hit)
        add(m["depth"], pix, spp, p["depth"][0].double() * hit)
        add(m["lum"], pix, spp, p["lum"])
        for c in range(3):
            add(m["color"][c], pix, spp, p["radiance"][c].double())
            add(m["sqrt"][c], pix, spp, p["radiance"][c].double().sqrt())
            add(m["normal"][c], pix, spp, p["normal"][c].double() * hit)
            a = p["albedo"][c].double() if "albedo" in p else p["pixel_albedo"][c].double()[pix]
            add(m["albedo"][c], pix, spp, a * hit)
    n = m["n"].clamp(min=1)
    m["lum"] = m["lum"] / n
    for k in ("color", "sqrt"):
        m[k] = [v / n for v in m[k]]
    for pix, spp, p in passes:
        add(m["m2"], pix, spp, (p["lum"] - m["lum"][pix]).square())
        for c in range(3):
            add(m["sq"][c], pix, spp, (p["radiance"][c].double().sqrt() - m["sqrt"][c][pix]).square())
    return m


def _axis(size, nodes, step):
    """Bilinear weights [nodes, size] of the pixel columns (or rows) at the grid's nodes."""
    c = torch.arange(size, device=DEV, dtype=torch.float64) / step
    lo = c.floor().clamp(0, nodes - 1)
    hi = (lo + 1).clamp(max=nodes - 1)
    t = (c - lo).clamp(0, 1)
    k = torch.arange(nodes, device=DEV, dtype=torch.float64)[:, None]
    return torch.where(k == lo, 1 - t, torch.where(k == hi, t, torch.zeros_like(t)))


def _screen_bins(size, nodes, step, support):
    """Screen bin of each (node, pixel column): a pixel's samples stay in its bin (support a multiple of 4)."""
    x = torch.arange(size, device=DEV)[None, :]
    left = torch.arange(nodes, device=DEV)[:, None] * step - support // 2
    return torch.div(x - left, support // 4, rounding_mode="floor").clamp(0, 3)


def _sensitivity(grid):
    """Bias-adjusted explained variance and sample mass of [nodes, (w, wy) bins, totals] sums."""
    wb, yb, w, w2, y, y2 = grid
    mass = torch.where(w2 > 0, w * w / w2.clamp(min=1e-300), torch.zeros_like(w))
    mean = y / torch.where(w > 0, w, torch.ones_like(w))
    total = y2 - w * mean * mean
    live = wb > 1e-18
    delta = yb / torch.where(live, wb, torch.ones_like(wb)) - mean
    between = torch.where(live, wb * delta * delta, torch.zeros_like(wb)).sum(0)
    active = live.sum(0).double()
    eta2 = (between / torch.where(total > 1e-18, total, torch.ones_like(total))).clamp(0, 1)
    adj = (1 - (1 - eta2) * (mass - 1) / torch.where(mass > active, mass - active, torch.ones_like(mass))).clamp(min=0)
    ok = (mass > 2) & (total > 1e-18) & (active >= 2) & (mass > active)
    return torch.where(ok, adj.sqrt(), torch.zeros_like(adj)), mass


def _rpd(passes, m, w, h, cfg):
    """Node fields of the sensitivity grid: confidence of the dominant component, all, and the six components."""
    support = cfg.rpf_tile_size
    step = max(1, support // 2)
    nx, ny = max(2, -(-w // step) + 1), max(2, -(-h // step) + 1)
    ax, ay = _axis(w, nx, step), _axis(h, ny, step)
    bx, by = _screen_bins(w, nx, step, support), _screen_bins(h, ny, step, support)
    np_ = w * h

    def collect(v):  # pixel sums -> node sums
        return ay @ v.reshape(h, w) @ ax.T

    def per_pixel(value):
        out = torch.zeros(np_, dtype=torch.float64, device=DEV)
        for pix, spp, p in passes:
            _add(out, pix, spp, value(p))
        return out

    def binned(bin_of, bins, valid):
        cnt = torch.zeros(np_ * bins, dtype=torch.float64, device=DEV)
        sy = torch.zeros_like(cnt)
        for pix, _, p in passes:
            ok = valid(p)
            at = pix * bins + bin_of(p)
            cnt.index_add_(0, at, ok)
            sy.index_add_(0, at, ok * p["lum"])
        cut = lambda v: torch.stack([collect(v[b::bins]) for b in range(bins)])  # noqa: E731
        return cut(cnt), cut(sy)

    def totals(valid):
        c, y, y2 = (per_pixel(lambda p, e=e: valid(p) * p["lum"] ** e) for e in range(3))
        c2 = (ay * ay) @ c.reshape(h, w) @ (ax * ax).T
        return c, y, (collect(c), c2, collect(y), collect(y2))

    def screen(c, y):
        cut = lambda v: torch.stack([(ay * (by == j)) @ v.reshape(h, w) @ (ax * (bx == i)).T  # noqa: E731
                                     for j in range(4) for i in range(4)])
        return cut(c), cut(y)

    def uv(name):
        return lambda p: ((p[name][1] * 4).long().clamp(0, 3) * 4 + (p[name][0] * 4).long().clamp(0, 3))

    dims = [(0x08, uv("brdf_u"), 16, "brdf_u"), (0x04, uv("lens_u"), 16, "lens_u"), (0x10, uv("light_u"), 16, "light_u"),
            (0x20, lambda p: (p["category"][0] & 15).long(), 16, "category"), (0x40, uv("env_u"), 16, "env_u"),
            (0x80, lambda p: ((p["category"][0] >> 4) & 1).long(), 2, "category")]
    raw, conf = [], []
    n0 = _f(cfg.rpf_confidence_samples)
    for bit, bin_of, bins, plane in dims:
        if plane not in passes[0][2]:
            z = torch.zeros(ny, nx, dtype=torch.float64, device=DEV)
            raw.append((z, z))
            conf.append((z, z))
            continue
        valid = lambda p, b=bit: ((p["flags"][0] & b) != 0).double()  # noqa: E731
        seen = lambda p, b=bit: (((p["flags"][0] & b) != 0) & ((p["flags"][0] & 2) != 0)).double()  # noqa: E731
        _, _, t = totals(valid)
        s1, m1 = _sensitivity((*binned(bin_of, bins, valid), *t))
        c, y, t = totals(seen)
        s2, m2 = _sensitivity((*screen(c, y), *t))
        raw.append((s1, s2))
        conf.append((m1 / (m1 + n0), m2 / (m2 + n0)))
    # node features: 3x3 averages at the node's pixel
    px = (torch.arange(nx, device=DEV) * step).clamp(max=w - 1)
    py = (torch.arange(ny, device=DEV) * step).clamp(max=h - 1)

    def local(v):
        v = v.reshape(h, w)
        acc = sum((v[(py + dy).clamp(0, h - 1)][:, (px + dx).clamp(0, w - 1)]) / (1 + dx * dx + dy * dy)
                  for dy in (-1, 0, 1) for dx in (-1, 0, 1))
        return acc / sum(1 / (1 + dx * dx + dy * dy) for dy in (-1, 0, 1) for dx in (-1, 0, 1))

    nn = torch.stack([local(v) for v in m["f_normal"]])
    z = nn.square().sum(0)
    nn = torch.where(z > 1e-8, nn / z.clamp(min=1e-300).sqrt(), nn)
    nd, na = local(m["f_depth"]), torch.stack([local(v) for v in m["f_albedo"]])
    acc = [[0.0, 0.0] for _ in range(6)]
    ws = [[0.0, 0.0] for _ in range(6)]
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            ys, xs = torch.arange(ny, device=DEV) + dy, torch.arange(nx, device=DEV) + dx
            ok = (((ys >= 0) & (ys < ny))[:, None] & ((xs >= 0) & (xs < nx))[None, :]).double()
            at = lambda v: v[..., ys.clamp(0, ny - 1), :][..., xs.clamp(0, nx - 1)]  # noqa: E731
            wn = (((nn * at(nn)).sum(0) + 1) * 0.5).clamp(0, 1)
            wd = torch.exp(-4 * (nd - at(nd)).abs() / torch.maximum(nd.abs(), at(nd).abs()).clamp(min=1e-8))
            wa = torch.exp(-2.5 * (na - at(na)).square().sum(0).sqrt())
            base = ok * wn * wd * wa / (1 + dx * dx + dy * dy)
            for f in range(6):
                for k in range(2):
                    wt = base * at(conf[f][k]).clamp(min=_f(0.05))
                    acc[f][k] = acc[f][k] + wt * at(raw[f][k])
                    ws[f][k] = ws[f][k] + wt
    rel, rc, sc = [], [], []
    for f in range(6):
        fin = []
        for k in range(2):
            prior = torch.where(ws[f][k] > 1e-8, acc[f][k] / ws[f][k].clamp(min=1e-300), raw[f][k])
            fin.append(prior + (raw[f][k] - prior) * conf[f][k])
        r = fin[0].clamp(0, 1)
        rc.append(conf[f][0].clamp(0, 1))
        sc.append(conf[f][1])
        rel.append(r / (r + fin[1]).clamp(min=1e-8) * torch.minimum(rc[-1], sc[-1]))
    rel, rc, sc = torch.stack(rel), torch.stack(rc), torch.stack(sc)
    best = torch.zeros(ny, nx, dtype=torch.int64, device=DEV)
    top = rel[0]
    for f in range(1, 6):
        best = torch.where(top < rel[f], torch.full_like(best, f), best)
        top = torch.maximum(top, rel[f])
    pick = lambda v: v.gather(0, best[None])[0]  # noqa: E731
    all_conf = torch.minimum(pick(rc), pick(sc))
    expand = lambda v: ay.T @ v @ ax  # noqa: E731
    every = expand(top)
    xs, ys = torch.arange(w, device=DEV), torch.arange(h, device=DEV)
    gx = every[:, (xs + 1).clamp(max=w - 1)] - every[:, (xs - 1).clamp(min=0)]
    gy = every[(ys + 1).clamp(max=h - 1)] - every[(ys - 1).clamp(min=0)]
    grad = (0.5 * (gx * gx + gy * gy).sqrt()).clamp(0, 1)
    comps = torch.stack([(expand(rel[f]).clamp(0, 1) * (1 - grad)).clamp(0, 1) for f in range(6)])
    return expand(all_conf), comps


def _t_crit(df, alpha):
    df = df.clamp(min=1.0)
    a = min(max(alpha, 1e-8), 0.999999)
    z = 1.28
    for lim, v in ((0.10, 1.64), (0.05, 1.96), (0.02, 2.33), (0.01, 2.58), (0.005, 2.81), (0.001, 3.29)):
        z = v if a <= _f(lim) else z
    for level, tab in ((0.05, _T05), (0.01, _T01)):
        if abs(a - level) < 1e-4:
            t = torch.tensor([_f(v) for v in tab], dtype=torch.float64, device=DEV)
            lo, hi = df.floor().clamp(1, 30), df.ceil().clamp(1, 30)
            v0, v1 = t[lo.long() - 1], t[hi.long() - 1]
            v = v0 + (v1 - v0) * (df - lo)
            return torch.where(df < 30.5, torch.where(lo == hi, v0, v), torch.full_like(df, _f(z)))
    return torch.where(df < 30, _f(z) * (df / (df - 1).clamp(min=1)).sqrt(), torch.full_like(df, _f(z)))


def _shift(v, dy, dx, fill=0.0):
    """v at (y + dy, x + dx), `fill` outside the image."""
    out = torch.full_like(v, fill)
    h, w = v.shape[-2:]
    y0, y1, x0, x1 = max(0, -dy), min(h, h - dy), max(0, -dx), min(w, w - dx)
    if y0 < y1 and x0 < x1:
        out[..., y0:y1, x0:x1] = v[..., y0 + dy:y1 + dy, x0 + dx:x1 + dx]
    return out


def _far(di, dj, limit):
    return (di - dj).abs() / torch.maximum(di.abs(), dj.abs()).clamp(min=1e-8) > limit


def _window(m, rpd, w, h, cfg):
    img = lambda v: torch.stack(v).reshape(len(v), h, w) if isinstance(v, list) else v.reshape(h, w)  # noqa: E731
    n = img(m["n"])
    hit = img(m["hits"]) > 0
    smax2 = _f(cfg.color_sigma_max) ** 2
    var0 = torch.where(n > 1, img(m["m2"]) / (n - 1).clamp(min=1), torch.zeros_like(n))
    n1 = n.clamp(min=1)
    vm = (var0.clamp(1e-8, smax2) / n1).clamp(min=1e-8)
    rp = 1 / (n1 - 1).clamp(min=1)
    sv = torch.where(n > 1, img(m["sq"]) / (n - 1).clamp(min=1), torch.zeros_like(n)).div(n1).clamp(min=1e-8)
    ys, xs = torch.arange(h, device=DEV), torch.arange(w, device=DEV)
    avg = sum(sv[:, (ys + dy).clamp(0, h - 1)][:, :, (xs + dx).clamp(0, w - 1)] / (1 + dx * dx + dy * dy)
              for dy in (-1, 0, 1) for dx in (-1, 0, 1))
    sv = torch.maximum(sv, avg / sum(1 / (1 + dx * dx + dy * dy) for dy in (-1, 0, 1) for dx in (-1, 0, 1)))
    sm, cm = img(m["sqrt"]), img(m["color"])
    fn, fd, fa = img(m["f_normal"]), img(m["f_depth"]), img(m["f_albedo"])
    r = cfg.color_window_radius
    zero = torch.zeros_like(n)
    wsum, wsq, wvar, taken, csum = zero.clone(), zero.clone(), zero.clone(), zero.clone(), torch.zeros_like(cm)
    scale, alpha = _f(cfg.rpf_shrinkage_scale), _f(cfg.color_compat_alpha)
    for dy in range(-r, r + 1):
        for dx in range(-r, r + 1):
            at = lambda v: _shift(v, dy, dx)  # noqa: E731
            ok = _shift(hit, dy, dx, False) & ~((fn * at(fn)).sum(0) < _f(cfg.color_normal_threshold))
            ok &= ~_far(fd, at(fd), _f(cfg.color_depth_threshold))
            ok &= ~((fa - at(fa)).square().sum(0).sqrt() > _f(0.12))
            svj, rpj, nj = at(sv), at(rp), at(n1)
            vs = sv + svj
            den = sv * sv * rp + svj * svj * rpj
            df = torch.where(den > 1e-8, vs * vs / den.clamp(min=1e-30), (n1 + nj - 2).expand_as(den))
            q = ((sm - at(sm)).square() / vs.clamp(min=1e-8) / _t_crit(df, alpha).square()).amax(0)
            q = q / (1 + (scale * torch.minimum(rpd, at(rpd)).amax(0).clamp(0, 1)).clamp(0, 1))
            ok &= ~(q > 25)
            sw = 1 / (1 + dx * dx + dy * dy)
            wt = torch.where(ok, sw * torch.exp(-0.5 * q), zero)
            csum += wt * at(cm)
            wsum += wt
            wsq += wt * wt
            wvar += wt * wt * at(vm)
            if dx or dy:
                taken += (wt > 0.05 * sw).double()
    some = wsum > 1e-8
    inv = 1 / torch.where(some, wsum, torch.ones_like(wsum))
    mean = torch.where(some, csum * inv, cm)
    vnb = torch.where(some, wvar * inv * inv, vm)
    eff = wsum * wsum / wsq.clamp(min=1e-8)
    blend = torch.where((taken >= 2) & (wsum >= 1.1), (1 - 1 / eff.clamp(min=1e-300).sqrt()).clamp(0, 0.8), zero)
    a = 1 - blend
    unc = a * a * vm + blend * blend * vnb + 2 * a * blend / wsum.clamp(min=1e-8) * vm
    den = torch.where(hit, cm + (mean - cm) * blend, cm)
    return den.permute(1, 2, 0).contiguous(), torch.where(hit, unc, var0 / n1)


def _variance(m, w, h, cfg):
    n = m["n"].reshape(h, w)
    hit = m["hits"].reshape(h, w) > 0
    raw = torch.where(n > 1, m["m2"].reshape(h, w) / (n - 1).clamp(min=1), torch.zeros_like(n))
    raw = raw.clamp(1e-8, _f(cfg.adaptive_sigma_max) ** 2)
    fn, fd = torch.stack(m["f_normal"]).reshape(3, h, w), m["f_depth"].reshape(h, w)
    r, k = cfg.var_window_radius, _f(cfg.var_shrinkage_k)
    v = raw
    for _ in range(cfg.var_iterations):
        ws, acc = torch.zeros_like(v), torch.zeros_like(v)
        for dy in range(-r, r + 1):
            for dx in range(-r, r + 1):
                if dx == 0 and dy == 0:
                    continue
                vj = _shift(v, dy, dx, 1.0)
                ok = _shift(hit, dy, dx, False) & ~((fn * _shift(fn, dy, dx)).sum(0) < _f(cfg.var_normal_threshold))
                ok &= ~_far(fd, _shift(fd, dy, dx), _f(cfg.var_depth_threshold))
                ok &= ~((v - vj).abs() / (v * vj).sqrt().clamp(min=1e-8) > _f(cfg.var_compat_sigma))
                wt = ok.double() / (1 + dx * dx + dy * dy)
                ws += wt
                acc += wt * vj
        nb = torch.where(ws > 1e-8, acc / ws.clamp(min=1e-300), v)
        b = ((nb - v).clamp(min=0) / (v + nb + k).clamp(min=1e-8)).clamp(0, 1)
        v = torch.where(hit, v + (nb - v) * b, v)
    return torch.maximum(v, raw)


def _exact_frame(case, seed):
    w, h = case["width"], case["height"]
    cfg = _config(case, w, h)
    passes = []
    for planes, counts in _passes(case, seed):
        p = _decode16(planes, DEPTH_SCALE) if case.get("storage") == "fp16" else planes
        spp = case["spp"] if counts is None else 0
        n = torch.arange(w * h, device=DEV)
        pix = n.repeat_interleave(case["spp"] if counts is None else counts.long())
        p["lum"] = sum(_LUM[c] * p["radiance"][c].double() for c in range(3))
        passes.append((pix, spp, p))
    m = _moments(w * h, passes)
    hits = m["hits"].clamp(min=1)
    fn = torch.stack([v / hits for v in m["normal"]])
    z = fn.square().sum(0)
    fn = torch.where(z > 1e-8, fn / z.clamp(min=1e-300).sqrt(), fn)
    m["f_normal"], m["f_depth"], m["f_albedo"] = list(fn), m["depth"] / hits, [v / hits for v in m["albedo"]]
    conf, comps = _rpd(passes, m, w, h, cfg)
    den, unc = _window(m, comps, w, h, cfg)
    if case["kind"] == "host":
        return {"denoised": den}
    out = {"denoised": den, "uncertainty": unc, "variance_denoised": _variance(m, w, h, cfg),
           "sensitivity_confidence": conf}
    # the adaptive counts are whole numbers decided by a sequential sum: they have no nearby 64-bit value
    return {**out, "counts": None} if case["kind"] == "adaptive" else out


def _unit(v, limit=1e-8):
    z = v.square().sum(-1, keepdim=True)
    return torch.where(z > limit, v / z.clamp(min=1e-300).sqrt(), v)


def _angle(a, b):
    return torch.acos((a * b).sum(-1).clamp(-1, 1))


def _clamped(v, dy, dx):
    h, w = v.shape[:2]
    ys = (torch.arange(h, device=DEV) + dy).clamp(0, h - 1)
    xs = (torch.arange(w, device=DEV) + dx).clamp(0, w - 1)
    return v[ys][:, xs], ys, xs


def _half_inverse_square(sigma):
    return 1.0 / (2.0 * _f(sigma) ** 2)


def exact(case, seed):
    kind = case["kind"]
    if kind == "served":
        return None  # its samples are the server's own generator's, its counts the sequential allocation's
    if kind == "batch":
        return [_exact_frame(dict(kind="frame", width=w, height=h, spp=spp, scene=case["scene"], storage="fp16",
                                  knobs=case["knobs"]), seed + 1000 * k) for k, (w, h, spp) in enumerate(_frames(case))]
    if kind not in ("atrous", "bilateral"):
        return _exact_frame(case, seed)
    raw, nrm, alb = (t.double() for t in _images(case["width"], case["height"], seed))
    kc, kn, ka = (_half_inverse_square(case[s]) for s in ("sigma_c", "sigma_n", "sigma_a"))
    if kind == "atrous":
        b3 = (1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16)
        n, v = _unit(nrm), raw
        lum = torch.tensor(_LUM, dtype=torch.float64, device=DEV)
        for it in range(case["iterations"]):
            acc, ws = torch.zeros_like(v), torch.zeros_like(v[..., :1])
            for ky in range(5):
                for kx in range(5):
                    dy, dx = (ky - 2) << it, (kx - 2) << it
                    p, nj, aj = (_clamped(t, dy, dx)[0] for t in (v, n, alb))
                    e = ((v - p) @ lum).square() * kc + _angle(n, nj).square() * kn
                    wt = (b3[ky] * b3[kx] * torch.exp(-(e + (alb - aj).square().sum(-1) * ka)))[..., None]
                    acc += wt * p
                    ws += wt
            v = torch.where(ws > 1e-8, acc / ws.clamp(min=1e-300), v)
        return [v]
    kp = _half_inverse_square(case["sigma_p"])
    n, r = _unit(nrm * 2 - 1), max(1, math.ceil(3 * case["sigma_p"]))
    h, w = raw.shape[:2]
    y, x = torch.arange(h, device=DEV), torch.arange(w, device=DEV)
    acc, ws = [torch.zeros_like(raw) for _ in range(3)], [torch.zeros_like(raw[..., :1]) for _ in range(3)]
    for dy in range(-r, r + 1):
        for dx in range(-r, r + 1):
            c, ys, xs = _clamped(raw, dy, dx)
            nj, aj = _clamped(n, dy, dx)[0], _clamped(alb, dy, dx)[0]
            eg = ((ys - y).square()[:, None] + (xs - x).square()[None, :]).double() * kp
            ec = eg + (raw - c).square().sum(-1) * 0.5 * kc
            ej = ec + _angle(n, nj).square() * 1.5 * kn + (alb - aj).square().sum(-1) * ka
            for k, e in enumerate((eg, ec, ej)):
                wt = torch.exp(-e)[..., None]
                acc[k] += wt * c
                ws[k] += wt
    return [a / s for a, s in zip(acc, ws)]
