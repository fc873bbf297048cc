"""Timed cases of the metric path, through the Python entry points a program calls.

A case is one call (or one batch-plan replay) over RGBA8 image pairs.  Images are seeded 1/f noise with
the distortion the metric's workload uses (iqm_b200/synth.py states them), made on the GPU.  A program
keeps one Runtime and calls it over and over with new images, so the Runtime is made once per process;
the images, the score buffer and, for plans, the captured plan belong to each state.

Scores are FP64 sums of FP32 per-pixel values.  The programs modelled here keep their score tables in
float32, which is what `run` returns; maps are float32 as the library writes them.

Fields: metric (ssim, fsim, flip, msvd, or ssim+fsim), call (dev: images already on the GPU; host:
images and results in host memory; plan: a captured batch plan), w, h, pairs, precision (fp32, mixed,
mixed_fast), ppd (FLIP's viewing set-up), sizes (0: every pair w x h; else the seed of uneven sizes
drawn from [w, h] as both sides), map (host calls: the per-pixel map is wanted too).
"""
import math

import numpy as np
import torch

import iqm_b200

PRECISION = {"fp32": iqm_b200.IQM_FP32, "mixed": iqm_b200.IQM_MIXED, "mixed_fast": iqm_b200.IQM_MIXED_FAST}
PI = 3.141592653589  # the value the metric definitions use


def _case(name, metric, call, w, h, pairs, precision="fp32", ppd=0.0, sizes=0, want_map=False):
    return {"name": name, "metric": metric, "call": call, "w": w, "h": h, "pairs": pairs, "precision": precision,
            "ppd": ppd, "sizes": sizes, "map": want_map}


def listed():
    return [
        # one small grey pair: the reference's smallest configuration, a call inside a larger program
        _case("ssim_512", "ssim", "dev", 512, 512, 1),
        # video frames scored in batches
        _case("ssim_1080p_x16", "ssim", "dev", 1920, 1080, 16),
        # the same at 4K in the split-precision tensor-core form
        _case("ssim_4k_mixed_x4", "ssim", "dev", 3840, 2160, 4, "mixed"),
        # one still image of an image-quality database (512 x 384)
        _case("fsim_512x384", "fsim", "dev", 512, 384, 1),
        # the headline workload: 1080p RGB frames in batches
        _case("fsim_1080p_x32", "fsim", "dev", 1920, 1080, 32),
        # 720p frames, whose planes (427 x 240) are not the 1080p ones
        _case("fsim_720p_x16", "fsim", "dev", 1280, 720, 16),
        # 4K frames in the split-precision tensor-core form
        _case("fsim_4k_mixed_x16", "fsim", "dev", 3840, 2160, 16, "mixed"),
        # rendered frames at 67 pixels per degree
        _case("flip_1080p_x4", "flip", "dev", 1920, 1080, 4, ppd=67.0),
        # one odd-sized picture from host memory with its error map, at a desktop full-HD monitor
        _case("flip_map_1021x763", "flip", "host", 1021, 763, 1, ppd=38.0, want_map=True),
        # block-coded frames
        _case("msvd_1080p_x16", "msvd", "dev", 1920, 1080, 16),
        # a folder of pictures of every size, both metrics, replayed as one captured plan
        _case("uneven_plan_x24", "ssim+fsim", "plan", 256, 2048, 24, sizes=3000),
        # frames that arrive in page-locked host memory
        _case("fsim_host_1080p_x8", "fsim", "host", 1920, 1080, 8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another size, batch and option of the same work."""
    metric = rng.choice(["ssim", "fsim", "flip", "msvd", "ssim+fsim"])
    if metric == "ssim+fsim":
        return {k: v for k, v in _case("", metric, "plan", 256, rng.randint(512, 2048), rng.randint(4, 16),
                                       sizes=rng.randint(1, 1 << 20)).items() if k != "name"}
    short = _log_int(rng, 192, 2160)
    w, h = int(round(short * rng.uniform(1.0, 1.9))), short
    if rng.random() < 0.2:
        w, h = h, w
    most = max(1, min(32, 40_000_000 // (w * h)))
    pairs = _log_int(rng, 1, most)
    precision = rng.choice(["fp32", "fp32", "mixed", "mixed_fast"]) if metric in ("ssim", "fsim") else "fp32"
    ppd = rng.uniform(30.0, 90.0) if metric == "flip" else 0.0
    if metric == "flip":
        pairs = min(pairs, max(1, 12_000_000 // (w * h)))
    return {k: v for k, v in _case("", metric, "dev", w, h, pairs, precision, ppd).items() if k != "name"}


# ------------------------------------------------------------------------------------- inputs
def _sizes(case):
    if not case["sizes"]:
        return [(case["w"], case["h"])] * case["pairs"]
    rng = np.random.Generator(np.random.PCG64(case["sizes"]))
    return [(int(rng.integers(case["w"], case["h"] + 1)), int(rng.integers(case["w"], case["h"] + 1)))
            for _ in range(case["pairs"])]


def _pink(gen, c, h, w):
    fy = torch.fft.fftfreq(h, device="cuda")[:, None]
    fx = torch.fft.rfftfreq(w, device="cuda")[None, :]
    amp = torch.rsqrt((fx * fx + fy * fy).clamp_min(1e-12))
    amp[0, 0] = 0.0
    x = torch.fft.irfft2(torch.fft.rfft2(torch.randn(c, h, w, device="cuda", generator=gen)) * amp, s=(h, w))
    lo, hi = x.amin((1, 2), keepdim=True), x.amax((1, 2), keepdim=True)
    return ((x - lo) / (hi - lo) * 255.0).round().clamp(0, 255)


def _noise(gen, x, sigma):
    return torch.randn(x.shape, device="cuda", generator=gen) * sigma


def _rgba(x):
    h, w = x.shape[1:]
    out = torch.full((h, w, 4), 255, dtype=torch.uint8, device="cuda")
    out[..., :3] = x.round().clamp(0, 255).to(torch.uint8).permute(1, 2, 0)
    return out


def _pair(gen, metric, w, h):
    """(distorted, reference) RGBA8 tensors (h, w, 4) on the GPU."""
    if metric == "ssim":  # grey: noise sigma 8, 3x3 box blur
        ref = _pink(gen, 1, h, w)
        d = torch.nn.functional.pad((ref + _noise(gen, ref, 8.0))[None], (1, 1, 1, 1), mode="replicate")
        return _rgba(torch.nn.functional.avg_pool2d(d, 3, 1)[0].expand(3, h, w)), _rgba(ref.expand(3, h, w))
    ref = _pink(gen, 3, h, w)
    if metric in ("fsim", "ssim+fsim"):  # noise sigma 10 and a gain per channel
        gain = torch.rand(3, 1, 1, device="cuda", generator=gen) * 0.2 + 0.9
        return _rgba((ref + _noise(gen, ref, 10.0)) * gain), _rgba(ref)
    # 8x8-block quantisation with a step of 4..24, noise sigma 4
    step = torch.rand(3, (h + 7) // 8, (w + 7) // 8, device="cuda", generator=gen) * 20.0 + 4.0
    step = step.repeat_interleave(8, 1).repeat_interleave(8, 2)[:, :h, :w]
    return _rgba((ref / step).round() * step + _noise(gen, ref, 4.0)), _rgba(ref)


def _images(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7919 + 13)
    return [_pair(gen, case["metric"], w, h) for w, h in _sizes(case)]


# ------------------------------------------------------------------------------------- the calls
_program = {}


def _runtime():
    """The program's Runtime and the stream that it runs on."""
    if not _program:
        _program["stream"] = torch.cuda.Stream()
        _program["rt"] = iqm_b200.Runtime(torch.cuda.current_device())
        _program["rt"].set_stream(_program["stream"].cuda_stream)
    return _program["rt"], _program["stream"]


def _flip_args(case):
    # a monitor 0.6 m wide seen from 0.7 m, with the resolution that gives the wanted pixels per degree
    return iqm_b200.FLIPArguments(case["ppd"] * (180.0 / math.pi) * 0.6 / 0.7, 0.7, 0.6)


def _metric(case, rt):
    if case["metric"] == "ssim":
        m = iqm_b200.SSIM(rt)
        m.precision = PRECISION[case["precision"]]
        return m
    if case["metric"] == "fsim":
        return iqm_b200.FSIM(rt, PRECISION[case["precision"]])
    return iqm_b200.FLIP(rt) if case["metric"] == "flip" else iqm_b200.SVD(rt)


def _pinned(x):
    return torch.empty(x.shape, dtype=x.dtype, pin_memory=True).copy_(x).numpy()


def prepare(case, seed):
    rt, stream = _runtime()
    images = _images(case, seed)
    state = {"case": case, "stream": stream}
    if case["metric"] != "ssim+fsim":
        state["metric"] = _metric(case, rt)
    if case["metric"] == "flip":
        state["args"] = (_flip_args(case),)
    else:
        state["args"] = ()
    if case["call"] == "host":
        state["host"] = [(_pinned(a), _pinned(b)) for a, b in images]
        return state
    per_pair = {"ssim": 1, "fsim": 2, "flip": 1, "msvd": 1, "ssim+fsim": 3}[case["metric"]]
    scores = torch.zeros(per_pair * len(images), dtype=torch.float64, device="cuda")
    pairs = [(a.data_ptr(), b.data_ptr(), a.shape[1], a.shape[0], a.shape[1] * 4) for a, b in images]
    state.update(images=images, scores=scores, pairs=pairs, table=torch.zeros_like(scores, dtype=torch.float32))
    if case["call"] == "plan":
        torch.cuda.synchronize()  # the plan evaluates the pairs once while it is built
        state["plan"] = iqm_b200.BatchPlan(rt, iqm_b200.METRIC_SSIM | iqm_b200.METRIC_FSIM, pairs, scores.data_ptr(),
                                           precision=PRECISION[case["precision"]])
    return state


def run(state):
    case = state["case"]
    if case["call"] == "host":
        m = state["metric"]
        if case["metric"] == "flip":
            (a, b), = state["host"]
            r = m.compute_metric(a, b, *state["args"], want_map=case["map"])
            return {"score": float(r.mean_flip), "map": r.image_data}
        return np.asarray(m.compute_batch(state["host"]), np.float32)
    if case["call"] == "plan":
        state["plan"].run()
    else:
        state["metric"].compute_dev(state["pairs"], state["scores"].data_ptr(), *state["args"])
    with torch.cuda.stream(state["stream"]):
        return state["table"].copy_(state["scores"])


# ------------------------------------------------------------------------------------- work
def _plane(w, h):
    f = max(1, int(math.floor(min(w, h) / 256.0 + 0.5)))
    return f, int(math.floor(w / f + 0.5)), int(math.floor(h / f + 0.5))


def work(case):
    """Bytes: both RGBA8 images read once, the map written once; for host calls the same bytes cross the
    host link.  Operations per pixel pair: SSIM lumas (10), four window sums of two 11-tap passes (176) and
    the quotient (30); FLIP colour transforms (80), the taps of both images' six row and seven column
    filters, and the error terms (150); M-SVD per 8x8 block two bidiagonalisations (8/3 n^3) and their
    singular values (about 30 n^2 each).  FSIM: the downscale (6 per pixel), one forward and 32 inverse
    complex transforms of the plane (5 N log2 N) and about 40 operations per plane pixel and response."""
    nbytes, flops = 0, 0.0
    for w, h in _sizes(case):
        n = w * h
        for metric in case["metric"].split("+"):
            nbytes += 8 * n
            if metric == "ssim":
                flops += 216.0 * n
            elif metric == "flip":
                rf = math.ceil(3 * 0.5 * 0.082 * case["ppd"])
                rc = math.ceil(3 * math.sqrt(0.04 / (2 * PI * PI)) * case["ppd"])
                flops += n * (230.0 + 2 * 2 * (7 * (2 * rf + 1) + 6 * (2 * rc + 1)))
            elif metric == "msvd":
                flops += (w // 8) * (h // 8) * 2 * (8 / 3 * 512 + 30 * 64)
            else:
                _, w2, h2 = _plane(w, h)
                flops += 6.0 * n + w2 * h2 * (33 * 5 * math.log2(w2 * h2) + 32 * 40)
        if case["map"]:
            nbytes += 4 * n
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------------- in 64 bits
def _f64(x):
    return torch.as_tensor(x, dtype=torch.float64, device="cuda")


def _taps(plane, taps, dim, clamp):
    """sum_j taps[j + r] plane[i - j] along dim; outside the plane: the edge value (clamp) or nothing."""
    r, n = len(taps) // 2, plane.shape[dim]
    out = torch.zeros_like(plane)
    at = torch.arange(n, device="cuda")
    for j in range(-r, r + 1):
        src = at - j
        term = plane.index_select(dim, src.clamp(0, n - 1)) * float(taps[j + r])
        if not clamp:
            keep = ((src >= 0) & (src < n)).to(torch.float64)
            term = term * (keep[:, None] if dim == 0 else keep[None, :])
        out += term
    return out


def _ssim64(a, b):
    r = 5
    g = [math.exp(-k * k / (2 * 1.5 * 1.5)) for k in range(-r, r + 1)]
    la, lb = ((0.299 * x[..., 0] + 0.581 * x[..., 1] + 0.114 * x[..., 2]) / 255.0 for x in (a.double(), b.double()))
    window = lambda x: _taps(_taps(x, g, 0, False), g, 1, False)  # noqa: E731
    weight = window(torch.ones_like(la))
    ma, mb = window(la) / weight, window(lb) / weight
    va, vb = window(la * la) / weight - ma * ma, window(lb * lb) / weight - mb * mb
    cov = window(la * lb) / weight - ma * mb
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    s = (2 * ma * mb + c1) * (2 * cov + c2) / ((ma * ma + mb * mb + c1) * (va + vb + c2))
    h, w = s.shape
    return [s[r:h - r + 1, r:w - r + 1].sum() / ((w - 2 * r + 1) * (h - 2 * r + 1))]


def _freq(n):
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    return (torch.remainder(i + n // 2, n) - n // 2) / n


def _filters64(w2, h2):
    sx, sy = _freq(w2)[None, :], _freq(h2)[:, None]
    radius = torch.sqrt(sx * sx + sy * sy)
    low = 1.0 / (1.0 + (radius / 0.45) ** 30)
    theta = torch.atan2((-sy).expand(h2, w2), sx.expand(h2, w2))
    sigma = PI / 4 / 1.2
    out = []
    for o in range(4):
        d = theta - o * PI / 4
        d = torch.atan2(torch.sin(d), torch.cos(d)).abs()
        angular = torch.exp(-d * d / (2 * sigma * sigma))
        for s in range(4):
            v = torch.exp(-torch.log(radius * 6.0 * 2.0 ** s) ** 2 / (2 * math.log(0.55) ** 2)) * low
            v[0, 0] = 0.0
            out.append(v * angular)
    return torch.stack(out)


def _yiq64(x, f, w2, h2):
    h, w = x.shape[:2]
    off = f // 2
    canvas = torch.zeros(3, h2 * f + f, w2 * f + f, dtype=torch.float64, device="cuda")
    hh, ww = min(h, h2 * f + f - off), min(w, w2 * f + f - off)
    canvas[:, off:off + hh, off:off + ww] = x[:hh, :ww, :3].permute(2, 0, 1).double()
    box = canvas[:, :h2 * f, :w2 * f].reshape(3, h2, f, w2, f).sum((2, 4)) / (f * f)
    m = _f64([[0.596, -0.274, -0.322], [0.211, -0.523, 0.312], [0.299, 0.587, 0.114]])
    return (m @ box.reshape(3, -1)).reshape(3, h2, w2)


def _fsim64(a, b):
    h, w = a.shape[:2]
    f, w2, h2 = _plane(w, h)
    filters = _filters64(w2, h2)
    n, half = w2 * h2, (w2 * h2 + 1) // 2
    re = torch.fft.ifft2(filters).real.reshape(4, 4, n)[:, :, :half]
    an2 = (re * re).sum((1, 2)) * n
    cross = ((re[:, :3].sum(1) ** 2 - (re[:, :3] ** 2).sum(1)) / 2 + re[:, :3].sum(1) * re[:, 3]).sum(1) * n
    em = (filters[::4] ** 2).sum((1, 2))
    pc, grad, iq = [], [], []
    for img in (a, b):
        i, q, y = _yiq64(img, f, w2, h2)
        eo = torch.fft.ifft2(filters * torch.fft.fft2(y)).reshape(4, 4, h2, w2)
        total = eo.sum(1)
        unit = total / (total.abs() + 1e-4)
        along = eo * unit.conj()[:, None]
        energy = (along.real - along.imag.abs()).sum(1)
        amp = eo.abs().sum(1).sum(0)
        mid = (eo[:, 0].abs() ** 2).reshape(4, n).sort(1).values[:, n // 2]
        power = -mid / math.log(0.5) / em
        tau = torch.sqrt((2 * power * an2 + 4 * power * cross) / 2)
        t = (tau * math.sqrt(PI / 2) + 2 * tau * math.sqrt(2 - PI / 2)) / 1.7
        pc.append((energy - t[:, None, None]).clamp_min(0).sum(0) / amp)
        p = torch.nn.functional.pad(y, (1, 1, 1, 1))
        gx = 3 * (p[:-2, :-2] - p[:-2, 2:] + p[2:, :-2] - p[2:, 2:]) + 10 * (p[1:-1, :-2] - p[1:-1, 2:])
        gy = 3 * (p[:-2, :-2] + p[:-2, 2:] - p[2:, :-2] - p[2:, 2:]) + 10 * (p[:-2, 1:-1] - p[2:, 1:-1])
        grad.append(torch.sqrt(gx * gx + gy * gy) / 16.0)
        iq.append((i, q))
    like = lambda u, v, c: (2 * u * v + c) / (u * u + v * v + c)  # noqa: E731
    top = torch.maximum(*pc)
    s = like(*pc, 0.85) * like(*grad, 160.0) * top
    chroma = (like(iq[0][0], iq[1][0], 200.0) * like(iq[0][1], iq[1][1], 200.0)).abs() ** 0.03
    return [s.sum() / top.sum(), (s * chroma).sum() / top.sum()]


_RGB_TO_XYZ = np.array([[10135552 / 24577794, 8788810 / 24577794, 4435075 / 24577794],
                        [2613072 / 12288897, 8788810 / 12288897, 887015 / 12288897],
                        [1425312 / 73733382, 8788810 / 73733382, 70074185 / 73733382]], np.float32).astype(np.float64)
_XYZ_TO_RGB = np.array([[3.241003275, -1.537398934, -0.498615861], [-0.969224334, 1.875930071, 0.041554224],
                        [0.055639423, -0.204011202, 1.057148933]], np.float32).astype(np.float64)


def _hunt64(xyz):
    delta = 6.0 / 29.0
    f = torch.where(xyz > 0.008856, xyz.clamp_min(0) ** (1 / 3), xyz / (3 * delta * delta) + 4.0 / 29.0)
    light = 116 * f[1] - 16
    return torch.stack([light, 500 * (f[0] - f[1]) * 0.01 * light, 200 * (f[1] - f[2]) * 0.01 * light])


def _hyab64(u, v):
    return (u[0] - v[0]).abs() + torch.sqrt((u[1] - v[1]) ** 2 + (u[2] - v[2]) ** 2)


def _flip_map64(a, b, args):
    res, dist, width = (np.float32(v) for v in (args.monitor_resolution_x, args.monitor_distance, args.monitor_width))
    ppd = float(np.float32(dist * np.float32(res / width))) * (math.pi / 180.0)
    to_xyz, to_rgb, white = _f64(_RGB_TO_XYZ), _f64(_XYZ_TO_RGB), _f64(_RGB_TO_XYZ.sum(1))[:, None, None]
    mix = lambda m, x: (m @ x.reshape(3, -1)).reshape(x.shape)  # noqa: E731
    k = 2 * math.ceil(3 * 0.5 * 0.082 * ppd) + 1
    ppd = float(np.float32(ppd))
    sd = 0.5 * 0.082 * ppd
    x = np.arange(k) - math.ceil(3 * sd)
    g = np.exp(-x * x / (2 * sd * sd))
    feature = []
    for t in (g, -x * g, (x * x / (sd * sd) - 1) * g):
        pos, neg = t[t > 0].sum(), -t[t < 0].sum()
        feature.append(np.where(t > 0, t / pos, t / (neg if neg > 0 else 1.0)))
    rc = math.ceil(3 * math.sqrt(0.04 / (2 * PI * PI)) * ppd)
    d = (np.arange(-rc, rc + 1) / ppd) ** 2
    csf = []
    for p in np.array([(1, 0.0047, 0, 1e-5), (1, 0.0053, 0, 1e-5), (34.1, 0.04, 13.5, 0.025)], np.float32).astype(np.float64):
        v = p[0] * np.sqrt(PI / p[1]) * np.exp(-PI * PI * d / p[1]) + p[2] * np.sqrt(PI / p[3]) * np.exp(-PI * PI * d / p[3])
        csf.append(v / v.sum())
    edges, points, lab = [], [], []
    for img in (a, b):
        c = img[..., :3].permute(2, 0, 1).double() / 255.0
        xyz = mix(to_xyz, torch.where(c > 0.04045, ((c + 0.055) / 1.055) ** 2.4, c / 12.92)) / white
        light = xyz[1]
        rows = [_taps(light, t, 1, True) for t in feature]
        edges.append(torch.hypot(_taps(rows[1], feature[0], 0, True), _taps(rows[0], feature[1], 0, True)))
        points.append(torch.hypot(_taps(rows[2], feature[0], 0, True), _taps(rows[0], feature[2], 0, True)))
        ycc = (116 * xyz[1] - 16, 500 * (xyz[0] - xyz[1]), 200 * (xyz[1] - xyz[2]))
        f = [_taps(_taps(p, t, 1, True), t, 0, True) for p, t in zip(ycc, csf)]
        yy = (f[0] + 16) / 116
        lin = mix(to_rgb, torch.stack([yy + f[1] / 500, yy, yy - f[2] / 200]) * white).clamp(0, 1)
        lab.append(_hunt64(mix(to_xyz, lin) / white))
    error = torch.sqrt(torch.maximum((edges[0] - edges[1]).abs(), (points[0] - points[1]).abs()) / math.sqrt(2))
    ends = [_hunt64(mix(to_xyz, _f64(v)[:, None, None]) / white) for v in ([0.0, 1.0, 0.0], [0.0, 0.0, 1.0])]
    cmax = _hyab64(*ends) ** 0.7
    de = _hyab64(*lab) ** 0.7
    dec = torch.where(de < 0.4 * cmax, 0.95 / (0.4 * cmax) * de, 0.95 + (de - 0.4 * cmax) / (0.6 * cmax) * 0.05)
    return dec ** (1 - error)


def _msvd64(a, b):
    h, w = a.shape[:2]
    vx, vy = (w - 1) // 8, (h - 1) // 8
    s = []
    for img in (a, b):
        r, g, bl = (img[:8 * vy, :8 * vx, i].to(torch.int32) for i in range(3))
        grey = (r * 9798 + g * 19235 + bl * 3735 + 16384) >> 15
        m = grey.double().reshape(vy, 8, vx, 8).permute(0, 2, 1, 3).reshape(-1, 8, 8)
        # the Gram matrix of whole numbers is exact in 64 bits
        s.append(torch.linalg.eigvalsh((m.mT @ m).cpu()).clamp_min(0).sqrt().cuda())
    n = (w // 8) * (h // 8)
    d = torch.zeros(n, dtype=torch.float64, device="cuda")
    d[:vx * vy] = torch.sqrt(((s[0] - s[1]) ** 2).sum(1))
    return [(d - d.sort().values[n // 2]).abs().sum() / n]


def exact(case, seed):
    images = _images(case, seed)
    if case["metric"] == "flip":
        args = _flip_args(case)
        maps = [_flip_map64(a, b, args) for a, b in images]
        if case["call"] == "host":
            return {"score": float(maps[0].mean()), "map": maps[0].cpu().numpy()}
        return torch.stack([m.mean() for m in maps])
    scores = {"ssim": _ssim64, "fsim": _fsim64, "msvd": _msvd64}
    out = [torch.stack([v for a, b in images for v in scores[m](a, b)]) for m in case["metric"].split("+")]
    out = torch.cat(out)
    return out.reshape(-1, 2).cpu().numpy() if case["call"] == "host" else out
