"""What a user of the scorer has it do, as timed cases.

A case is one call (or one list of calls) through `vqm_b200.ss2`: a pair
scored by a pipeline, candidates scored against an uploaded reference, a list
of pairs scored by a batch, images in host memory scored through a pool.
`exact` states the same metric in double precision with torch alone.

Content: seeded textures (eight plane waves a channel, a gradient and a few
flat rectangles), distorted by noise, a Gaussian blur or 8x8 block
quantisation, encoded in the case's pixel format.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

from vqm_b200 import ss2

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"

# name: samples' bits, colour family, chroma subsampling, alpha, curve.
FORMATS = {
    "rgb8": dict(bits=8, yuv=False, sub=0, alpha=False, curve="srgb"),
    "rgba8": dict(bits=8, yuv=False, sub=0, alpha=True, curve="srgb"),
    "rgb16": dict(bits=16, yuv=False, sub=0, alpha=False, curve="srgb"),
    "yuv420p8": dict(bits=8, yuv=True, sub=1, alpha=False, curve="bt709"),
    "yuv420p10": dict(bits=10, yuv=True, sub=1, alpha=False, curve="bt709"),
    "yuv444p10": dict(bits=10, yuv=True, sub=0, alpha=False, curve="bt709"),
    "pq420p10": dict(bits=10, yuv=True, sub=1, alpha=False, curve="pq"),
    "hlg420p10": dict(bits=10, yuv=True, sub=1, alpha=False, curve="hlg"),
}
# A pair's cost per pixel next to an 8-bit RGB pair's, for the sizes of drawn
# cases.
COST = {"rgb8": 1.0, "yuv420p8": 1.4, "yuv420p10": 1.4, "yuv444p10": 1.4,
        "rgba8": 9.0, "rgb16": 9.0, "pq420p10": 9.0, "hlg420p10": 9.0}
MOST = 120e6  # pixels times COST of a drawn case
MIXED = ((640, 360), (1280, 720), (1920, 1080), (2560, 1440), (3840, 2160))
MIXED_SHARE = (0.2, 0.3, 0.3, 0.1, 0.1)
BACKGROUND = 0.5


def listed():
    return [
        # A thumbnail or an icon compared as it is saved: the smallest call.
        dict(name="still_256_rgb8", call="pair", format="rgb8", width=256, height=256),
        # One decoded 1080p frame pair a call, frames already on the device.
        dict(name="frame_1080p_rgb8", call="pair", format="rgb8", width=1920, height=1080),
        # Scoring a clip or a test set of equal sizes in one list.
        dict(name="list_1080p_rgb8_x64", call="list", format="rgb8", width=1920, height=1080,
             pairs=64, uneven=False, half=False),
        # A ladder of renditions or a mixed test set: every pair its own size.
        dict(name="list_uneven_yuv420p10_x64", call="list", format="yuv420p10", width=3840,
             height=2160, pairs=64, uneven=True, half=False),
        # A 4K stream from a hardware decoder, frame by frame.
        dict(name="frame_4k_yuv420p10", call="pair", format="yuv420p10", width=3840, height=2160),
        # The same of an HDR10 stream (ST 2084, BT.2020).
        dict(name="frame_4k_pq420p10", call="pair", format="pq420p10", width=3840, height=2160),
        # A piece of an HLG broadcast.
        dict(name="list_1080p_hlg420p10_x16", call="list", format="hlg420p10", width=1920,
             height=1080, pairs=16, uneven=False, half=False),
        # Web images with transparency (odd sizes, as such images have).
        dict(name="list_rgba8_1001x667_x8", call="list", format="rgba8", width=1001, height=667,
             pairs=8, uneven=False, half=False),
        # A photograph developed to 16 bits: the largest still.
        dict(name="photo_rgb16_3999x2667", call="pair", format="rgb16", width=3999, height=2667),
        # An encoder search: candidates against one reference kept on the device.
        dict(name="search_720p_yuv420p8_x4", call="search", format="yuv420p8", width=1280,
             height=720, pairs=4),
        # Many pairs with the pyramid kept in half precision to save memory.
        dict(name="list_1080p_rgb8_half_x32", call="list", format="rgb8", width=1920, height=1080,
             pairs=32, uneven=False, half=True),
        # Decoded images of mixed sizes and formats in host memory, through a pool.
        dict(name="pool_host_mixed_x32", call="pool", pairs=32),
    ]


def draw(rng: random.Random):
    call = rng.choices(("pair", "list", "search", "pool"), (0.4, 0.4, 0.15, 0.05))[0]
    if call == "pool":
        return dict(call="pool", pairs=rng.randint(4, 31))
    fmt = rng.choice(sorted(FORMATS))
    w = round(math.exp(rng.uniform(math.log(160), math.log(4096))))
    h = max(120, min(2304, round(w * rng.uniform(0.45, 0.9))))
    if FORMATS[fmt]["sub"]:
        w, h = w + w % 2, h + h % 2
    case = dict(call=call, format=fmt, width=w, height=h)
    if call == "pair":
        return case
    room = MOST / (COST[fmt] * w * h)
    if call == "search":
        return dict(case, pairs=max(1, min(8, int(room), rng.randint(2, 8))))
    pairs = round(math.exp(rng.uniform(math.log(2), math.log(64))))
    return dict(case, pairs=max(1, min(pairs, int(room))), uneven=rng.random() < 0.4,
                half=rng.random() < 0.15)


# --- inputs -------------------------------------------------------------------


def _jobs(case, seed):
    """(format, width, height, seed) of each pair (the search's first image is
    every pair's original)."""
    rng = random.Random(1000003 * seed + 17)
    if case["call"] == "pool":
        # The same sizes whichever the seed (the shares dealt out in turn), in
        # an order of the seed's own.
        n = case["pairs"]
        sizes = []
        for size, share in zip(MIXED, MIXED_SHARE):
            sizes += [size] * round(share * n)
        sizes = (sizes + [MIXED[1]] * n)[:n]
        rng.shuffle(sizes)
        return [(("rgb8", "yuv420p10")[i % 2], w, h, 7919 * seed + i)
                for i, (w, h) in enumerate(sizes)]
    fmt, w, h = case["format"], case["width"], case["height"]
    n = case.get("pairs", 1)
    if not case.get("uneven"):
        return [(fmt, w, h, 7919 * seed + i) for i in range(n)]
    jobs = []
    sizes = random.Random(n)  # the sizes are the case's, the pixels the seed's
    for i in range(n):
        pw = max(64, round(w * sizes.uniform(1 / 12, 1)))
        ph = max(64, round(h * sizes.uniform(1 / 12, 1)))
        if FORMATS[fmt]["sub"]:
            pw, ph = pw + pw % 2, ph + ph % 2
        jobs.append((fmt, pw, ph, 7919 * seed + i))
    return jobs


def _texture(w, h, rng):
    """[3, h, w] in 0..1."""
    x = torch.arange(w, device=DEVICE, dtype=torch.float32)
    y = torch.arange(h, device=DEVICE, dtype=torch.float32)
    rows, cols = [], []
    for _ in range(24):
        theta, phase = rng.uniform(0, math.pi), rng.uniform(0, 2 * math.pi)
        k = 2 * math.pi / rng.uniform(4, 64)
        amp = rng.uniform(0.3, 1.0)
        a, b = k * math.cos(theta) * x, k * math.sin(theta) * y + phase
        cols += [amp * a.sin(), amp * a.cos()]
        rows += [b.cos(), b.sin()]
    cols = torch.stack(cols).view(3, 16, w)
    rows = torch.stack(rows).view(3, 16, h)
    img = torch.bmm(rows.transpose(1, 2), cols)
    for c in range(3):
        img[c] += rng.uniform(-2, 2) * x / w + (rng.uniform(-2, 2) * y / h)[:, None]
    lo, hi = img.amin((1, 2), keepdim=True), img.amax((1, 2), keepdim=True)
    img = (img - lo) / (hi - lo)
    for _ in range(16):
        rw, rh = rng.randint(2, max(3, w // 6)), rng.randint(2, max(3, h // 6))
        x0, y0 = rng.randint(0, max(0, w - rw)), rng.randint(0, max(0, h - rh))
        for c in range(3):
            img[c, y0:y0 + rh, x0:x0 + rw] = rng.random()
    return img


def _smooth(img, sigma):
    r = max(1, math.ceil(3 * sigma))
    k = torch.exp(-0.5 * (torch.arange(-r, r + 1, device=DEVICE, dtype=torch.float32) / sigma) ** 2)
    k = k / k.sum()
    h, w = img.shape[1:]
    p = torch.nn.functional.pad(img[None], (r, r, r, r), mode="replicate")[0]
    p = sum(k[i] * p[:, :, i:i + w] for i in range(2 * r + 1))
    return sum(k[i] * p[:, i:i + h] for i in range(2 * r + 1))


def _distort(img, rng, gen):
    kind = rng.randrange(3)
    if kind == 0:
        noise = torch.randn(img.shape, generator=gen, device=DEVICE)
        return img + noise * (rng.uniform(1, 8) / 255)
    if kind == 1:
        return _smooth(img, rng.uniform(0.5, 3))
    step = rng.uniform(4, 32) / 255
    c, h, w = img.shape
    pad = torch.nn.functional.pad(img[None], (0, -w % 8, 0, -h % 8), mode="replicate")[0]
    blocks = pad.view(c, pad.shape[1] // 8, 8, pad.shape[2] // 8, 8)
    mean = blocks.mean((2, 4), keepdim=True)
    return (blocks - mean + step * torch.round(mean / step)).reshape(pad.shape)[:, :h, :w]


def _luma(curve):
    return (0.2627, 0.0593) if curve in ("pq", "hlg") else (0.2126, 0.0722)


def _codes(img, fmt, alpha):
    """The planes' integer samples."""
    f = FORMATS[fmt]
    img = img.clamp(0, 1)
    if not f["yuv"]:
        top = (1 << f["bits"]) - 1
        planes = [torch.round(img[c] * top) for c in range(3)]
        if f["alpha"]:
            planes.append(torch.round(alpha * top))
        return planes
    if f["curve"] == "pq":
        img = img * 0.75  # up to about 1000 cd/m2
    kr, kb = _luma(f["curve"])
    y = kr * img[0] + (1 - kr - kb) * img[1] + kb * img[2]
    cb, cr = (img[2] - y) / (2 - 2 * kb), (img[0] - y) / (2 - 2 * kr)
    if f["sub"]:
        cb, cr = (torch.nn.functional.avg_pool2d(p[None, None], 2)[0, 0] for p in (cb, cr))
    s = 1 << (f["bits"] - 8)
    return [torch.round(16 * s + 219 * s * y), torch.round(128 * s + 224 * s * cb),
            torch.round(128 * s + 224 * s * cr)]


def _pair_codes(job):
    fmt, w, h, seed = job
    rng = random.Random(seed)
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    ref = _texture(w, h, rng)
    alpha = None
    if FORMATS[fmt]["alpha"]:
        # A soft-edged cut-out: opaque inside, clear outside.
        x = torch.linspace(-1, 1, w, device=DEVICE)
        y = torch.linspace(-1, 1, h, device=DEVICE)[:, None]
        alpha = ((rng.uniform(0.7, 1.2) - (x * x + y * y).sqrt()) * 8).clamp(0, 1)
    return _codes(ref, fmt, alpha), _codes(_distort(ref, rng, gen), fmt, alpha)


def _search_codes(case, seed):
    """The search's original and its candidates' samples."""
    jobs = _jobs(case, seed)
    original = _pair_codes(jobs[0])[0]
    fmt, w, h, s = jobs[0]
    ref = _texture(w, h, random.Random(s))
    out = []
    for i in range(len(jobs)):
        gen = torch.Generator(device=DEVICE)
        gen.manual_seed(s + i)
        out.append(_codes(_distort(ref, random.Random(s + 31 * i + 1), gen), fmt, None))
    return original, out


def _format(fmt):
    f = FORMATS[fmt]
    kind = ss2.PixelType.Byte if f["bits"] == 8 else ss2.PixelType.Word
    if not f["yuv"]:
        return ss2.ImageFormat(type=kind, alpha=ss2.AlphaType.Straight if f["alpha"]
                               else ss2.AlphaType.None_)
    hdr = f["curve"] in ("pq", "hlg")
    return ss2.ImageFormat(
        type=kind, family=ss2.ColorFamily.Yuv, range=ss2.PixelRange.Limited,
        matrix=ss2.MatrixCoefficients.Bt2020Ncl if hdr else ss2.MatrixCoefficients.Bt709,
        transfer={"pq": ss2.TransferCharacteristics.St2084,
                  "hlg": ss2.TransferCharacteristics.AribB67,
                  "bt709": ss2.TransferCharacteristics.Bt709}[f["curve"]],
        primaries=ss2.ColorPrimaries.Bt2020 if hdr else ss2.ColorPrimaries.Bt709,
        subsample_w=f["sub"], subsample_h=f["sub"], depth=f["bits"] if f["bits"] != 8 else 0)


def _bytes(planes, fmt):
    """The packed image: each plane on a 4-byte boundary."""
    wide = FORMATS[fmt]["bits"] > 8
    parts = []
    for p in planes:
        b = p.to(torch.int32).to(torch.uint16 if wide else torch.uint8).contiguous().view(-1)
        b = b.view(torch.uint8)
        parts.append(b)
        if b.numel() % 4:
            parts.append(torch.zeros(4 - b.numel() % 4, dtype=torch.uint8, device=DEVICE))
    return torch.cat(parts)


def _device_image(planes, fmt):
    data = _bytes(planes, fmt)
    h, w = planes[0].shape
    return ss2.DeviceImage.packed(w, h, _format(fmt), data.data_ptr(), owner=data)


def _host_image(planes, fmt):
    data = _bytes(planes, fmt)
    pinned = torch.empty(data.shape, dtype=torch.uint8, pin_memory=torch.cuda.is_available())
    pinned.copy_(data)
    h, w = planes[0].shape
    return ss2.Image(w, h, _format(fmt), pinned.numpy())


def prepare(case, seed):
    call = case["call"]
    if call == "search":
        original, candidates = _search_codes(case, seed)
        pipe = ss2.Ssimulacra2Pipeline(case["width"], case["height"])
        reference = pipe.upload(_device_image(original, case["format"]))
        images = [_device_image(c, case["format"]) for c in candidates]
        torch.cuda.synchronize()
        return dict(call=call, pipe=pipe, reference=reference, images=images)
    image = _host_image if call == "pool" else _device_image
    pairs = []
    for job in _jobs(case, seed):
        o, d = _pair_codes(job)
        pairs.append((image(o, job[0]), image(d, job[0])))
    torch.cuda.synchronize()
    if call == "pair":
        return dict(call=call, pair=pairs[0],
                    pipe=ss2.Ssimulacra2Pipeline(case["width"], case["height"]))
    if call == "list":
        return dict(call=call, pairs=pairs, batch=ss2.Ssimulacra2Batch(half_planes=case["half"]))
    return dict(call=call, pairs=pairs, pool=ss2.Ssimulacra2Pool(workers=2, chunk=8))


def run(state):
    call = state["call"]
    if call == "pair":
        results = [state["pipe"].compute(*state["pair"])]
    elif call == "search":
        results = [state["pipe"].compute(state["reference"], d) for d in state["images"]]
    elif call == "list":
        results = state["batch"].compute_many(state["pairs"])
    else:
        results = state["pool"].compute_many(state["pairs"])
    return dict(norms=np.concatenate([r.norms.reshape(-1) for r in results]),
                scores=np.array([r.score() for r in results]))


# --- the work of a pass ---------------------------------------------------------


def _plan(w, h):
    """The levels' sizes."""
    sizes = []
    while len(sizes) < 6 and w >= 8 and h >= 8:
        if sizes:
            w, h = (w + 1) // 2, (h + 1) // 2
        sizes.append((w, h))
    return sizes


def _kept(channel, scale, scales):
    at = (channel * scales + scale) * 6
    return max(WEIGHTS[at:at + 6]) > 0.01


def _image_bytes(fmt, w, h):
    f = FORMATS[fmt]
    planes = 4 if f["alpha"] else 3
    samples = w * h * (1 + 2 / (1 << 2 * f["sub"])) if f["yuv"] else w * h * planes
    return samples * (1 if f["bits"] == 8 else 2)


def work(case):
    """Bytes: each image read once, the norms and the score written. Operations:
    per kept pixel of a pair the five 13-tap blurs along both axes and the maps
    (130 multiply-adds and about 34 others), per pixel of a pyramid level and
    image the opsin mix, two to three cube roots and the average (about 60), per
    sample the transfer curve (about 25)."""
    jobs = _jobs(case, 1)
    total, flops = 0.0, 0.0
    images = 0
    for i, (fmt, w, h, _) in enumerate(jobs):
        n = 1 if case["call"] == "search" else 2  # the reference is kept between calls
        images += n
        total += n * _image_bytes(fmt, w, h) + 8 * 109
        plan = _plan(w, h)
        kept = sum(pw * ph for s, (pw, ph) in enumerate(plan) for c in range(3)
                   if _kept(c, s, len(plan)))
        flops += 294 * kept + n * (60 * sum(pw * ph for pw, ph in plan) + 75 * w * h)
    return dict(bytes=total, flops=flops)


# --- the metric in double precision ------------------------------------------------

# The weighted sum's weights, row channel * scales + scale: mean and 4-norm
# columns of the SSIM', ringing and blurring maps (SSIM' mean, ringing mean,
# blurring mean, then their 4-norms).
WEIGHTS = [
    0.0, 0.0007376606707406586, 0.0, 0.0, 0.0007793481682867309, 0.0,
    0.0, 0.0004371155730107379, 0.0, 1.1041726426657346, 0.00066284834129271, 0.00015231632783718752,
    0.0, 0.0016406437456599754, 0.0, 1.8422455520539298, 11.441172603757666, 0.0,
    0.0007989109436015163, 0.000176816438078653, 0.0, 1.8787594979546387, 10.94906990605142, 0.0,
    0.0007289346991508072, 0.9677937080626833, 0.0, 0.00014003424285435884, 0.9981766977854967,
    0.00031949755934435053,
    0.0004550992113792063, 0.0, 0.0, 0.0013648766163243398, 0.0, 0.0,
    0.0, 0.0, 0.0, 7.466890328078848, 0.0, 17.445833984131262,
    0.0006235601634041466, 0.0, 0.0, 6.683678146179332, 0.00037724407979611296, 1.027889937768264,
    225.20515300849274, 0.0, 0.0, 19.213238186143016, 0.0011401524586618361, 0.001237755635509985,
    176.39317598450694, 0.0, 0.0, 24.43300999870476, 0.28520802612117757, 0.0004485436923833408,
    0.0, 0.0, 0.0, 34.77906344483772, 44.835625328877896, 0.0,
    0.0, 0.0, 0.0, 0.0, 0.0, 0.0,
    0.0, 0.0008680556573291698, 0.0, 0.0, 0.0, 0.0,
    0.0, 0.0005313191874358747, 0.0, 0.00016533814161379112, 0.0, 0.0,
    0.0, 0.0, 0.0, 0.0004179171803251336, 0.0017290828234722833, 0.0,
    0.0020827005846636437, 0.0, 0.0, 8.826982764996862, 23.19243343998926, 0.0,
    95.1080498811086, 0.9863978034400682, 0.9834382792465353, 0.0012286405048278493,
    171.2667255897307, 0.9807858872435379,
    0.0, 0.0, 0.0, 0.0005130064588990679, 0.0, 0.00010854057858411537,
]


def _rgb_to_xyz(primaries):
    xyz = np.array([[x / y, 1.0, (1 - x - y) / y] for x, y in primaries]).T
    white = np.array([0.3127 / 0.3290, 1.0, (1 - 0.3127 - 0.3290) / 0.3290])
    return xyz * np.linalg.solve(xyz, white)


def _mix(m, planes):
    return [sum(float(m[r][c]) * planes[c] for c in range(3)) for r in range(3)]


def _linear(planes, fmt):
    """Linear BT.709 light of the samples, [3] of [h, w] float64."""
    f = FORMATS[fmt]
    p = [x.double() for x in planes]
    curve = f["curve"]
    if not f["yuv"]:
        top = float((1 << f["bits"]) - 1)
        rgb = [x / top for x in p[:3]]
        if f["alpha"]:
            a = p[3] / top
            rgb = [a * x + (1 - a) * BACKGROUND for x in rgb]
        return [torch.where(x <= 0.04045, x / 12.92,
                            ((x.clamp(min=0.04045) + 0.055) / 1.055) ** 2.4) for x in rgb]
    s = float(1 << (f["bits"] - 8))
    y = (p[0] - 16 * s) / (219 * s)
    cb, cr = ((x - 128 * s) / (224 * s) for x in p[1:])
    if f["sub"]:
        cb, cr = (_upsampled(x, y.shape) for x in (cb, cr))
    kr, kb = _luma(curve)
    kg = 1 - kr - kb
    r, b = y + (2 - 2 * kr) * cr, y + (2 - 2 * kb) * cb
    rgb = [r, (y - kr * r - kb * b) / kg, b]
    if curve == "bt709":
        return [x.clamp(min=0) ** 2.4 for x in rgb]
    if curve == "pq":
        m1, m2, c1, c2, c3 = 0.1593017578125, 78.84375, 0.8359375, 18.8515625, 18.6875
        v = [x.clamp(min=0) ** (1 / m2) for x in rgb]
        rgb = [100 * ((x - c1).clamp(min=0) / (c2 - c3 * x)) ** (1 / m1) for x in v]
    else:
        v = [x.clamp(min=0) for x in rgb]
        v = [torch.where(x <= 0.5, x * x / 3,
                         (torch.exp((x - 0.55991073) / 0.17883277) + 0.28466892) / 12) for x in v]
        gain = 10 * (kr * v[0] + kg * v[1] + kb * v[2]).clamp(min=1e-38) ** 0.2
        rgb = [x * gain for x in v]
    from2020 = np.linalg.solve(_rgb_to_xyz(((0.640, 0.330), (0.300, 0.600), (0.150, 0.060))),
                               _rgb_to_xyz(((0.708, 0.292), (0.170, 0.797), (0.131, 0.046))))
    return _mix(from2020, rgb)


def _upsampled(c, shape):
    """4:2:0 chroma at the luma samples, bilinear: sited left (on the even
    columns) and midway between the rows."""
    h, w = shape
    right = torch.cat([c[:, 1:], c[:, -1:]], 1)
    wide = torch.stack([c, 0.5 * (c + right)], 2).reshape(c.shape[0], w)
    above = torch.cat([wide[:1], wide[:-1]], 0)
    below = torch.cat([wide[1:], wide[-1:]], 0)
    return torch.stack([0.25 * above + 0.75 * wide, 0.75 * wide + 0.25 * below], 1).reshape(h, w)


def _xyb(rgb):
    bias = 0.0037930732552754493
    opsin = ((0.30, 1 - 0.078 - 0.30, 0.078), (0.23, 1 - 0.078 - 0.23, 0.078),
             (0.24342268924547819, 0.20476744424496821, 1 - 0.24342268924547819
              - 0.20476744424496821))
    l, m, s = ((x + bias).clamp(min=0) ** (1 / 3) - bias ** (1 / 3) for x in _mix(opsin, rgb))
    return (14 * 0.5 * (l - m) + 0.42, 0.5 * (l + m) + 0.01, s - 0.5 * (l + m) + 0.55)


def _blur(x):
    w = torch.exp(-0.5 * (torch.arange(-6, 7, device=DEVICE, dtype=torch.float64) / 1.5) ** 2)
    w = (w / w.sum()).tolist()
    n, h, wd = x.shape
    p = torch.nn.functional.pad(x, (6, 6))
    x = sum(w[i] * p[:, :, i:i + wd] for i in range(13))
    p = torch.nn.functional.pad(x, (0, 0, 6, 6))
    return sum(w[i] * p[:, i:i + h] for i in range(13))


def _halved(x):
    h, w = x.shape
    if w % 2:
        x = torch.cat([x, x[:, -1:]], 1)
    if h % 2:
        x = torch.cat([x, x[-1:]], 0)
    return 0.25 * (x[0::2, 0::2] + x[0::2, 1::2] + x[1::2, 0::2] + x[1::2, 1::2])


def _both_norms(x):
    return x.mean(), (x ** 4).mean() ** 0.25


def _metric(original, distorted, fmt):
    """The 18 norms a scale, and the score."""
    a, b = _linear(original, fmt), _linear(distorted, fmt)
    plan = _plan(a[0].shape[1], a[0].shape[0])
    norms = torch.zeros((len(plan), 18), dtype=torch.float64, device=DEVICE)
    for s in range(len(plan)):
        if s:
            a, b = [_halved(x) for x in a], [_halved(x) for x in b]
        keep = [c for c in range(3) if _kept(c, s, len(plan))]
        if not keep:
            continue
        xa, xb = _xyb(a), _xyb(b)
        for c in keep:
            i1, i2 = xa[c], xb[c]
            mu1, mu2, s11, s22, s12 = _blur(torch.stack([i1, i2, i1 * i1, i2 * i2, i1 * i2]))
            num = (1 - (mu1 - mu2) ** 2) * (2 * (s12 - mu1 * mu2) + 0.0009)
            den = (s11 - mu1 * mu1) + (s22 - mu2 * mu2) + 0.0009
            ssim = (1 - num / den).clamp(min=0)
            edge = (1 + (i2 - mu2).abs()) / (1 + (i1 - mu1).abs()) - 1
            norms[s, 2 * c], norms[s, 2 * c + 1] = _both_norms(ssim)
            norms[s, 6 + 4 * c], norms[s, 7 + 4 * c] = _both_norms(edge.clamp(min=0))
            norms[s, 8 + 4 * c], norms[s, 9 + 4 * c] = _both_norms((-edge).clamp(min=0))
    norms = norms.cpu().numpy()
    error = 0.0
    for c in range(3):
        for s in range(len(plan)):
            w = WEIGHTS[(c * len(plan) + s) * 6:][:6]
            n = norms[s]
            error += (w[0] * n[2 * c] + w[1] * n[6 + 4 * c] + w[2] * n[8 + 4 * c]
                      + w[3] * n[2 * c + 1] + w[4] * n[7 + 4 * c] + w[5] * n[9 + 4 * c])
    error *= 0.9562382616834844
    mapped = (2.326765642916932 * error - 0.020884521182843837 * error ** 2
              + 6.248496625763138e-05 * error ** 3)
    return norms, 100.0 - 10.0 * mapped ** 0.6276336467831387 if mapped > 0 else 100.0


def exact(case, seed):
    if case["call"] == "search":
        original, candidates = _search_codes(case, seed)
        done = [_metric(original, c, case["format"]) for c in candidates]
    else:
        done = []
        for job in _jobs(case, seed):
            o, d = _pair_codes(job)
            done.append(_metric(o, d, job[0]))
    return dict(norms=np.concatenate([n.reshape(-1) for n, _ in done]),
                scores=np.array([s for _, s in done]))
