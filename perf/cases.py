"""Timed cases of the BIMP keypoint detector: what its users call, over the range of sizes they call it with.

Kinds of case (`kind`):

* ``detect``     getKeypoints() on an image in device memory, its result kept in the program's own matrix;
* ``queue``      bimp_detect_device_async(): the same on a stream, nothing waited for (a device-resident pipeline);
* ``host``       detect_host(): a host image in, host records out, one call per frame;
* ``stream``     Pipeline push/pop: host frames with several in flight;
* ``batch``      Batch load, run and keypoints(): images of mixed sizes in one replay;
* ``responses``  Context.loadImage() and getResponses(): the summed maps D and S of every scale;
* ``adjoint``    Adjoint.forward() and backward(): loss, image gradient and parameter gradients.

Sizes and wavelength banks are those of the package's workloads (vga, hd, mixed, uhd, adjoint), of its tests, and odd
sizes between them.  Images are seeded 1/f^2 noise with filled polygons, the content model of ``bimp_b200.synth``,
made on the device.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "cuda-bimp_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

NUM_ORI = 8


def bank(n: int) -> str:
    """The first n wavelengths 4 * 2^(k/2), accumulated in float32 (makeLambdasLog with two scales per octave)."""
    lam, out = np.float32(4.0), []
    for _ in range(n):
        out.append(repr(float(lam)))
        lam = np.float32(lam * np.float32(2.0 ** 0.5))
    return ",".join(out)


VGA = "4,8,16,32"


def lambdas_of(case) -> list:
    return [float(x) for x in str(case["lambdas"]).split(",")]


def listed():
    return [
        # a thumbnail: nothing but launches and the latency of one wave
        {"name": "detect_160x120", "kind": "detect", "w": 160, "h": 120, "lambdas": bank(3), "capacity": 8000},
        # an odd size with wavelengths outside the built-in offset sets (the stencil's general path)
        {"name": "detect_333x277_custom", "kind": "detect", "w": 333, "h": 277, "lambdas": "4,6,11", "capacity": 8000},
        # a webcam frame, four octaves
        {"name": "detect_vga", "kind": "detect", "w": 640, "h": 480, "lambdas": VGA, "capacity": 16384},
        # the headline workload: 1080p frames, 8 scales
        {"name": "queue_hd", "kind": "queue", "w": 1920, "h": 1080, "lambdas": bank(8), "capacity": 131072},
        # 4K frames with the 12-scale bank
        {"name": "queue_uhd", "kind": "queue", "w": 3840, "h": 2160, "lambdas": bank(12), "capacity": 524288},
        # a camera loop that waits for each frame's records
        {"name": "host_hd", "kind": "host", "w": 1920, "h": 1080, "lambdas": bank(8), "capacity": 131072},
        # a video with four frames in flight
        {"name": "stream_hd", "kind": "stream", "w": 1920, "h": 1080, "lambdas": bank(8), "capacity": 65536,
         "depth": 4, "frames": 8},
        # a photo collection of mixed sizes, W in [320, 1920], H in [240, 1080]
        {"name": "batch_mixed", "kind": "batch", "n": 16, "sizes_seed": 1002, "lambdas": bank(8), "capacity": 65536},
        # the dense maps of an image for display or further processing, the Context's own 9-scale bank
        {"name": "responses_vga", "kind": "responses", "w": 640, "h": 480, "lambdas": bank(9), "capacity": 65536},
        # gradient of two small images whose sides are no power of two
        {"name": "adjoint_2x96x80", "kind": "adjoint", "n": 2, "w": 96, "h": 80, "lambdas": bank(4)},
        # the training workload: 16 images of 512 x 512, 6 scales
        {"name": "adjoint_16x512x512", "kind": "adjoint", "n": 16, "w": 512, "h": 512, "lambdas": bank(6)},
        # one ragged photo with many scales
        {"name": "adjoint_1x1333x1001", "kind": "adjoint", "n": 1, "w": 1333, "h": 1001, "lambdas": bank(10)},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["detect", "queue", "host", "stream", "batch", "responses", "adjoint", "adjoint"])
    if kind == "batch":
        return {"kind": kind, "n": _log_int(rng, 2, 16), "sizes_seed": rng.randrange(1 << 20),
                "lambdas": bank(rng.randint(4, 8)), "capacity": 65536}
    if kind == "adjoint":
        w, h = _log_int(rng, 64, 1400), _log_int(rng, 64, 1100)
        n = max(1, min(16, _log_int(rng, 1, 16), 4_000_000 // (w * h)))
        scales = rng.randint(2, 6 if min(w, h) < 256 else 10)
        return {"kind": kind, "n": n, "w": w, "h": h, "lambdas": bank(scales)}
    if kind in ("detect", "queue"):
        w, h = _log_int(rng, 120, 3840), _log_int(rng, 96, 2160)
        scales = rng.randint(2, 6 if min(w, h) < 256 else 12)
    else:
        w, h = _log_int(rng, 320, 1920), _log_int(rng, 240, 1080)
        scales = rng.randint(3, 9)
    lam = rng.choice([bank(scales), bank(scales), VGA, "4,6,11"])
    case = {"kind": kind, "w": w, "h": h, "lambdas": lam, "capacity": 65536 if w * h < 1 << 21 else 524288}
    if kind == "stream":
        case.update(depth=rng.randint(2, 4), frames=rng.randint(4, 8))
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _image(w, h, seed, polygons=None):
    """uint8 CUDA image: 1/f^2 noise (mean 128, std 30) and filled polygons of random intensity."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    fy = torch.fft.fftfreq(h, device="cuda", dtype=torch.float64)[:, None]
    fx = torch.fft.rfftfreq(w, device="cuda", dtype=torch.float64)[None, :]
    f = torch.sqrt(fx * fx + fy * fy)
    f[0, 0] = math.inf
    white = torch.randn((h, w), generator=gen, device="cuda", dtype=torch.float64)
    field = torch.fft.irfft2(torch.fft.rfft2(white) / f, s=(h, w))
    img = 128.0 + 30.0 * (field - field.mean()) / field.std()
    rng = np.random.default_rng(int(seed))
    for _ in range(max(2, min(150, w * h // 15000)) if polygons is None else polygons):
        nv = int(rng.integers(3, 7))
        cx, cy, rad = rng.uniform(0, w), rng.uniform(0, h), rng.uniform(0.02, 0.15) * min(w, h)
        ang, rr = np.sort(rng.uniform(0, 2 * np.pi, nv)), rad * rng.uniform(0.5, 1.0, nv)
        xs, ys, value = cx + rr * np.cos(ang), cy + rr * np.sin(ang), float(rng.uniform(0, 255))
        x0, x1 = max(int(xs.min()), 0), min(int(xs.max()) + 2, w)
        y0, y1 = max(int(ys.min()), 0), min(int(ys.max()) + 2, h)
        if x1 <= x0 or y1 <= y0:
            continue
        px = torch.arange(x0, x1, device="cuda", dtype=torch.float64)[None, :, None]
        py = torch.arange(y0, y1, device="cuda", dtype=torch.float64)[:, None, None]
        v = torch.tensor(np.stack([xs, ys, np.roll(xs, -1), np.roll(ys, -1)]), device="cuda")
        crosses = ((v[1] > py) != (v[3] > py)) & (px < v[0] + (v[2] - v[0]) * (py - v[1]) / (v[3] - v[1]))
        inside = crosses.sum(-1) % 2 == 1
        img[y0:y1, x0:x1].masked_fill_(inside, value)
    return img.round_().clamp_(0, 255).to(torch.uint8)


def _sizes(case):
    rng = np.random.default_rng(int(case["sizes_seed"]))
    return [(int(rng.integers(20, 121)) * 16, int(rng.integers(15, 68)) * 16) for _ in range(case["n"])]


def _inputs(case, seed):
    """The seeded images of a case (and, for the adjoint, the loss weights of one image after the other)."""
    if case["kind"] == "batch":
        return [_image(w, h, 1000 * seed + i) for i, (w, h) in enumerate(_sizes(case))]
    if case["kind"] == "stream":
        base = _image(case["w"], case["h"], seed)
        return [torch.roll(base, (37 * k, 101 * k), (0, 1)) for k in range(case["frames"])]
    if case["kind"] == "adjoint":
        # uint8 content with its quantisation noise restored, on the [0, 1] scale
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int(seed) + 1)
        img = torch.stack([_image(case["w"], case["h"], 1000 * seed + i) for i in range(case["n"])])
        img = (img.float() + torch.rand(img.shape, generator=gen, device="cuda") - 0.5) / 255.0
        cells = sum(s["dataW"] * s["dataH"] for s in _scales(case["w"], case["h"], lambdas_of(case)))
        return img, torch.randn(case["n"] * cells, generator=gen, device="cuda")
    return _image(case["w"], case["h"], seed)


def prepare(case, seed):
    from bimp_b200 import api

    kind, lam, x, cap = case["kind"], lambdas_of(case), _inputs(case, seed), case.get("capacity")
    state = {"kind": kind, "capacity": cap}

    def store(n=1):   # the program's own keypoint matrices (columns after the last keypoint stay 0)
        return [torch.zeros((7, cap), device="cuda") for _ in range(n)]

    if kind == "detect":
        state.update(cs=api.CudaStuff(case["w"], case["h"], lam), image=x, keep=store())
    elif kind == "queue":
        state.update(cs=api.CudaStuff(case["w"], case["h"], lam), image=x, keep=store(),
                     count=torch.zeros(1, dtype=torch.int32, device="cuda"))
    elif kind == "host":
        state.update(cs=api.CudaStuff(case["w"], case["h"], lam), image=x.cpu().numpy(),
                     keep=[np.zeros((cap, 7), np.float32)])
    elif kind == "stream":
        pinned = [f.cpu().pin_memory() for f in x]
        state.update(pipe=api.Pipeline(case["w"], case["h"], lam, depth=case["depth"], capacity=cap),
                     frames=[p.numpy() for p in pinned], pinned=pinned, depth=case["depth"],
                     keep=[np.zeros((cap, 7), np.float32) for _ in pinned])
    elif kind == "batch":
        state.update(batch=api.Batch(_sizes(case), lam, kp_capacity=cap), images=x, keep=store(case["n"]))
    elif kind == "responses":
        ctx = api.Context(x.cpu().numpy(), lambdas=lam)
        ctx.capacity = cap
        # the context takes images of its upload size (an image below 350 pixels is upscaled there)
        state.update(ctx=ctx, image=ctx.current_image.clone())
    else:
        images, masks = x
        adj = api.Adjoint(case["w"], case["h"], case["n"], lam)
        state.update(adj=adj, images=images, masks=masks, grad=torch.empty_like(images))
    return state


def run(state):
    from bimp_b200 import _lib, api

    kind, keep = state["kind"], state.get("keep")
    if kind == "detect":
        kp = api.getKeypoints(state["image"], state["cs"], capacity=state["capacity"])
        keep[0][:, : kp.shape[1]] = kp
        return [keep[0], kp.shape[1]]
    if kind == "queue":
        img, cs, kp, count = state["image"], state["cs"], keep[0], state["count"]
        _lib.check(_lib.lib().bimp_detect_device_async(
            cs.handle, img.data_ptr(), img.stride(0), cs.width, cs.height, kp.data_ptr(), kp.stride(0),
            state["capacity"], count.data_ptr(), torch.cuda.current_stream().cuda_stream), "detect")
        return [kp, count]
    if kind == "host":
        rec, total, _ = api.detect_host(state["cs"], state["image"], capacity=state["capacity"])
        return _kept(keep[0], rec) + [total]
    if kind == "stream":
        pipe, out = state["pipe"], []
        for f in state["frames"]:
            if pipe.in_flight() == state["depth"]:
                out.append(_kept(keep[len(out)], pipe.pop()[0]))
            pipe.push(f)
        while pipe.in_flight():
            out.append(_kept(keep[len(out)], pipe.pop()[0]))
        return out
    if kind == "batch":
        b = state["batch"]
        b.load(state["images"])
        b.run()
        for i, k in enumerate(keep):
            kp = b.keypoints(i)
            k[:, : kp.shape[1]] = kp
        return keep
    if kind == "responses":
        ctx = state["ctx"]
        ctx.loadImage(state["image"])
        return [m for r in ctx.getResponses() for m in (r["D"], r["S"])]
    adj = state["adj"]
    loss = adj.forward(state["images"], state["masks"])
    grad, gparams = adj.backward(state["grad"])
    return {"loss": loss, "grad": grad, "gparams": gparams}


def _kept(store, rec):
    """Host records in the program's own array: the float fields (x, y, size, angle, response) and the whole ones."""
    store[: len(rec)] = rec.view(np.float32).reshape(-1, 7)
    return [store[:, :5], store.view(np.int32)[:, 5:], len(rec)]


# ---------------------------------------------------------------------------
# work that the path cannot do without
# ---------------------------------------------------------------------------
def _snap(n):
    n = (n + 15) // 16 * 16
    up = 1 << (n - 1).bit_length()
    return up if up <= 1024 or up == n else (n + 511) // 512 * 512


def _scales(w, h, lambdas):
    """Geometry of every scale: pyramid level, data and torus sizes, kernel size, stencil offsets."""
    out = []
    for l2 in sorted(np.float32(x) for x in lambdas):
        pyr, level = np.float32(1), 0
        while float(l2 / pyr) >= 7.5:
            pyr, level = np.float32(pyr * 2), level + 1
        lam = np.float32(l2 / pyr)
        fs = np.float32(7.0 * float(lam))
        if int(fs) % 2 == 0:
            fs = np.float32(fs + np.float32(1))
        s = {"lam": lam, "pyr": pyr, "level": level, "fs": fs, "kX": int(float(fs) / 2), "kW": int(fs),
             "dataW": int(np.float32(w) / pyr), "dataH": int(np.float32(h) / pyr), "off": int(lam)}
        s["fftW"], s["fftH"] = _snap(s["dataW"]), _snap(s["dataH"])
        th = [float(np.float32(o * math.pi / NUM_ORI)) for o in range(NUM_ORI)]
        rha = lambda v: int(math.copysign(math.floor(abs(v) + 0.5), v))  # noqa: E731
        s["es"] = [(rha(0.6 * float(lam) * math.cos(t)), rha(0.6 * float(lam) * math.sin(t))) for t in th]
        s["in"] = [(b, a) for a, b in s["es"]]
        s["ih"] = [(rha(0.5 * a), rha(0.5 * b)) for a, b in s["in"]]
        out.append(s)
    return out


def _pixels(case):
    if case["kind"] == "batch":
        return [(w, h) for w, h in _sizes(case)]
    return [(case["w"], case["h"])] * int(case.get("n", case.get("frames", 1)))


def work(case):
    """Images in, records (about one keypoint per 180 scale pixels) or maps out; one real forward and eight complex
    inverse transforms of each scale's torus (5 N log2 N each) and about 110 operations a pixel for the stencils;
    the adjoint's backward adds eight forward and one inverse transform and the same stencils again."""
    bytes_, flops = 0.0, 0.0
    for w, h in _pixels(case):
        for s in _scales(w, h, lambdas_of(case)):
            n, torus = s["dataW"] * s["dataH"], s["fftW"] * s["fftH"]
            fft = 5.0 * torus * math.log2(torus)
            flops += 8.5 * fft + 110.0 * n
            if case["kind"] == "adjoint":
                flops += 8.5 * fft + 110.0 * n
                bytes_ += 4 * n                      # the loss weights
            elif case["kind"] == "responses":
                bytes_ += 8 * n                      # D and S
            else:
                bytes_ += 28 * n / 180.0             # the records
        bytes_ += w * h * (8 if case["kind"] == "adjoint" else 1)
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _taps32(s, o):
    """Even and odd taps as the bank holds them: float32 arithmetic, the sum of the even taps removed."""
    f = np.float32
    lam, th = s["lam"], f(o * math.pi / NUM_ORI)
    sig = f(float(lam) * 0.56)
    d = np.arange(s["kW"]) - s["kX"]
    x, y = d[None, :].astype(f), d[:, None].astype(f)
    c, sn = np.cos(th, dtype=f), np.sin(th, dtype=f)
    a, b = x * c + y * sn, y * c - x * sn
    env = np.exp(f(-1) / (f(2) * f(sig * sig)) * (a * a + f(0.5) * b * b))
    freq = (2 * math.pi * a.astype(np.float64) / float(lam)).astype(f)
    even, odd = env * np.cos(freq), env * np.cos(freq + f(-math.pi / 2))
    total = np.add.accumulate(even.ravel(), dtype=f)[-1]
    even = even - total / (s["fs"] * s["fs"])
    return (torch.from_numpy(v.astype(np.float64)).cuda() for v in (even, odd))


def _taps64(s, o, alpha, rho):
    """The taps as differentiable functions of the wavelength scale and the sigma ratio (kernel size fixed)."""
    lam0 = float(s["lam"])
    lam = alpha * lam0
    sig, fs = rho * lam, 7.0 * lam + (float(s["fs"]) - 7.0 * lam0)
    t = float(np.float32(o * math.pi / NUM_ORI))
    d = torch.arange(s["kW"], device="cuda", dtype=torch.float64) - s["kX"]
    a = d[None, :] * math.cos(t) + d[:, None] * math.sin(t)
    b = d[:, None] * math.cos(t) - d[None, :] * math.sin(t)
    env = torch.exp(-(a * a + 0.5 * b * b) / (2 * sig * sig))
    even, odd = env * torch.cos(2 * math.pi * a / lam), env * torch.sin(2 * math.pi * a / lam)
    return even - even.sum() / fs ** 2, odd


def _pad(n_fft, n, half):
    t = torch.arange(n_fft, device="cuda")
    return torch.where(t < n, t, torch.where(t < n + half, n - 1, 0))


def _cells(data, s, taps):
    """Complex cells |even + i odd| over the stencil window (dataH + 1) x (dataW + 1) of the padded torus."""
    H, W = s["fftH"], s["fftW"]
    X = torch.fft.fft2(data[_pad(H, s["dataH"], s["kX"])[:, None], _pad(W, s["dataW"], s["kX"])[None, :]])
    k = torch.arange(s["kW"], device="cuda") - s["kX"]
    at = ((k % H)[:, None] * W + (k % W)[None, :]).reshape(-1)
    r = torch.arange(s["dataH"] + 1, device="cuda")[:, None]
    flat = (r * W + torch.arange(s["dataW"] + 1, device="cuda")[None, :]) % (H * W)
    out = []
    for o in range(NUM_ORI):
        even, odd = taps(s, o)
        q = torch.zeros(H * W, device="cuda", dtype=torch.complex128)
        q = q.index_add(0, at, torch.complex(even, odd).reshape(-1)).view(H, W)
        z = torch.fft.ifft2(X * torch.fft.fft2(q))
        m2 = z.real ** 2 + z.imag ** 2
        # responses up to 3e-5 pass no gradient
        m = torch.where(m2 > 9e-10, torch.sqrt(torch.clamp(m2, min=9e-10)), torch.sqrt(m2.detach()))
        out.append(m.reshape(-1)[flat])
    return out


def _maps(C, s, wt=1.0, wr=1.0):
    """Summed keypoint map D and single-stopped map S of one scale."""
    H, W = s["dataH"], s["dataW"]
    y, x = torch.arange(H, device="cuda")[:, None], torch.arange(W, device="cuda")[None, :]

    def at(c, dy, dx):
        return c[(y + dy).clamp(0, H), (x + dx).clamp(0, W)]

    def ok(o1, o2):
        a, b = 2 * abs(o1), 2 * abs(o2)
        return ((y >= a) & (y <= H - a) & (x >= b) & (x <= W - b)).double()

    relu = torch.relu
    S = D = T = R = 0.0
    for o in range(NUM_ORI):
        c, cp = C[o], C[(o + 4) % NUM_ORI]
        (e1, e2), (i1, i2), (h1, h2) = s["es"][o], s["in"][o], s["ih"][o]
        me, mi, cen = ok(e1, e2), ok(i1, i2), at(c, 0, 0)
        S = S + me * relu(at(c, -e1, e2) - at(c, e1, -e2))
        D = D + me * relu(cen - 0.5 * at(c, -2 * e1, 2 * e2) - 0.5 * at(c, 2 * e1, -2 * e2))
        T = T + mi * relu(at(c, -i1, -i2) - cen)
        R = R + mi * relu(relu(cen - 16.0 * at(cp, h1, h2)) + cen - 16.0 * at(cp, -h1, -h2))
    return D - (wt * T + wr * R), S - (wt * T + wr * R)


def _reflect(i, n):
    i = i.abs() % max(2 * n - 2, 1)
    return torch.where(i >= n, 2 * n - 2 - i, i)


def _pyr_sums(img):
    """Sums of the 5 x 5 binomial window (weights of sum 256) at every second pixel, reflected at the border."""
    h, w = img.shape
    k = torch.arange(-2, 3, device="cuda")
    rows = _reflect(2 * torch.arange((h + 1) // 2, device="cuda")[:, None] + k, h)
    cols = _reflect(2 * torch.arange((w + 1) // 2, device="cuda")[:, None] + k, w)
    wts = (1.0, 4.0, 6.0, 4.0, 1.0)
    tmp = sum(wts[j] * img[rows[:, j], :] for j in range(5))
    return sum(wts[j] * tmp[:, cols[:, j]] for j in range(5))


def _levels(img, n, whole):
    """Pyramid of an image in float64: rounded to whole values (ties to even) for bytes."""
    out = [img.double()]
    for _ in range(n):
        v = _pyr_sums(out[-1]) / 256.0
        out.append(v.round().clamp(0, 255) if whole else v)
    return out


def _responses(image, lambdas):
    """D and S of every scale of a byte image."""
    h, w = image.shape
    scales = _scales(w, h, lambdas)
    levels = _levels(image, max(s["level"] for s in scales), True)
    out = []
    for s in scales:
        data = levels[s["level"]][: s["dataH"], : s["dataW"]] * (255.0 / 65536.0)
        out += _maps(_cells(data, s, _taps32), s)
    return out


def _adjoint(case, images, masks):
    n, (w, h) = case["n"], (case["w"], case["h"])
    scales = _scales(w, h, lambdas_of(case))
    X = images.double().requires_grad_()
    theta = torch.tensor([1.0, 0.56, 1.0, 1.0], device="cuda", dtype=torch.float64, requires_grad=True)
    total, at = 0.0, 0
    for i in range(n):
        for s in scales:   # one scale of one image at a time bounds the memory of the graph
            level = _levels(X[i], s["level"], False)[-1]
            data = level[: s["dataH"], : s["dataW"]] * (65025.0 / 65536.0)
            C = _cells(data, s, lambda s_, o: _taps64(s_, o, theta[0], theta[1]))
            M = masks[at:at + s["dataW"] * s["dataH"]].double().view(s["dataH"], s["dataW"])
            at += M.numel()
            loss = (M * _maps(C, s, theta[2], theta[3])[0]).sum()
            loss.backward()
            total += loss.detach()
    return {"loss": total.reshape(1), "grad": X.grad, "gparams": theta.grad}


def exact(case, seed):
    """None for keypoint lists: which pixels are listed is a decision on the maps of ``responses``."""
    kind = case["kind"]
    if kind == "adjoint":
        return _adjoint(case, *_inputs(case, seed))
    if kind == "responses" and min(case["w"], case["h"]) >= 350:   # a smaller one is upscaled in whole arithmetic
        with torch.no_grad():
            return _responses(_inputs(case, seed), lambdas_of(case))
    return None
