"""The work a program has this package do, as cases that can be timed: background subtraction of a camera's
frames (SuBSENSE, PAWCS, LOBSTER, ViBe, PBAS; one stream or many in a batch), dense LBSP descriptors, and the
scoring of masks against ground truth, each through the package's public entry points.

A case is a dict of plain values:

* ``kind``: ``stream`` (one subtractor's ``apply``, one frame a pass), ``clip`` (``apply`` over every frame of a
  short clip, then ``getBackgroundImage``), ``mix`` (one ``batch_apply`` over a mix of streams a pass), ``lbsp``
  (``lbsp_compute2`` of a frame) or ``score`` (``BinClassif`` over one mask);
* ``algo``, ``w``, ``h``, ``c``: the algorithm and the frame;
* ``io``: where frames and masks live: ``device`` (CUDA tensors), ``pinned`` (page-locked host tensors) or
  ``host`` (numpy arrays);
* ``mix``: the streams of a mix, as ``count x width x height x channels`` terms.

The scenes are a Gaussian-smoothed (sigma 4) random texture with contrast, sensor noise and moving shapes, or a
thermal-like gradient with warm blobs, as in the package's own synthetic streams. Streams are in progress when a
pass begins: the model is initialized and has seen a few frames.
"""
import math
import random

import numpy as np
import torch
import torch.nn.functional as F

import litiv_gb300 as lv
from litiv_gb300.metrics import BinClassif, COUNTERS, METRICS

RING = 8  # frames kept of a scene, played forth and back
WARM = 8  # frames a stream has seen before the first pass

SUBTRACTORS = {
    "subsense": lv.BackgroundSubtractorSuBSENSE,
    "pawcs": lv.BackgroundSubtractorPAWCS,
    "lobster": lv.BackgroundSubtractorLOBSTER,
    "vibe": lv.BackgroundSubtractorViBe,
    "pbas": lv.BackgroundSubtractorPBAS,
}

# bytes of one pixel's model that a frame step reads and writes, without samples: ten float maps read and
# written, last colour and descriptor read and written (per channel), byte maps (SuBSENSE's feedback; PAWCS
# keeps the same maps); PBAS keeps R, T and D
MAP_BYTES = {"subsense": (92, 6), "pawcs": (92, 6), "lobster": (0, 3), "vibe": (0, 0), "pbas": (24, 0)}
SAMPLE_BYTES = {"subsense": 3, "pawcs": 15, "lobster": 3, "vibe": 1, "pbas": 2}  # per channel and sample


def listed():
    return [
        # One low-resolution camera, frames already on the GPU: the smallest frame step, where launches count.
        {"name": "subsense-qvga", "kind": "stream", "algo": "subsense", "w": 320, "h": 240, "c": 3, "io": "device"},
        # One full-HD camera, the ordinary single-stream use of the default algorithm.
        {"name": "subsense-1080p", "kind": "stream", "algo": "subsense", "w": 1920, "h": 1080, "c": 3, "io": "device"},
        # A dataset sequence of ragged size read into host memory, gray: a clip's masks and its background.
        {"name": "subsense-clip-gray", "kind": "clip", "algo": "subsense", "w": 595, "h": 245, "c": 1, "io": "host"},
        # A server's tick: 64 cameras of four resolutions, three quarters in colour, frames on the GPU.
        {"name": "subsense-mix64", "kind": "mix", "algo": "subsense", "io": "device",
         "mix": "12x320x240x3+4x320x240x1+18x640x480x3+6x640x480x1+12x1280x720x3+4x1280x720x1+6x1920x1080x3+2x1920x1080x1"},
        # A small site's tick: 12 cameras, frames and masks in page-locked host memory.
        {"name": "subsense-mix12-pinned", "kind": "mix", "algo": "subsense", "io": "pinned",
         "mix": "5x320x240x3+1x357x288x1+4x640x480x3+2x1279x719x3"},
        # A thermal camera with the word-dictionary model.
        {"name": "pawcs-vga-gray", "kind": "stream", "algo": "pawcs", "w": 640, "h": 480, "c": 1, "io": "device"},
        # The word-dictionary model on a colour camera.
        {"name": "pawcs-vga", "kind": "stream", "algo": "pawcs", "w": 640, "h": 480, "c": 3, "io": "device"},
        # The lighter algorithms, for sites that cannot afford the above: full HD, ragged, and small.
        {"name": "lobster-odd-720", "kind": "stream", "algo": "lobster", "w": 1277, "h": 719, "c": 3, "io": "device"},
        {"name": "vibe-qvga", "kind": "stream", "algo": "vibe", "w": 320, "h": 240, "c": 3, "io": "device"},
        {"name": "pbas-1080p", "kind": "stream", "algo": "pbas", "w": 1920, "h": 1080, "c": 3, "io": "device"},
        # Dense descriptors of a frame in host memory, as a feature extractor's user calls it.
        {"name": "lbsp-720p", "kind": "lbsp", "w": 1280, "h": 720, "c": 3, "io": "host"},
        # A mask the subtractor left on the GPU, scored against ground truth inside a region of interest.
        {"name": "score-1080p", "kind": "score", "w": 1920, "h": 1080, "io": "device"},
    ]


def draw(rng):
    kind = rng.choice(["stream"] * 8 + ["clip", "mix", "mix", "lbsp", "score"])
    c = rng.choice([1, 3, 3])
    io = rng.choice(["device", "device", "pinned", "host"])

    def size(lo, hi):
        # width over its logarithm, ragged or rounded to what cameras give, at a camera's aspect
        w = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if rng.random() < 0.5:
            w = max(16, w // 16 * 16)
        h = max(64, int(w * rng.choice([9 / 16, 3 / 4, 0.5621, 0.41])))
        return w, h

    if kind == "mix":
        terms = []
        for _ in range(rng.randint(2, 6)):
            w, h = size(160, 1920)
            terms.append("%dx%dx%dx%d" % (rng.randint(1, 6), w, h, rng.choice([1, 3, 3])))
        return {"kind": "mix", "algo": "subsense", "io": io, "mix": "+".join(terms)}
    if kind == "lbsp":
        w, h = size(160, 1920)
        return {"kind": "lbsp", "w": w, "h": h, "c": c, "io": "host"}
    if kind == "score":
        w, h = size(160, 1920)
        return {"kind": "score", "w": w, "h": h, "io": "device"}
    algo = rng.choice(["subsense"] * 4 + ["pawcs"] * 2 + ["lobster", "vibe", "pbas"])
    w, h = size(160, 640 if algo == "pawcs" or kind == "clip" else 1920)
    if kind == "clip" and algo == "pawcs":
        algo = "subsense"
    return {"kind": kind, "algo": algo, "w": w, "h": h, "c": c, "io": io}


def _streams(case):
    """(width, height, channels) of every stream of a case"""
    if case["kind"] != "mix":
        return [(case["w"], case["h"], case.get("c", 1))]
    out = []
    for term in case["mix"].split("+"):
        n, w, h, c = (int(v) for v in term.split("x"))
        out += [(w, h, c)] * n
    return out


def _scene(w, h, c, seed, frames, thermal=False):
    """`frames` frames [T, h, w(, c)] uint8 of a seeded scene on the GPU, and the shapes' mask of the last"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rng = random.Random(seed)
    if thermal:
        gx = torch.linspace(0, 1, w, device="cuda")[None, :, None]
        gy = torch.linspace(0, 1, h, device="cuda")[:, None, None]
        coarse = torch.rand((1, 1, h // 64 + 2, w // 64 + 2), generator=g, device="cuda")
        wave = F.interpolate(coarse, size=(h, w), mode="bilinear", align_corners=False)[0].permute(1, 2, 0)
        base = 80 + 30 * (gx + gy) + 20 * (wave - 0.5)
        sigma, n_shapes = 2.0, 6
    else:
        t = torch.rand((1, c, h + 24, w + 24), generator=g, device="cuda") * 255
        for _ in range(4):  # four 7-wide boxes: sigma 4
            t = F.avg_pool2d(t, 7, stride=1)
        base = (128 + 6 * (t[0] - 127.5)).permute(1, 2, 0).contiguous()
        sigma, n_shapes = rng.uniform(2, 6), rng.randint(2, 10)
    big = max(16, min(w, h) // 5)
    shapes = []
    for _ in range(n_shapes):
        shapes.append({"x": rng.uniform(0, w), "y": rng.uniform(0, h), "vx": rng.uniform(-3, 3),
                       "vy": rng.uniform(-3, 3), "sx": rng.randint(8, big), "sy": rng.randint(8, big),
                       "round": thermal or rng.random() < 0.5,
                       "col": [rng.uniform(180, 240) if thermal else rng.uniform(0, 255) for _ in range(c)]})
    out = torch.empty((frames, h, w, c), dtype=torch.uint8, device="cuda")
    gt = torch.zeros((h, w), dtype=torch.uint8, device="cuda")
    for k in range(frames):
        img = base.clone()
        for s in shapes:
            x0, y0 = int(s["x"] + k * s["vx"]) % w, int(s["y"] + k * s["vy"]) % h
            x1, y1 = min(w, x0 + s["sx"]), min(h, y0 + s["sy"])
            col = torch.tensor(s["col"], device="cuda")
            box = img[y0:y1, x0:x1]
            if s["round"]:
                u = (torch.arange(x1 - x0, device="cuda") * 2 - s["sx"])[None, :] / s["sx"]
                v = (torch.arange(y1 - y0, device="cuda") * 2 - s["sy"])[:, None] / s["sy"]
                inside = (u * u + v * v) <= 1
                box.copy_(torch.where(inside[:, :, None], col, box))
            else:
                inside = torch.ones((y1 - y0, x1 - x0), dtype=torch.bool, device="cuda")
                box.copy_(col.expand_as(box))
            if k == frames - 1:
                gt[y0:y1, x0:x1][inside] = 255
        noise = torch.randn((h, w, c), generator=g, device="cuda")
        out[k] = (img + sigma * noise).round().clamp(0, 255).to(torch.uint8)
    return (out[:, :, :, 0].contiguous() if c == 1 else out), gt


def _placed(t, io):
    if io == "device":
        return t
    if io == "pinned":
        return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)
    return t.cpu().numpy()


def prepare(case, seed):
    kind, io = case["kind"], case["io"]
    sizes = _streams(case)
    if kind == "score":
        (w, h, _), = sizes
        frames, gt = _scene(w, h, 1, seed, 1)
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        flip = torch.rand((h, w), generator=g, device="cuda") < 0.02
        mask = torch.where(flip, 255 - gt, gt)
        code = torch.rand((h, w), generator=g, device="cuda")
        gt[code < 0.01] = 170  # unknown
        gt[(code > 0.99) & (gt == 0)] = 50  # shadow
        roi = torch.full((h, w), 255, dtype=torch.uint8, device="cuda")
        roi[: h // 16] = 0
        return {"case": case, "mask": mask, "gt": gt, "roi": roi}
    if kind == "lbsp":
        (w, h, c), = sizes
        return {"case": case, "frame": _scene(w, h, c, seed, 1)[0][0].cpu().numpy()}
    state = {"case": case, "frames": [], "masks": [], "subs": [], "t": 0}
    thermal = case["algo"] == "pawcs" and sizes[0][2] == 1
    for i, (w, h, c) in enumerate(sizes):
        frames, _ = _scene(w, h, c, seed * 1009 + i, RING, thermal)
        sub = SUBTRACTORS[case["algo"]](seed=seed * 131 + i)
        torch.cuda.synchronize()
        sub.initialize(frames[0])
        state["frames"].append(_placed(frames, io))
        masks = torch.zeros((RING if kind == "clip" else 1, h, w), dtype=torch.uint8, device="cuda")
        state["masks"].append(_placed(masks, io))
        state["subs"].append(sub)
    torch.cuda.synchronize()
    for _ in range(WARM if kind != "clip" else 1):
        run(state)
    return state


def _tick(state):
    """index of the next frame: the ring forth and back, as a camera's continuing stream"""
    k = state["t"] % (2 * RING - 2)
    state["t"] += 1
    return k if k < RING else 2 * RING - 2 - k


def run(state):
    kind = state["case"]["kind"]
    if kind == "score":
        scored = BinClassif().accumulate(state["mask"], state["gt"], state["roi"])
        return {"counts": scored.as_dict(), "metrics": scored.metrics()}
    if kind == "lbsp":
        return lv.lbsp_compute2(state["frame"])
    if kind == "mix":
        k = _tick(state)
        masks = [m[0] for m in state["masks"]]
        lv.batch_apply(state["subs"], [f[k] for f in state["frames"]], masks)
        return masks
    sub, frames, masks = state["subs"][0], state["frames"][0], state["masks"][0]
    if kind == "clip":
        for k in range(RING):
            sub.apply(frames[k], masks[k])
        return {"masks": masks, "background": sub.getBackgroundImage()}
    sub.apply(frames[_tick(state)], masks[0])
    return masks[0]


def work(case):
    kind = case["kind"]
    if kind == "score":
        px = case["w"] * case["h"]
        return {"bytes": 3 * px, "flops": 0}
    if kind == "lbsp":
        v = case["w"] * case["h"] * case["c"]
        return {"bytes": 3 * v, "flops": 16 * v}
    algo = case["algo"]
    total = ops = 0
    for w, h, c in _streams(case):
        px = w * h
        fixed, per_channel = MAP_BYTES[algo]
        # frame in, mask out, maps, two samples that have to match, one sample written now and then
        step = px * (c + 1 + fixed + per_channel * 2 * c + SAMPLE_BYTES[algo] * c * 2.25)
        steps = RING if kind == "clip" else 1
        total += step * steps
        if kind == "clip":  # the background image: the mean of every sample's colour
            total += px * c * (1 + 50)
        ops += px * c * 16 * 3 * steps  # 16 taps against the pixel and two samples
    return {"bytes": total, "flops": ops}


LBSP_TAPS = [(-2, 0), (2, 0), (0, -2), (0, 2), (-2, 2), (2, -2), (2, 2), (-2, -2),
             (0, 1), (-1, 0), (0, -1), (1, 0), (-1, -1), (1, 1), (1, -1), (-1, 1)]


def exact(case, seed):
    """LBSP descriptors and scores in 64 bits; masks are decisions on a random model and have no such value"""
    if case["kind"] == "lbsp":
        img = prepare(case, seed)["frame"].astype(np.int64)
        h, w = img.shape[:2]
        mid = img[2:h - 2, 2:w - 2]
        # the relative threshold is a single-precision number, rounded half to even
        thr = np.clip(np.rint((mid.astype(np.float32) * np.float32(0.333)).astype(np.float64)), 0, 255)
        bits = np.zeros(mid.shape, np.int64)
        for n, (dx, dy) in enumerate(LBSP_TAPS):
            tap = img[2 + dy:h - 2 + dy, 2 + dx:w - 2 + dx]
            bits |= (np.abs(tap - mid) > thr).astype(np.int64) << n
        out = np.zeros(img.shape, np.uint16)
        out[2:h - 2, 2:w - 2] = bits
        return out
    if case["kind"] == "score":
        s = prepare(case, seed)
        mask, gt, roi = (s[k].cpu().numpy() for k in ("mask", "gt", "roi"))
        dc = (gt == 85) | (gt == 170) | (roi == 0)
        pos, want = mask == 255, gt == 255
        tp, tn = int((~dc & pos & want).sum()), int((~dc & ~pos & ~want).sum())
        fp, fn = int((~dc & pos & ~want).sum()), int((~dc & ~pos & want).sum())
        counts = [tp, tn, fp, fn, int((~dc & pos & (gt == 50)).sum()), int(dc.sum())]

        def over(a, b):
            return a / b if b else 0.0

        recall, precision = over(tp, tp + fn), over(tp, tp + fp)
        den = math.sqrt(float(tp + fp) * (tp + fn) * (tn + fp) * (tn + fn))
        values = [recall, over(tn, tn + fp), over(fp, fp + tn), over(fn, tp + fn),
                  100.0 * over(fn + fp, tp + tn + fp + fn), precision,
                  over(2 * recall * precision, recall + precision), over(float(tp * tn - fp * fn), den)]
        return {"counts": dict(zip(COUNTERS, counts)), "metrics": dict(zip(METRICS, values))}
    return None
