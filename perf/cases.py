"""What the disparity path is timed on: its public entry points over the sizes
they are used at.

``listed()`` names the cases, ``draw(rng)`` gives others of the same ranges,
``prepare(case, seed)`` makes what a program holds before the call (images in
device memory, plans, weights), ``run(state)`` is one pass through the entry
point and ``exact(case, seed)`` the same outputs in 64 bits from plain torch.
The images are seeded scenes of slanted textured planes with an exact right
view, as the package's own generator (synth.py) makes them, rendered on the GPU
so that a batch is made quickly.
"""

from __future__ import annotations

import importlib.util
import math
import os
import random
import sys
import zlib

import numpy as np
import torch
import torch.nn.functional as F

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEVICE = "cuda"
# refine_disparity's parameters
REFINE = dict(R=10, P1=12.0, P2=150.0, rx=4, ry=3)
TOL = 2.0
PROBE_WIDTH, MAX_WIDTH, PASSES = 64, 320, 3


def _package():
    """The package; its folder's name is not an identifier, so it is loaded by path."""
    if "sv_b200" not in sys.modules:
        folder = os.path.join(ROOT, "from-scratch-stereo-vision_b200")
        spec = importlib.util.spec_from_file_location(
            "sv_b200", os.path.join(folder, "__init__.py"), submodule_search_locations=[folder])
        sys.modules["sv_b200"] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules["sv_b200"])
    return sys.modules["sv_b200"]


_NET = []


def _net():
    """The shipped checkpoint, read once as a program does."""
    if not _NET:
        _NET.append(_package().weights.load_model())
    return _NET[0]


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the drop-in a script calls on float grays: the small 160x120 scene
        dict(name="lr_refine_160x120_f64", kind="lr_refine", W=160, H=120, dmax=30, image="f64"),
        # the device-resident refinement of the usual 450x375 pair
        dict(name="refiner_450x375", kind="refiner", W=450, H=375, dmax=80, image="u8"),
        # the same call on the largest pair of a test split, odd in both sizes
        dict(name="refiner_1397x1101", kind="refiner", W=1397, H=1101, dmax=200, image="u8"),
        # census + SGM over the whole range (labels and controls): disp0 = R
        dict(name="full_range_640x480", kind="full_range", W=640, H=480, dmax=150, image="u8"),
        # one network forward at the largest work width
        dict(name="forward_320x266", kind="forward", W=320, H=266, dmax=40, image="f32"),
        # the network at native resolution in BF16
        dict(name="predict_bf16_640x480", kind="predict_bf16", W=640, H=480, dmax=44,
             image="u8"),
        # the whole path for one pair: predict_auto + lr_refine
        dict(name="pair_450x375", kind="pair", W=450, H=375, dmax=80, image="u8"),
        # the whole path for a test split of uneven sizes
        dict(name="batch_20_uneven", kind="batch", pairs=20, W=1400, H=1100, dmax=200,
             image="u8"),
        # refinement, superpixel planes and median of a colour pair
        dict(name="refine_disparity_450x375", kind="refine_disparity", W=450, H=375, dmax=80,
             image="u8"),
        # a training step's gradients: 64 crops of the harness's size
        dict(name="train_64x96x64", kind="train", pairs=64, W=96, H=64, dmax=36, image="f32"),
        # the learned band around lr_refine: thin bars, disparities up to 150 px
        dict(name="learned_band_640x480", kind="band", W=640, H=480, dmax=150, image="u8"),
        # both views of a colour pair from PNG bytes to FP64 on the device
        dict(name="read_png_450x375", kind="png", W=450, H=375, dmax=80, image="u8"),
    ]


def draw(rng: random.Random):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))

    kind = rng.choice(["lr_refine", "refiner", "refiner", "full_range", "forward",
                       "predict_bf16", "pair", "pair", "batch", "refine_disparity", "train",
                       "band", "png"])
    image = "u8"
    if kind in ("refiner", "pair"):
        W, H = size(160, 1400), size(120, 1100)
        image = rng.choice(["u8", "u8", "f32", "f64"])
    elif kind == "lr_refine":
        W, H = size(48, 640), size(32, 480)
        image = rng.choice(["u8", "f64"])
    elif kind == "full_range":
        W, H = size(200, 640), size(150, 480)
    elif kind == "forward":
        W, H = size(64, 320), size(48, 266)
        image = "f32"
    elif kind == "train":
        W, H = 4 * rng.randint(16, 32), 4 * rng.randint(12, 24)
        image = "f32"
    else:
        W, H = size(200, 640), size(150, 480)
    dmax = {"forward": 40, "predict_bf16": 44, "train": 36}.get(kind) or \
        rng.randint(20, int(min(200, max(24, 0.3 * W))))
    case = dict(kind=kind, W=W, H=H, dmax=int(dmax), image=image)
    if kind == "batch":
        case.update(pairs=rng.randint(2, 20), W=1400, H=1100, dmax=200)
    if kind == "train":
        case.update(pairs=size(4, 40))
    return case


def _batch_sizes(case):
    """The batch's (W, H, dmax): part of the plan, the same for every seed."""
    rnd = random.Random(7 * case["pairs"])
    out = []
    for _ in range(case["pairs"]):
        W, H = rnd.randint(200, case["W"]), rnd.randint(150, case["H"])
        out.append((W, H, min(rnd.uniform(10.0, case["dmax"]), 0.6 * W)))
    return out


# ------------------------------------------------------------------ scenes
def _blur(t):
    """Separable Gaussian, sigma 1, reflected borders."""
    k = [math.exp(-0.5 * i * i) for i in range(-3, 4)]
    s = sum(k)
    for dim in (0, 1):
        p = F.pad(t[None, None], (0, 0, 3, 3) if dim == 0 else (3, 3, 0, 0), mode="reflect")[0, 0]
        t = sum(p.narrow(dim, i, t.shape[dim]) * (k[i] / s) for i in range(7))
    return t


def _scene(seed, W, H, dmin, dmax, planes=(4, 9), bars=0, low=0.15):
    """(left, right) uint8 [H][W], the left view's disparity FP64 and which of
    its pixels the right view shows."""
    rnd = random.Random(seed)
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    span = dmax - dmin
    tw = W + int(math.ceil(dmax)) + 8
    x = torch.arange(W, device=DEVICE, dtype=torch.float64).expand(H, W)
    y = torch.arange(H, device=DEVICE, dtype=torch.float64)[:, None].expand(H, W)

    def texture(mean, amp):
        t = _blur(torch.rand(H, tw, generator=gen, device=DEVICE, dtype=torch.float64))
        t = (t - t.mean()) / t.std()
        return mean + 0.5 * amp * t

    far = dmin + rnd.uniform(0.0, 0.15) * span
    near = far + rnd.uniform(0.05, 0.25) * span
    tex = texture(rnd.uniform(0.35, 0.65), rnd.uniform(0.35, 0.6))
    for _ in range(3):                                 # low-texture patches of the background
        ph, pw = max(4, H // rnd.randint(3, 8)), max(4, W // rnd.randint(3, 8))
        py, px = rnd.randint(0, max(0, H - ph)), rnd.randint(0, max(0, W - pw))
        patch = tex[py:py + ph, px:px + pw]
        tex[py:py + ph, px:px + pw] = patch.mean() + 0.1 * (patch - patch.mean())
    surfaces = [(far, rnd.uniform(-0.02, 0.02) * span / W, (near - far) / max(1, H - 1),
                 -1e9, 0, 1e9, H, tex)]
    for _ in range(rnd.randint(*planes)):
        ow, oh = rnd.randint(max(6, W // 8), max(7, W // 2)), rnd.randint(max(6, H // 8),
                                                                          max(7, H // 2))
        ox, oy = rnd.randint(0, max(0, W - ow)), rnd.randint(0, max(0, H - oh))
        sx = rnd.uniform(-0.08, 0.08) * min(1.0, span / ow)
        sy = rnd.uniform(-0.08, 0.08) * min(1.0, span / oh)
        a = dmin + rnd.uniform(0.35, 1.0) * span - sx * (ox + ow / 2) - sy * (oy + oh / 2)
        amp = rnd.uniform(0.35, 0.6) * (0.1 if rnd.random() < low else 1.0)
        surfaces.append((a, sx, sy, ox, oy, ox + ow, oy + oh, texture(rnd.uniform(0.2, 0.8), amp)))
    for _ in range(bars):
        bw, bh = rnd.randint(2, 6), rnd.randint(H // 3, H)
        bx, by = rnd.randint(0, W - bw), rnd.randint(0, H - bh)
        surfaces.append((dmin + rnd.uniform(0.8, 1.0) * span, 0.0, 0.0, bx, by, bx + bw, by + bh,
                         texture(rnd.uniform(0.15, 0.85), 0.5)))

    def render(right):
        best = torch.full((H, W), -1e30, device=DEVICE, dtype=torch.float64)
        val = torch.zeros_like(best)
        for a, bx, cy, x0, y0, x1, y1, t in surfaces:
            # right pixel xr shows the left column x with x - d(x, y) = xr
            xs = (x + a + cy * y) / (1.0 - bx) if right else x
            d = a + bx * xs + cy * y
            m = (xs >= x0 - 0.5) & (xs < x1 - 0.5) & (y >= y0) & (y < y1) & (d > best)
            u = (xs + 4.0).clamp(0.0, tw - 1.000001)
            i = u.floor().long()
            f = u - i
            v = t.gather(1, i) * (1.0 - f) + t.gather(1, i + 1) * f
            best, val = torch.where(m, d, best), torch.where(m, v, val)
        return best, (val * 255.0).round().clamp(0, 255).to(torch.uint8)

    dl, left = render(False)
    dr, right = render(True)
    xr = (x - dl).round().long()
    seen = (xr >= 0) & (xr < W) & (dr.gather(1, xr.clamp(0, W - 1)) <= dl + 0.5)
    return left, right, dl.clamp(min=0.0), seen


def _image(u8, kind):
    """The image as the call takes it: samples, or grays in [0, 1]."""
    if kind == "u8":
        return u8.reshape(-1).contiguous()
    return (u8.reshape(-1).double() / 255.0).to(torch.float64 if kind == "f64" else torch.float32)


def _network_like(disp, seed):
    """A disparity map as the network gives it: at work resolution (edges
    smeared over a few pixels), a smooth error of about a pixel, upsampled."""
    H, W = disp.shape
    w = min(W, max(48, min(MAX_WIDTH, int(W / 2.3))))
    h = max(8, int(H * w / W + 0.5))
    gen = torch.Generator(device=DEVICE).manual_seed(seed + 17)
    d = F.interpolate(disp[None, None], size=(h, w), mode="bilinear", align_corners=False)
    e = torch.randn(h, w, generator=gen, device=DEVICE, dtype=torch.float64)
    d = d[0, 0] + 2.5 * (W / w) * _blur(_blur(e))
    d = F.interpolate(d[None, None], size=(H, W), mode="bilinear", align_corners=False)[0, 0]
    return d.clamp(min=0.0).reshape(-1).contiguous()


def _pair(case, seed, **kw):
    left, right, disp, seen = _scene(seed, case["W"], case["H"], 0.0, float(case["dmax"]), **kw)
    return _image(left, case["image"]), _image(right, case["image"]), disp, seen


def _crops(case, seed):
    s = [_scene(seed * 1000 + k, case["W"], case["H"], 2.0, float(case["dmax"]), planes=(2, 4),
                bars=1) for k in range(case["pairs"])]
    return [torch.stack([c[0].float() / 255.0 for c in s]),
            torch.stack([c[1].float() / 255.0 for c in s]),
            torch.stack([c[2].float() for c in s]),
            torch.stack([c[3].to(torch.uint8) for c in s])]


def _colour(u8):
    """8-bit RGB [H][W][3]: the gray level and two smooth transforms of it."""
    H, W = u8.shape
    g = u8.double() / 255.0
    xx = torch.arange(W, device=DEVICE, dtype=torch.float64) / max(1, W - 1)
    yy = torch.arange(H, device=DEVICE, dtype=torch.float64)[:, None] / max(1, H - 1)
    rgb = torch.stack([g, 0.5 * g + 0.5 * xx, 1.0 - 0.7 * g * yy], dim=-1)
    return (rgb * 255.0).round().to(torch.uint8)


def _png(rgb):
    """An 8-bit RGB PNG whose rows cycle through the five filters."""
    H, W, _ = rgb.shape
    cur = rgb.reshape(H, 3 * W).astype(np.int32)
    up = np.vstack([np.zeros((1, 3 * W), np.int32), cur[:-1]])
    left = np.pad(cur, ((0, 0), (3, 0)))[:, :-3]
    corner = np.pad(up, ((0, 0), (3, 0)))[:, :-3]
    p = left + up - corner
    pa, pb, pc = abs(p - left), abs(p - up), abs(p - corner)
    paeth = np.where((pa <= pb) & (pa <= pc), left, np.where(pb <= pc, up, corner))
    guess = [np.zeros_like(cur), left, up, (left + up) >> 1, paeth]
    raw = np.empty((H, 3 * W + 1), np.uint8)
    for y in range(H):
        raw[y, 0] = y % 5
        raw[y, 1:] = (cur[y] - guess[y % 5][y]) & 255

    def chunk(tag, body):
        return (len(body).to_bytes(4, "big") + tag + body +
                zlib.crc32(tag + body).to_bytes(4, "big"))

    head = W.to_bytes(4, "big") + H.to_bytes(4, "big") + bytes([8, 2, 0, 0, 0])
    return (b"\x89PNG\r\n\x1a\n" + chunk(b"IHDR", head) +
            chunk(b"IDAT", zlib.compress(raw.tobytes(), 6)) + chunk(b"IEND", b""))


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    sv, kind, W, H = _package(), case["kind"], case["W"], case["H"]
    s = dict(case)
    dtype = {"u8": torch.uint8, "f32": torch.float32, "f64": torch.float64}[case["image"]]
    if kind in ("lr_refine", "refiner"):
        s["left"], s["right"], disp, _ = _pair(case, seed)
        s["disp0"] = _network_like(disp, seed)
        if kind == "refiner":
            s["call"] = sv.refine.LRRefiner(W, H, **REFINE, tol=TOL)
            s["out"] = torch.empty(W * H, dtype=torch.float64, device=DEVICE)
            s["status"] = torch.empty(W * H, dtype=torch.uint8, device=DEVICE)
    elif kind == "full_range":
        s["left"], s["right"], _, _ = _pair(case, seed, bars=2)
        s["R"] = _full_range_R(case)
        s["disp0"] = torch.full((W * H,), float(s["R"]), dtype=torch.float64, device=DEVICE)
    elif kind == "forward":
        s["left"], s["right"], _, _ = _pair(case, seed)
        s["half"] = F.avg_pool2d(s["left"].reshape(1, H, W), 2).reshape(-1).contiguous()
        s["net"] = _net()
    elif kind == "predict_bf16":
        s["left"], s["right"], _, _ = _pair(case, seed)
        s["net"] = _net()
    elif kind == "pair":
        s["call"] = sv.pipeline.PairPipeline(W, H, _net(), image_dtype=dtype, **REFINE, tol=TOL)
        left, right, _, _ = _pair(case, seed)
        s["call"].left.copy_(left)
        s["call"].right.copy_(right)
    elif kind == "batch":
        sizes = _batch_sizes(case)
        s["call"] = sv.batch.NetBatch([(w, h) for w, h, _ in sizes], _net(), dtype=dtype, **REFINE,
                                      tol=TOL)
        s["stream"] = torch.cuda.Stream()
        for i, (w, h, d) in enumerate(sizes):
            left, right, _, _ = _scene(seed * 1000 + i, w, h, 0.0, d)
            s["call"].left[i].copy_(_image(left, case["image"]))
            s["call"].right[i].copy_(_image(right, case["image"]))
    elif kind == "refine_disparity":
        left, right, disp, _ = _scene(seed, W, H, 0.0, float(case["dmax"]))
        s["left"], s["right"] = _image(left, case["image"]), _image(right, case["image"])
        s["rgb"] = (_colour(left).double() / 255.0).reshape(-1).contiguous()
        s["disp0"] = _network_like(disp, seed)
    elif kind == "train":
        s["crops"] = _crops(case, seed)
        s["call"] = sv.train.Trainer(_net(), lr=1.0e-4)
    elif kind == "band":
        s["left"], s["right"], disp, _ = _pair(case, seed, bars=2)
        s["disp0"] = _network_like(disp, seed)
        gen = torch.Generator(device=DEVICE).manual_seed(seed + 29)
        unsure = _blur(_blur(torch.rand(H, W, generator=gen, device=DEVICE, dtype=torch.float64)))
        s["spread"] = (4.0 * unsure).reshape(-1).contiguous()
        s["pmax"] = (1.0 - unsure).reshape(-1).contiguous()
        s["call"] = sv.band.LearnedBandRefiner(W, H, sv.band.BandNet.load(), dmax=160, **REFINE,
                                               tol=TOL)
        s["out"] = torch.empty(W * H, dtype=torch.float64, device=DEVICE)
        s["status"] = torch.empty(W * H, dtype=torch.uint8, device=DEVICE)
    elif kind == "png":
        s["files"] = [_png(_colour(v).cpu().numpy())
                      for v in _scene(seed, W, H, 0.0, float(case["dmax"]))[:2]]
    return s


def _full_range_R(case):
    return (case["dmax"] + 2) // 2 + 1


# --------------------------------------------------------------------- run
def run(s):
    sv, kind, W, H = _package(), s["kind"], s["W"], s["H"]
    if kind == "lr_refine":
        return sv.refine.lr_refine(s["left"], s["right"], s["disp0"], W, H, tol=TOL, **REFINE)
    if kind == "refiner":
        s["call"].run(s["left"], s["right"], s["disp0"], s["out"], s["status"])
        return s["out"], s["status"]
    if kind == "full_range":
        return sv.refine.lr_refine(s["left"], s["right"], s["disp0"], W, H, tol=TOL,
                                   **dict(REFINE, R=s["R"]))
    if kind == "forward":
        return sv.network.forward(s["net"], s["left"], s["right"], H, W, s["half"], s["left"])
    if kind == "predict_bf16":
        return sv.network.predict(s["net"], s["left"], s["right"], W, H, precision="bf16")
    if kind == "pair":
        call, here = s["call"], torch.cuda.current_stream()
        call.stream.wait_stream(here)
        call.run_device()
        here.wait_stream(call.stream)
        return call.disp0, call.out, call.status
    if kind == "batch":
        call, here = s["call"], torch.cuda.current_stream()
        s["stream"].wait_stream(here)
        with torch.cuda.stream(s["stream"]):
            call.run()
        here.wait_stream(s["stream"])
        return [[call.disparity(i), call.out[i], call.status[i]] for i in range(s["pairs"])]
    if kind == "refine_disparity":
        return sv.post.refine_disparity(s["left"], s["right"], s["rgb"], s["disp0"], W, H,
                                        **REFINE, tol=TOL)
    if kind == "train":
        loss, pred = s["call"].compute_grads(*s["crops"], pred=True)
        return loss, pred, s["call"].grads()
    if kind == "band":
        s["call"].run(s["left"], s["right"], 0, s["disp0"], s["out"], s["status"],
                      torch.cuda.current_stream().cuda_stream, s["spread"], s["pmax"])
        return s["out"], s["status"]
    return [sv.image.decode_image(f, out="cuda")[:2] for f in s["files"]]


# -------------------------------------------------------------------- work
def _net_flops(W, H):
    a = _net().arch
    q, half, full = W * H / 16.0, W * H / 4.0, float(W * H)
    front = 2 * (half * a.feat_C * 9 + q * 3 * a.feat_C * a.feat_C * 9) * 2
    volume = 2 * q * a.D * 27 * (a.feat_C * a.cost_C + a.cost_C * a.cost_C + a.cost_C)
    level = 2 * 9 * (2 * a.refine_C + (len(a.refine_dil) - 1) * a.refine_C ** 2 + a.refine_C)
    return front + volume + level * (half + full)


def _refine_flops(W, H, K):
    """Two views: 8 paths of about 8 operations a candidate, the Hamming cost and the sums."""
    return 2 * W * H * K * (8 * 8 + 2 + 8)


def work(case):
    """Each input read once, each output written once; the operations of the method."""
    kind, W, H = case["kind"], case["W"], case["H"]
    N, px = W * H, {"u8": 1, "f32": 4, "f64": 8}[case["image"]]
    K = 2 * REFINE["R"] + 1
    if kind in ("lr_refine", "refiner"):
        return dict(bytes=N * (2 * px + 8 + 9), flops=_refine_flops(W, H, K))
    if kind == "full_range":
        return dict(bytes=N * (2 * px + 8 + 9),
                    flops=_refine_flops(W, H, 2 * _full_range_R(case) + 1))
    if kind == "forward":
        return dict(bytes=N * (3 * 4 + 1) + 8 * (N + N // 4 + N // 16), flops=_net_flops(W, H))
    if kind == "predict_bf16":
        return dict(bytes=N * (2 * px + 8), flops=_net_flops(W, H))
    if kind in ("pair", "batch"):
        sizes = _batch_sizes(case) if kind == "batch" else [(W, H, case["dmax"])]
        ops = 0
        for w, h, d in sizes:                          # the probe and one chosen work width
            ww = min(w, MAX_WIDTH, max(48, int(w * 20.0 / d)))
            ops += (_refine_flops(w, h, K) + _net_flops(PROBE_WIDTH, PROBE_WIDTH * h / w) +
                    _net_flops(ww, ww * h / w))
        return dict(bytes=sum(w * h for w, h, _ in sizes) * (2 * px + 8 + 9), flops=ops)
    if kind == "refine_disparity":
        # 5 SLIC sweeps (4 windows a pixel, 14 operations) and 40 trial planes a pixel
        return dict(bytes=N * (2 * px + 24 + 8 + 9),
                    flops=_refine_flops(W, H, K) + N * (5 * 4 * 14 + 40 * 6))
    if kind == "train":
        return dict(bytes=case["pairs"] * N * (4 * 4 + 1), flops=case["pairs"] * 3 * _net_flops(W, H))
    if kind == "band":
        net = 2 * 9 * (8 * 16 + 16 * 16 + 16 * 16 + 16 * 2)
        return dict(bytes=N * (2 * px + 3 * 8 + 9), flops=_refine_flops(W, H, K) + N * (net + 161 * 2))
    return dict(bytes=2 * N * (3 + 32), flops=2 * N * 8)


# ------------------------------------------------------------------- exact
def _popcount(v):
    for shift, mask in ((1, 0x5555555555555555), (2, 0x3333333333333333),
                        (4, 0x0F0F0F0F0F0F0F0F), (8, 0x00FF00FF00FF00FF),
                        (16, 0x0000FFFF0000FFFF), (32, 0x00000000FFFFFFFF)):
        v = (v & mask) + ((v >> shift) & mask)
    return v


def _census(img, rx, ry):
    """[H][W] -> the 62 comparisons of each pixel with its clamped window."""
    H, W = img.shape
    ys = torch.arange(-ry, H + ry, device=img.device).clamp(0, H - 1)
    xs = torch.arange(-rx, W + rx, device=img.device).clamp(0, W - 1)
    p = img[ys][:, xs]
    bits = torch.zeros(H, W, dtype=torch.int64, device=img.device)
    for dy in range(2 * ry + 1):
        for dx in range(2 * rx + 1):
            if (dy, dx) != (ry, rx):
                bits = bits * 2 + (p[dy:dy + H, dx:dx + W] < img)
    return bits


def _sweep(cost, base, dx, dy, P1, P2):
    """The path costs of one direction: [H][W][K] integers."""
    flip = (dx if dy == 0 else dy) < 0
    if dy == 0:
        cost, base, side = cost.transpose(0, 1), base.transpose(0, 1), 0
    else:
        side = dx
    if flip:
        cost, base = cost.flip(0), base.flip(0)
    cost, base = cost.contiguous(), base.contiguous()
    n, m, K = cost.shape
    big = 1 << 20
    out = torch.empty_like(cost)
    out[0] = cost[0]
    pad = torch.full((m, 3 * K + 4), big, dtype=cost.dtype, device=cost.device)
    row = torch.arange(m, device=cost.device)
    before = (row - side).clamp(0, m - 1)
    outside = ((row - side < 0) | (row - side >= m))[:, None]
    k = torch.arange(K, device=cost.device)
    for t in range(1, n):
        q = out[t - 1] if side == 0 else out[t - 1][before]
        bq = base[t - 1] if side == 0 else base[t - 1][before]
        least = q.amin(1, keepdim=True)
        pad[:, K + 2:2 * K + 2] = q
        step = (base[t] - bq).clamp(-K - 1, K + 1)[:, None]
        i = k + (K + 2) + step
        best = torch.minimum(pad.gather(1, i), torch.minimum(pad.gather(1, i - 1),
                                                             pad.gather(1, i + 1)) + P1)
        v = cost[t] + torch.minimum(best, least + P2) - least
        out[t] = v if side == 0 else torch.where(outside, cost[t], v)
    if flip:
        out = out.flip(0)
    return out.transpose(0, 1) if dy == 0 else out


def _one_view(cl, cr, disp0, R, P1, P2, invalid):
    H, W = disp0.shape
    K = 2 * R + 1
    base = (disp0 + 0.5).trunc().clamp(min=0).long()
    d = base[..., None] - R + torch.arange(K, device=disp0.device)
    xr = torch.arange(W, device=disp0.device)[None, :, None] - d
    ok = (d >= 0) & (xr >= 0) & (xr < W)
    match = cr.gather(1, xr.clamp(0, W - 1).reshape(H, -1)).reshape(H, W, K)
    cost = torch.where(ok, _popcount(cl[..., None] ^ match), invalid)
    del match, xr, ok, d
    total = torch.zeros_like(cost)
    for dx, dy in ((1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, 1), (1, -1), (-1, -1)):
        total += _sweep(cost, base, dx, dy, P1, P2)
    # the first smallest sum, then the parabola through its neighbours
    at = (total * 256 + torch.arange(K, device=disp0.device)).amin(2) % 256
    edge = (at == 0) | (at == K - 1)
    c = at.clamp(1, max(1, K - 2))[..., None]
    a, m, b = (total.gather(2, (c + o).clamp(0, K - 1))[..., 0].double() for o in (-1, 0, 1))
    den = a - 2.0 * m + b
    off = torch.where(den > 1.0e-9, 0.5 * (a - b) / torch.where(den > 1.0e-9, den, 1.0), 0.0)
    return torch.where(edge, disp0, (base - R + at).double() + off)


def _beside(value, hole, other):
    """Where `hole`: the smaller of the nearest values left and right that are none, or `other`."""
    H, W = value.shape
    x = torch.arange(W, device=value.device).expand(H, W)
    before = torch.where(hole, -1, x).cummax(1).values
    after = torch.where(hole, W, x).flip(1).cummin(1).values.flip(1)
    va = torch.where(before >= 0, value.gather(1, before.clamp(min=0)), 1.0e9)
    vb = torch.where(after < W, value.gather(1, after.clamp(max=W - 1)), 1.0e9)
    v = torch.minimum(va, vb)
    return torch.where(hole, torch.where(v < 1.0e8, v, other), value)


def _lr_refine(left, right, disp0, R, P1, P2, rx, ry):
    H, W = disp0.shape
    invalid = (2 * rx + 1) * (2 * ry + 1) - 1 + 4
    cl, cr = _census(left, rx, ry), _census(right, rx, ry)
    x = torch.arange(W, device=disp0.device, dtype=torch.float64)
    xr = (x - disp0 + 0.5).trunc().long()
    d0r = torch.full((H, W + 1), -1.0, dtype=torch.float64, device=disp0.device)
    d0r.scatter_reduce_(1, torch.where((xr >= 0) & (xr < W), xr, W), disp0, "amax")
    d0r = d0r[:, :W]
    d0r = _beside(d0r, d0r < 0.0, torch.zeros_like(d0r))
    dl = _one_view(cl, cr, disp0, R, int(P1), int(P2), invalid)
    dr = _one_view(cr.flip(1), cl.flip(1), d0r.flip(1), R, int(P1), int(P2), invalid).flip(1)
    xr = (x - dl + 0.5).trunc().long()
    out_of = (xr < 0) | (xr >= W)
    e = dr.gather(1, xr.clamp(0, W - 1))
    bad = ~out_of & ~((dl - e).abs() <= TOL)
    status = torch.where(out_of | (bad & (e > dl)), 1, torch.where(bad, 2, 0))
    out = _beside(torch.where(status == 2, disp0, dl), status == 1, disp0)
    return out.reshape(-1), status.to(torch.uint8).reshape(-1)


def _unit(t, H, W):
    """A prepared image as FP64 grays in [0, 1], [H][W]."""
    return (t.double() / 255.0 if t.dtype == torch.uint8 else t.double()).reshape(H, W)


def _params():
    """The checkpoint's blocks as FP64 tensors by layer."""
    w = _net()
    a, it = w.arch, iter(w.blocks)

    def take(*shape):
        return (torch.from_numpy(next(it)).to(DEVICE).reshape(shape),
                torch.from_numpy(next(it)).to(DEVICE))

    C, M, Rc = a.feat_C, a.cost_C, a.refine_C
    feat = [take(C, i, 3, 3) for i in (1, C, C, C)]
    cost = [take(o, i, 3, 3, 3) for i, o in ((C, M), (M, M), (M, 1))]
    refs = [[take(Rc, 2 if k == 0 else Rc, 3, 3) for k in range(len(a.refine_dil))] +
            [take(1, Rc, 3, 3)] for _ in range(2)]
    return feat, cost, refs


def _resize(x, H2, W2):
    """Bilinear, half-pixel centres, [..., H, W]."""
    H, W = x.shape[-2:]

    def taps(n, m):
        f = ((torch.arange(m, device=x.device, dtype=torch.float64) + 0.5) * (n / m) -
             0.5).clamp(min=0.0)
        i = f.long().clamp(max=n - 1)
        return i, (i + 1).clamp(max=n - 1), f - i

    y0, y1, wy = taps(H, H2)
    x0, x1, wx = taps(W, W2)
    wy = wy[:, None]
    r0, r1 = x[..., y0, :], x[..., y1, :]
    return (r0[..., x0] * ((1 - wy) * (1 - wx)) + r0[..., x1] * ((1 - wy) * wx) +
            r1[..., x0] * (wy * (1 - wx)) + r1[..., x1] * (wy * wx))


def _forward(params, left, right, half):
    """FP64 [B][H][W] -> the disparities at a quarter, half and full size, and
    the cost volume's distribution."""
    feat, cost, refs = params
    a = _net().arch

    def features(x):
        for i, (w, b) in enumerate(feat):
            x = F.conv2d(x, w, b, stride=2 if i < 2 else 1, padding=1)
            x = F.leaky_relu(x, 0.2) if i < 3 else x
        return x

    fl, fr = features(left[:, None]), features(right[:, None])
    w = fl.shape[-1]
    vol = torch.stack([F.pad((fl[..., d:] - fr[..., :w - d]).abs(), (d, 0), value=2.0)
                       for d in range(a.D)], dim=2)
    for i, (k, b) in enumerate(cost):
        vol = F.conv3d(vol, k, b, padding=1)
        vol = F.leaky_relu(vol, 0.2) if i < 2 else vol
    d = torch.arange(a.D, device=left.device, dtype=torch.float64)[:, None, None]
    x = torch.arange(w, device=left.device)
    vol = vol[:, 0] + torch.where((d >= 1) & (x < d), 8.0, 0.0)
    prob = torch.softmax(-vol, dim=1)
    maps = [(prob * d).sum(1)]
    for level, guide in ((0, half), (1, left)):
        up = 2.0 * _resize(maps[-1], *guide.shape[-2:])
        y = torch.stack([up, guide], dim=1)
        for (k, b), dil in zip(refs[level], list(a.refine_dil) + [1]):
            y = F.conv2d(y, k, b, padding=dil, dilation=dil)
            y = F.leaky_relu(y, 0.2) if k.shape[0] > 1 else y
        maps.append(torch.relu(up + y[:, 0]))
    return maps, prob


def _predict(params, left, right):
    half = F.avg_pool2d(left[None], 2)
    return _forward(params, left[None], right[None], half)[0][2][0]


def _predict_auto(params, left, right):
    H, W = left.shape
    target = _net().target_peak

    def width(peak):
        return max(48, min(W, MAX_WIDTH, int(W * target / max(peak, 1.0e-6) + 0.5)))

    def peak(d):
        v = d.reshape(-1).sort().values
        return max(float(v[int(v.numel() * 0.95)]), 0.5)

    def at_scale(w):
        if w >= W:
            return _predict(params, left, right)
        h = max(8, int(H * (w / W) + 0.5))
        d = _predict(params, _resize(left, h, w), _resize(right, h, w))
        return _resize(d, H, W) * (1.0 / (w / W))

    pw = min(PROBE_WIDTH, W)
    ph = max(8, int(H * pw / W + 0.5))
    probe = _predict(params, _resize(left, ph, pw), _resize(right, ph, pw))
    w = width(peak(probe) * (W / pw))
    d = at_scale(w)
    for _ in range(PASSES - 1):
        new = width(peak(d))
        if abs(new - w) <= 0.08 * w:
            break
        w = new
        d = at_scale(w)
    return d


def _train(case, seed):
    """Loss, prediction and gradients of the batch by FP64 autograd."""
    left, right, disp, seen = _crops(case, seed)
    left, right, disp, seen = left.double(), right.double(), disp.double(), seen.bool()
    params = _params()
    flat = [t for group in (params[0], params[1], params[2][0], params[2][1])
            for pair in group for t in pair]
    for t in flat:
        t.requires_grad_(True)

    def pool(t):
        return F.avg_pool2d(t, 2)

    def every(v):
        return v[:, ::2, ::2] & v[:, ::2, 1::2] & v[:, 1::2, ::2] & v[:, 1::2, 1::2]

    half, quarter = 0.5 * pool(disp), 0.25 * pool(pool(disp))
    seen2 = every(seen)
    seen4 = every(seen2)
    maps, prob = _forward(params, left, right, pool(left))
    loss = 0.0
    for weight, got, want, ok in ((0.5, maps[0], quarter, seen4), (0.7, maps[1], half, seen2),
                                  (1.0, maps[2], disp, seen)):
        r = torch.where(ok, torch.sqrt((got - want) ** 2 + 1.0) - 1.0, 0.0)
        loss = loss + weight * r.sum((1, 2)) / ok.sum((1, 2)).clamp(min=1)
    d = torch.arange(prob.shape[1], device=DEVICE, dtype=torch.float64)[:, None, None]
    q = torch.exp(-(d - quarter[:, None]) ** 2 / (2 * 0.8 * 0.8))
    mass = q.sum(1)
    ok = seen4 & (mass > 0)
    q = q / torch.where(mass > 0, mass, 1.0)[:, None]
    ce = -(q * prob.clamp(min=1.0e-300).log()).sum(1)
    loss = loss + 2.0 * torch.where(ok, ce, 0.0).sum((1, 2)) / ok.sum((1, 2)).clamp(min=1)
    loss.mean().backward()
    return (loss.detach(), maps[2].detach(),
            torch.cat([t.grad.reshape(-1) for t in flat]).cpu().numpy())


def exact(case, seed):
    kind, W, H = case["kind"], case["W"], case["H"]
    if kind in ("lr_refine", "refiner", "full_range"):
        left, right, disp, _ = _pair(case, seed, bars=2 if kind == "full_range" else 0)
        R = _full_range_R(case) if kind == "full_range" else REFINE["R"]
        d0 = _network_like(disp, seed).reshape(H, W) if kind != "full_range" else \
            torch.full((H, W), float(R), dtype=torch.float64, device=DEVICE)
        return _lr_refine(left.reshape(H, W), right.reshape(H, W), d0, **dict(REFINE, R=R))
    if kind == "forward":
        left, right, _, _ = _pair(case, seed)
        left, right = _unit(left, H, W), _unit(right, H, W)
        maps, _ = _forward(_params(), left[None], right[None], F.avg_pool2d(left[None], 2))
        return tuple(m.reshape(-1) for m in maps)
    if kind == "predict_bf16":
        left, right, _, _ = _pair(case, seed)
        return _predict(_params(), _unit(left, H, W), _unit(right, H, W)).reshape(-1)
    if kind == "pair":
        # the refined map takes discrete decisions on disp0's last bits
        left, right, _, _ = _pair(case, seed)
        d = _predict_auto(_params(), _unit(left, H, W), _unit(right, H, W))
        return d.reshape(-1), None, None
    if kind == "batch":
        params, out = _params(), []
        for i, (w, h, dmax) in enumerate(_batch_sizes(case)):
            left, right, _, _ = _scene(seed * 1000 + i, w, h, 0.0, dmax)
            left, right = (_unit(_image(v, case["image"]), h, w) for v in (left, right))
            out.append([_predict_auto(params, left, right).reshape(-1), None, None])
        return out
    if kind == "train":
        return _train(case, seed)
    if kind == "png":
        out = []
        for v in _scene(seed, W, H, 0.0, float(case["dmax"]))[:2]:
            rgb = _colour(v).double() / 255.0
            gray = 0.299 * rgb[..., 0] + 0.587 * rgb[..., 1] + 0.114 * rgb[..., 2]
            out.append((gray.reshape(-1), rgb.reshape(-1)))
        return out
    # the learned band and the superpixel planes: chains of discrete choices
    return None
