"""The work a user has this framework do, as cases that can be timed and compared.

A case names an entry point (`call`) and what goes through it:

  device   Engine.process_device: frames already on the GPU, maps left there, every frame of the
           program on one stream (a robotics or video pipeline);
  session  StereoSession.process: numpy images in, numpy maps out (the Python binding);
  batch    Batch.process_device: many pairs of uneven sizes in one call (dataset processing);
  server   Server.submit / wait: a burst of mixed requests from host memory (a service).

Modes are the presets (0 Fast, 1 Balanced, 2 HighQuality).  Sizes are those of the benchmark
(640x480 D64, 1242x375 D192, 1280x720 D128, 1920x1080 D256) and generic ones.  Inputs are seeded
synthetic rectified pairs made on the GPU: blurred noise with flat patches, a scene of slanted
planes, forward-warped with occlusions, sensor noise on both images.

No case has a 64-bit counterpart (`exact` gives None): the path quantises its matching costs,
takes integer minima along scanlines and picks winners, so its maps are decisions whose values
are defined by the single-precision steps themselves.
"""
import math

import numpy as np
import torch

import apg_sgm_b200 as apg
from apg_sgm_b200 import _lib

MAPS = (("disparity", torch.float32), ("confidence", torch.float32), ("invalid_reason", torch.uint8),
        ("reliable_mask", torch.uint8))
# (width, height, max_disparity) of the pairs in a batched call and of the requests of a burst (width
# 0; otherwise the case's own size, a narrower and a lower one in turn)
MIX = ((640, 480, 64), (1242, 375, 192), (1280, 720, 128))
_stream = None


def listed():
    def c(name, call, mode, w, h, d, ch=1, d0=0, hier=0, pairs=1):
        return {"name": name, "call": call, "mode": mode, "width": w, "height": h, "dmax": d, "channels": ch,
                "dmin": d0, "hier": hier, "pairs": pairs}

    return [
        # the smallest frames: thumbnails and low-power cameras, where launches and latency count
        c("small balanced 160x120", "device", 1, 160, 120, 64),
        # the benchmark's camera sizes
        c("balanced 640x480 d64", "device", 1, 640, 480, 64),
        c("balanced 1242x375 d192", "device", 1, 1242, 375, 192),
        c("fast 1280x720 d128", "device", 0, 1280, 720, 128),
        c("balanced 1280x720 d128", "device", 1, 1280, 720, 128),
        # colour frames of an odd size with a range off the 64-disparity grid and a margin below 0
        c("balanced colour 997x611", "device", 1, 997, 611, 90, ch=3, d0=-6),
        # full HD
        c("fast 1920x1080 d256", "device", 0, 1920, 1080, 256),
        # the coarse-to-fine mode
        c("hierarchical 1280x720 d128", "device", 1, 1280, 720, 128, hier=1),
        # the largest: eight paths, sparse prior and refiner at full HD
        c("high quality 1920x1080 d256", "device", 2, 1920, 1080, 256),
        # host arrays in and out through the Python binding
        c("session fast 1280x720 d128", "session", 0, 1280, 720, 128),
        # a call of uneven pairs, inputs and maps on the GPU
        c("batch of 12 uneven pairs", "batch", 1, 0, 0, 0, pairs=12),
        # a burst of mixed requests, one in four of them Fast
        c("server burst of 12", "server", 1, 0, 0, 0, pairs=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["device"] * 6 + ["session"] * 2 + ["batch", "server"])
    c = {"call": call, "mode": 1, "width": 0, "height": 0, "dmax": 0, "channels": 1, "dmin": 0, "hier": 0, "pairs": 1}
    if call in ("batch", "server"):
        c["pairs"] = rng.randint(2, 8)
        c["mode"] = rng.choice([0, 1, 1])
        c["width"] = _log(rng, 160, 960)
        c["height"] = min(_log(rng, 96, 600), c["width"])
        c["dmax"] = min(_log(rng, 16, 128), c["width"] // 2)
        return c
    c["mode"] = rng.choice([0, 0, 1, 1, 1, 2])
    c["width"] = _log(rng, 120, 1920)
    c["height"] = min(_log(rng, 64, 1080), c["width"])
    c["dmax"] = min(_log(rng, 16, 256), max(16, c["width"] - 1))
    c["channels"] = rng.choice([1, 1, 1, 3])
    c["dmin"] = rng.choice([0, 0, 0, 0, 8, -6]) if c["dmax"] > 24 and c["dmax"] < 250 else 0
    c["hier"] = int(c["mode"] == 1 and rng.random() < 0.2)
    return c


def _pairs(case):
    """(width, height, dmax, dmin, channels, mode) of every pair of the case."""
    if case["call"] in ("batch", "server"):
        w, h, d = case["width"], case["height"], case["dmax"]
        mix = ((w, h, d), (w * 3 // 4, h, d), (w, h // 2, max(16, d // 2))) if w else MIX
        return [mix[i % 3] + (0, 1, 0 if case["call"] == "server" and i % 4 == 3 else case["mode"])
                for i in range(case["pairs"])]
    return [(case["width"], case["height"], case["dmax"], case["dmin"], case["channels"], case["mode"])]


def _pair(w, h, dmin, dmax, ch, patches, seed):
    """A rectified pair, uint8 HxW or HxWx3 on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed & 0x7FFFFFFF)
    n = torch.arange(-5, 6, device="cuda", dtype=torch.float32)
    k = torch.exp(-0.5 * (n / 1.5) ** 2)
    k = k / k.sum()
    base = torch.rand((1, 1, h + 10, w + 10), device="cuda", generator=g)
    base = (base.unfold(3, 11, 1) * k).sum(-1)
    base = (base.unfold(2, 11, 1) * k).sum(-1)[0, 0]
    base = (base - base.min()) / (base.max() - base.min()).clamp_min(1e-9) * 255.0
    r = np.random.default_rng(seed)
    left = base.clone()
    for _ in range(patches):  # textureless patches
        pw, ph = int(r.integers(12, max(13, w // 10))), int(r.integers(12, max(13, h // 8)))
        x0, y0 = int(r.integers(0, max(1, w - pw))), int(r.integers(0, max(1, h - ph)))
        left[y0:y0 + ph, x0:x0 + pw] = float(r.integers(0, 256))
    lo, hi = max(0, dmin), max(1, int(0.94 * (dmax - 1)))
    yy = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    xx = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    near = torch.full((h, w), float("inf"), device="cuda")
    disp = torch.zeros((h, w), device="cuda")
    for _ in range(12):  # a Voronoi partition into slanted planes
        sx, sy = r.uniform(0, w), r.uniform(0, h)
        a, b, c = r.uniform(lo, hi), r.uniform(-0.02, 0.02), r.uniform(-0.02, 0.02)
        dist = (xx - sx) ** 2 + (yy - sy) ** 2
        closer = dist < near
        near = torch.where(closer, dist, near)
        disp = torch.where(closer, a + b * (xx - sx) + c * (yy - sy), disp)
    di = disp.clamp(lo, hi).round().to(torch.int64)
    xi = torch.arange(w, device="cuda").expand(h, w)
    xt = xi - di
    flat = (torch.arange(h, device="cuda")[:, None] * w + xt.clamp(0, w - 1)).reshape(-1)
    ok = ((xt >= 0) & (xt < w)).reshape(-1)
    # forward warp, the nearest surface in front: the largest (disparity, source column) per target
    key = torch.where(ok, (di * 4096 + xi).reshape(-1), torch.full_like(flat, -1))
    zbuf = torch.full((h * w,), -1, device="cuda", dtype=torch.int64)
    zbuf.scatter_reduce_(0, flat, key, "amax")
    src = (torch.arange(h, device="cuda")[:, None] * w + (zbuf.clamp_min(0) % 4096).reshape(h, w)).reshape(-1)
    noise = torch.rand((h * w,), device="cuda", generator=g) * 255.0
    right = torch.where(zbuf >= 0, left.reshape(-1)[src], noise).reshape(h, w)
    out = []
    for img in (left, right):
        if ch == 3:
            img = torch.stack([img, 255.0 - img, 0.5 * img + 40.0], -1)
        img = img + torch.randn(img.shape, device="cuda", generator=g) * 2.0
        out.append(img.round().clamp(0, 255).to(torch.uint8).contiguous())
    return out


def _config(mode, dmax, dmin, hier):
    return apg.config_from_mode(mode, dmax, dmin, hier_enable=hier)


def prepare(case, seed):
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()  # a program runs its device frames on one stream
    state = {"call": case["call"]}
    specs = _pairs(case)
    images = [_pair(w, h, dmin, dmax, ch, 24 if mode == 2 else 4, seed * 64 + i)
              for i, (w, h, dmax, dmin, ch, mode) in enumerate(specs)]
    torch.cuda.synchronize()
    w, h, dmax, dmin, ch, mode = specs[0]
    if case["call"] == "device":
        state["engine"] = apg.Engine(_config(mode, dmax, dmin, case["hier"]), stream=_stream.cuda_stream)
        state["images"] = images[0]
        state["out"] = {k: torch.empty((h, w), dtype=t, device="cuda") for k, t in MAPS}
        state["args"] = (images[0][0].data_ptr(), images[0][1].data_ptr(), w, h, w * ch, ch,
                         *(state["out"][k].data_ptr() for k, _ in MAPS))
    elif case["call"] == "session":
        name = ("fast", "balanced", "high_quality")[mode]
        state["session"] = apg.StereoSession(mode=name, max_disparity=dmax, min_disparity=dmin,
                                             memory_policy="bounded_reuse", hierarchical=bool(case["hier"]))
        state["images"] = [a.cpu().numpy() for a in images[0]]
    elif case["call"] == "batch":
        state["batch"] = apg.Batch(_config(mode, dmax, 0, 0))
        state["images"] = images
        state["out"] = [{k: torch.empty((s[1], s[0]), dtype=t, device="cuda") for k, t in MAPS} for s in specs]
        state["pairs"] = [_lib.Pair(a.data_ptr(), b.data_ptr(), s[0], s[1], s[0], 1, s[2],
                                    *(o[k].data_ptr() for k, _ in MAPS))
                          for (a, b), s, o in zip(images, specs, state["out"])]
    else:
        state["server"] = apg.Server(slots=4)
        for w, h, dmax, _, _, mode in sorted(set(specs)):
            state["server"].reserve(w, h, mode=mode, max_disparity=dmax, count=2)
        # page-locked request and result buffers, kept in a ring as a service keeps them
        state["requests"] = [([a.cpu().pin_memory().numpy() for a in im], s,
                              {k: torch.empty((s[1], s[0]), dtype=t).pin_memory().numpy() for k, t in MAPS})
                             for im, s in zip(images, specs)]
    torch.cuda.synchronize()
    return state


def run(state):
    if state["call"] == "device":
        state["engine"].process_device(*state["args"])
        return state["out"]
    if state["call"] == "session":
        r = state["session"].process(*state["images"])
        return {"disparity": r.disparity, "confidence": r.confidence, "invalid_reason": r.invalid_reason,
                "reliable_mask": r.reliable_mask}
    if state["call"] == "batch":
        state["batch"].process_device(state["pairs"])
        return state["out"]
    srv = state["server"]
    tickets = [srv.submit(im[0], im[1], mode=s[5], max_disparity=s[2], out=o) for im, s, o in state["requests"]]
    return [srv.wait(t)[0] for t in tickets]


def work(case):
    """Bytes: both images in, the four maps (10 bytes a pixel) out.  Operations: per voxel, the
    matching cost (descriptor difference, table, two more terms outside Fast, quantisation), the
    cross aggregation (two prefix sums, two differences, two divisions), every path (three candidate
    minima, the addition and subtraction, the running minimum, the sum) and the two winner searches."""
    nbytes = flops = 0.0
    for w, h, dmax, dmin, ch, mode in _pairs(case):
        n, d = w * h, dmax - dmin
        nbytes += 2.0 * n * ch + 10.0 * n
        per = 4 + (0 if mode == 0 else 6 + 6) + 7 * (8 if mode == 2 else 4) + 4
        if case["hier"]:
            per += per / 8  # the half-size pass at half the range
        flops += float(n) * d * per
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    return None
