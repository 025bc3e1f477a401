"""The workloads this framework's speed is judged by, and how to run one of them.

A case is a dict of plain values.  ``kind`` says which public entry point it goes through:

  pipe     ``rts_pipeline_run`` on device buffers: costs, aggregation, winner-takes-all of both
           views and the cross check (the whole-pair call)
  batch    ``rts_batch_run``: several pairs of uneven size in one call
  host     ``Context.pipeline``: the whole-pair call on numpy arrays, copies included
  m_cross  the reference driver's left-view chain, module by module on device buffers, with
           cross-based aggregation and the disparity refinement
  m_box    the same with rank and LoG costs and the box window
  m_aw     the same with adaptive support weights, in either matching direction

``scene`` is the picture: "dots" (the random-dot texture of the repository's benchmark, gray)
or "photo" (shaded colour surfaces with a little texture and noise, whose cross arms are long).
"""
import ctypes
import math
import random

import torch

import rtstereo_gb300 as R

_CTX = None


def _ctx():
    """One context for the process, as a program keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = R.Context(0)
    return _CTX


AGGR = {"box": R.AGGR_BOX, "aw": R.AGGR_AW, "cross": R.AGGR_CROSS}
COST = {"none": R.COST_NONE, "ad": R.COST_AD, "rank": R.COST_RANK, "census": R.COST_CENSUS, "log": R.COST_LOG,
        "ncc": R.COST_NCC}
# the sizes of a mixed stream of pairs (the batched form draws from them)
STREAM = ((320, 240), (640, 480), (1024, 768), (1280, 720), (1920, 1080))


def _pipe(name, aggr, w, h, d, cost1="ad", cost2="census", rad=0, f16=False, scene="dots", cost_out=False,
          kind="pipe"):
    return {"name": name, "kind": kind, "aggr": aggr, "w": w, "h": h, "d": d, "cost1": cost1, "cost2": cost2,
            "rad": rad, "f16": f16, "scene": scene, "cost_out": cost_out}


def listed():
    return [
        # the smallest pair of the benchmark: launches and latency count
        _pipe("cross 384x288 d16", "cross", 384, 288, 16),
        # a full-HD frame pair, the size a production stream has
        _pipe("cross 1080p d128", "cross", 1920, 1080, 128),
        # colour pictures of the size of the usual test pairs, with the driver's disparity range of 60
        _pipe("cross 450x375 d60 photo", "cross", 450, 375, 60, scene="photo"),
        # the benchmark's flagship: 33x33 adaptive support weights
        _pipe("aw 640x480 d64", "aw", 640, 480, 64, rad=16),
        # the same in the FP16 form on an odd colour pair, the cost volume kept for sub-pixel work
        _pipe("aw f16 450x375 d60 photo", "aw", 450, 375, 60, rad=16, f16=True, scene="photo", cost_out=True),
        # full HD with the 9x9 box
        _pipe("box 1080p d128", "box", 1920, 1080, 128, rad=4),
        # 7x7 NCC under the 9x9 box
        _pipe("ncc box 720p d64", "box", 1280, 720, 64, cost1="ncc", cost2="none", rad=4),
        # a batch from the mixed stream, FP16 form as the serving loop has it
        {"name": "batch of 6 f16", "kind": "batch", "n": 6, "pick": 5, "f16": True, "scene": "dots"},
        # a program with frames in host memory
        _pipe("host cross 640x480 d64", "cross", 640, 480, 64, scene="photo", kind="host"),
        # the driver's own order of module calls on device buffers
        {"name": "modules cross 640x480 d64", "kind": "m_cross", "w": 640, "h": 480, "d": 64, "scene": "photo"},
        {"name": "modules box 720p d64", "kind": "m_box", "w": 1280, "h": 720, "d": 64, "rad": 4, "scene": "dots"},
        {"name": "modules aw 240x180 d32", "kind": "m_aw", "w": 240, "h": 180, "d": 32, "rad": 16, "r2l": False,
         "scene": "photo"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, most, wmax=1920, hmax=1080, dmin=8, dmax=128):
    """Width, height and disparities, odd ones among them, of at most `most` cost entries."""
    while True:
        w, h, d = _log(rng, 160, wmax), _log(rng, 100, hmax), _log(rng, dmin, dmax)
        if rng.random() < 0.4:
            d = max(dmin, d // 16 * 16)  # ranges are often round
        if w * h * d <= most and d < w // 2:
            return w, h, d


def draw(rng):
    kind = rng.choice(["cross", "cross", "aw", "box", "ncc", "batch", "host", "m_cross", "m_box", "m_aw"])
    scene = rng.choice(["dots", "photo"])
    f16 = rng.random() < 0.3
    if kind == "cross":
        w, h, d = _size(rng, 130_000_000)
        c1, c2 = rng.choice([("ad", "census"), ("ad", "census"), ("census", "none"), ("rank", "census"),
                             ("log", "census"), ("ad", "none")])
        keep = rng.random() < 0.15 and w * h * d <= 40_000_000
        c = _pipe("", "cross", w, h, d, cost1=c1, cost2=c2, f16=f16 and not keep, scene=scene, cost_out=keep)
    elif kind == "aw":
        rad = rng.choice([16, 16, 8])
        w, h, d = _size(rng, 15_000_000, 960, 720)
        c = _pipe("", "aw", w, h, d, rad=rad, f16=f16, scene=scene, cost_out=rng.random() < 0.3)
    elif kind == "box":
        w, h, d = _size(rng, 200_000_000)
        keep = rng.random() < 0.25 and w * h * d <= 60_000_000
        c = _pipe("", "box", w, h, d, rad=rng.choice([1, 2, 4, 4]), f16=f16, scene=scene, cost_out=keep)
    elif kind == "ncc":
        w, h, d = _size(rng, 58_000_000, 1280, 720)
        c = _pipe("", "box", w, h, d, cost1="ncc", cost2="none", rad=rng.choice([1, 4]), scene=scene)
    elif kind == "batch":
        return {"kind": "batch", "n": rng.randint(2, 6), "pick": rng.randrange(1000), "f16": rng.random() < 0.5,
                "scene": scene}
    elif kind == "host":
        w, h, d = _size(rng, 30_000_000)
        c = _pipe("", "cross", w, h, d, f16=f16, scene=scene, kind="host")
    elif kind == "m_cross":
        w, h, d = _size(rng, 40_000_000, 1280, 720)
        return {"kind": "m_cross", "w": w, "h": h, "d": d, "scene": scene}
    elif kind == "m_box":
        w, h, d = _size(rng, 59_000_000, 1280, 720)
        return {"kind": "m_box", "w": w, "h": h, "d": d, "rad": rng.choice([1, 2, 4]), "scene": scene}
    else:
        w, h, d = _size(rng, 1_380_000, 280, 200, 8, 48)
        return {"kind": "m_aw", "w": w, "h": h, "d": d, "rad": rng.choice([8, 16]), "r2l": rng.random() < 0.4,
                "scene": scene}
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# pictures

def _box3(t):
    p = torch.nn.functional.pad(t[None, None].float(), (1, 1, 1, 1), mode="replicate")
    return torch.nn.functional.avg_pool2d(p, 3, 1)[0, 0]


def _lab(rgb):
    """8-bit CIE Lab of an 8-bit sRGB picture (D65)."""
    c = rgb.float() / 255
    c = torch.where(c <= 0.04045, c / 12.92, ((c + 0.055) / 1.055) ** 2.4)
    m = torch.tensor([[0.412453, 0.357580, 0.180423], [0.212671, 0.715160, 0.072169], [0.019334, 0.119193, 0.950227]],
                     device=rgb.device)
    xyz = (c[..., None, :] * m).sum(-1) / torch.tensor([0.950456, 1.0, 1.088754], device=rgb.device)
    f = torch.where(xyz > 0.008856, xyz.clamp_min(1e-9) ** (1 / 3), 7.787 * xyz + 16 / 116)
    lab = torch.stack([(116 * f[..., 1] - 16) * 255 / 100, 500 * (f[..., 0] - f[..., 1]) + 128,
                       200 * (f[..., 1] - f[..., 2]) + 128], -1)
    return lab.round().clamp(0, 255).to(torch.uint8).contiguous()


def _pair(w, h, d, scene, seed, dev="cuda"):
    """A seeded rectified pair: gray, RGB and Lab of both pictures."""
    rng = random.Random(seed * 1000003 + w * 7919 + h * 31 + d)
    g = torch.Generator(device=dev)
    g.manual_seed(rng.randrange(1 << 40))

    def rand(*s):
        return torch.rand(*s, device=dev, generator=g)

    disp = torch.full((h, w), min(4, d - 1), device=dev, dtype=torch.int64)
    boxes = []
    for _ in range(12 if d <= 64 else 24):
        bw, bh = rng.randint(max(1, w // 12), max(1, w // 3)), rng.randint(max(1, h // 12), max(1, h // 3))
        x, y = rng.randrange(max(1, w - bw)), rng.randrange(max(1, h - bh))
        boxes.append((x, y, bw, bh))
        disp[y:y + bh, x:x + bw] = rng.randrange(d)
    if scene == "dots":
        left = _box3((rand(h, w) * 256).floor())[..., None].expand(h, w, 3)
        sigma = 2.0
    else:
        left = torch.zeros(3, h, w, device=dev)
        for cell, amp in ((160, 110.0), (40, 30.0), (8, 7.0)):
            grid = rand(1, 3, h // cell + 2, w // cell + 2)
            up = torch.nn.functional.interpolate(grid, scale_factor=cell, mode="bilinear", align_corners=False)
            left += amp * up[0, :, :h, :w]
        for x, y, bw, bh in boxes:
            left[:, y:y + bh, x:x + bw] += 50 * rand(3, 1, 1)
        left = (left + 3 * rand(3, h, w)).permute(1, 2, 0)
        sigma = 1.5
    left = left.round().clamp(0, 255)
    xs = (torch.arange(w, device=dev)[None, :] + disp).clamp(max=w - 1)
    right = torch.gather(left, 1, xs[..., None].expand(h, w, 3).contiguous())
    noise = torch.randn(h, w, 1 if scene == "dots" else 3, device=dev, generator=g) * sigma
    right = (right + noise).round().clamp(0, 255)
    out = {}
    for side, im in (("l", left), ("r", right)):
        rgb = im.to(torch.uint8).contiguous()
        luma = im[..., 0] * 0.299 + im[..., 1] * 0.587 + im[..., 2] * 0.114
        out[side + "rgb"] = rgb
        out[side + "gray"] = (rgb[..., 0] if scene == "dots" else luma.round().clamp(0, 255).to(torch.uint8)).contiguous()
    return out


def _params(c):
    kw = {"disp_range": c["d"], "aggr": AGGR[c["aggr"]], "cost1": COST[c["cost1"]], "cost2": COST[c["cost2"]],
          "precision": R.PREC_F16 if c["f16"] else R.PREC_F32, "rank_rad": 3, "ncc_hrad": 3, "ncc_wrad": 3}
    if c["aggr"] == "box":
        kw["box_rad"] = c["rad"]
    elif c["aggr"] == "aw":
        kw["aw_rad"] = c["rad"]
    return R.params(**kw)


def _batch_dims(c):
    rng = random.Random(c["pick"])
    return [rng.choice(STREAM) + (rng.choice((32, 64, 128)),) for _ in range(c["n"])]


def _p(t):
    return 0 if t is None else t.data_ptr()


def _whole(w, h, p, im, scene, cost_out, lab):
    """What one whole-pair call on device buffers takes: the descriptors and the buffers behind them."""
    outs = [torch.empty(h, w, dtype=torch.uint8, device="cuda") for _ in range(3)]
    vol = torch.empty(h, w, p.disp_range, device="cuda") if cost_out else None
    rgb = scene == "photo"  # gray pairs pass no colour pictures
    labs = [_lab(im["lrgb"]), _lab(im["rrgb"])] if lab else [None, None]
    pair = R.Pair(w, h, _p(im["lgray"]), _p(im["rgray"]), _p(im["lrgb"]) if rgb else None,
                  _p(im["rrgb"]) if rgb else None, _p(labs[0]) or None, _p(labs[1]) or None)
    out = R.Out(_p(outs[0]), _p(outs[1]), _p(outs[2]), _p(vol) or None)
    return {"pair": pair, "out": out, "params": p, "outs": outs, "vol": vol, "keep": (im, labs)}


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "pipe":
        im = _pair(c["w"], c["h"], c["d"], c["scene"], seed)
        return {"case": c, **_whole(c["w"], c["h"], _params(c), im, c["scene"], c["cost_out"], c["aggr"] == "aw")}
    if kind == "batch":
        items = []
        for i, (w, h, d) in enumerate(_batch_dims(c)):
            p = R.params(disp_range=d, precision=R.PREC_F16 if c["f16"] else R.PREC_F32)
            items.append(_whole(w, h, p, _pair(w, h, d, c["scene"], seed * 64 + i), c["scene"], False, False))
        return {"case": c, "items": items}
    im = _pair(c["w"], c["h"], c["d"], c["scene"], seed)
    if kind == "host":
        names = ["lgray", "rgray"] + (["lrgb", "rrgb"] if c["scene"] == "photo" else [])
        return {"case": c, "params": _params(c), "in": [im[n].cpu().numpy() for n in names]}
    h, w, d = c["h"], c["w"], c["d"]

    def f(*s):
        return torch.empty(*s, device="cuda")

    def u8(*s):
        return torch.empty(*s, dtype=torch.uint8, device="cuda")

    s = {"case": c, **im, "cost1": f(h, w, d), "disp": u8(h, w)}
    if kind == "m_cross":
        s.update(cost2=f(h, w, d), fin=f(h, w, d), bl=u8(h, w, 63), br=u8(h, w, 63))
        for n in ("hl", "hr", "vl", "vr"):
            s[n] = torch.empty(h, w, 2, dtype=torch.int32, device="cuda")
    elif kind == "m_box":
        s.update(cost2=f(h, w, d), kl=u8(h, w), kr=u8(h, w), ll=f(h, w), lr=f(h, w),
                 mask=torch.from_numpy(R.LOG5x5).cuda())
    else:
        area = (2 * c["rad"] + 1) ** 2
        s.update(wl=f(h, w, area), wr=f(h, w, area), fin=None if c["r2l"] else f(h, w, d), llab=_lab(im["lrgb"]),
                 rlab=_lab(im["rrgb"]), prox=torch.from_numpy(_ctx().calcProxWeight(36.0, c["rad"])).cuda())
    return s


def run(state):
    s, c = state, state["case"]
    ctx, kind, dev = _ctx(), c["kind"], R.DEVICE
    if kind == "pipe":
        ctx.call("pipeline_run", dev, ctypes.byref(s["pair"]), ctypes.byref(s["params"]), ctypes.byref(s["out"]))
        return s["outs"] + ([s["vol"]] if s["vol"] is not None else [])
    if kind == "batch":
        items = s["items"]
        ctx.batch_run([i["pair"] for i in items], [i["params"] for i in items], [i["out"] for i in items])
        return [i["outs"] for i in items]
    if kind == "host":
        return list(ctx.pipeline(s["params"], *s["in"])[:3])
    h, w, d = c["h"], c["w"], c["d"]
    if kind == "m_cross":
        ctx.call("pixelBasedCostL2R_Color_trunc", dev, s["lrgb"], s["rrgb"], s["cost1"], d, h, w, 24.0, 0)
        ctx.call("calcCensusTrans", dev, s["lgray"], s["bl"], 4, 3, h, w)
        ctx.call("calcCensusTrans", dev, s["rgray"], s["br"], 4, 3, h, w)
        ctx.call("calcHammingDist", dev, s["bl"], s["br"], s["cost2"], 4, 3, h, w, d)
        ctx.call("combineCost", dev, s["cost1"], s["cost2"], 10.0, 10.0, h, w, d)
        ctx.call("findCross", dev, s["lrgb"], s["hl"], s["vl"], h, w)
        ctx.call("findCross", dev, s["rrgb"], s["hr"], s["vr"], h, w)
        ctx.call("aggregate_cost_horizontal", dev, s["cost1"], h, w, d)
        ctx.call("cross_stereo_aggregation", dev, s["cost1"], s["fin"], s["hl"], s["hr"], s["vl"], s["vr"], h, w, d)
        ctx.call("WTA", dev, s["fin"], s["disp"], h, w, d)
        ctx.call("disp_refinement", dev, s["disp"], s["hl"], s["vl"], h, w, d)
        return {n: s[n] for n in ("cost1", "cost2", "fin", "bl", "br", "hl", "hr", "vl", "vr", "disp")}
    if kind == "m_box":
        ctx.call("calculateRankFilt", dev, s["lgray"], s["kl"], 3, h, w)
        ctx.call("calculateRankFilt", dev, s["rgray"], s["kr"], 3, h, w)
        ctx.call("pixelBasedL2R", dev, s["kl"], s["kr"], s["cost1"], d, h, w)
        ctx.call("convolveImage", dev, s["lgray"], s["ll"], s["mask"], h, w, 2, 2)
        ctx.call("convolveImage", dev, s["rgray"], s["lr"], s["mask"], h, w, 2, 2)
        ctx.call("pixelBasedCostL2R_Float", dev, s["ll"], s["lr"], s["cost2"], d, h, w)
        ctx.call("combineCost", dev, s["cost1"], s["cost2"], 10.0, 10.0, h, w, d)
        ctx.call("boxAggregate", dev, s["cost1"], h, w, d, c["rad"])
        ctx.call("WTA", dev, s["cost1"], s["disp"], h, w, d)
        return {n: s[n] for n in ("cost1", "cost2", "kl", "kr", "ll", "lr", "disp")}
    r = c["rad"]
    ctx.call("pixelBasedR2L_Color" if c["r2l"] else "pixelBasedCostL2R_Color", dev, s["lrgb"], s["rrgb"], s["cost1"],
             d, h, w, 1)
    ctx.call("computeWeights", dev, s["wl"], s["prox"], s["llab"], 7.0, h, w, r)
    ctx.call("computeWeights", dev, s["wr"], s["prox"], s["rlab"], 7.0, h, w, r)
    if c["r2l"]:
        ctx.call("calcAWCostR2L", dev, s["wl"], s["wr"], s["cost1"], h, w, d, r)
    else:
        ctx.call("calcAWCostL2R", dev, s["wl"], s["wr"], s["cost1"], s["fin"], h, w, d, r)
    ctx.call("WTA", dev, s["cost1"] if c["r2l"] else s["fin"], s["disp"], h, w, d)
    return {n: s[n] for n in ("cost1", "wl", "wr", "fin", "disp") if s[n] is not None}


# ---------------------------------------------------------------------------
# work

def _pair_work(w, h, d, aggr, cost1, rad, colour, lab, cost_out, f16):
    """Pictures in, maps out; operations of both views at the least each entry takes."""
    px, e = w * h, w * h * d
    taps = (2 * rad + 1) ** 2
    agg = {"cross": 16, "box": taps + 1, "aw": 4 * taps + 1}[aggr]
    cost = 5 * 49 + 2 if cost1 == "ncc" else 8
    views = 1 if f16 and aggr != "cross" and cost1 != "ncc" else 2
    return {"bytes": px * (2 + 6 * colour + 6 * lab + 3) + 4 * e * cost_out, "flops": views * e * (agg + cost + 1)}


def work(case):
    c, kind = case, case["kind"]
    if kind in ("pipe", "host"):
        return _pair_work(c["w"], c["h"], c["d"], c["aggr"], c["cost1"], c["rad"], c["scene"] == "photo",
                          c["aggr"] == "aw", c["cost_out"], c["f16"])
    if kind == "batch":
        each = [_pair_work(w, h, d, "cross", "ad", 0, c["scene"] == "photo", False, False, c["f16"])
                for w, h, d in _batch_dims(c)]
        return {k: sum(x[k] for x in each) for k in ("bytes", "flops")}
    px = c["w"] * c["h"]
    e = px * c["d"]
    # each call reads its inputs and writes its outputs once
    if kind == "m_cross":
        # AD, census and Hamming, combine, arms, running sums, aggregation, WTA, refinement
        b = px * 6 + 4 * e + 2 * px * (1 + 63) + px * 126 + 4 * e + 12 * e + 2 * px * (3 + 16) + 8 * e \
            + 8 * e + 32 * px + 4 * e + px + 18 * px
        return {"bytes": b, "flops": e * 30}
    if kind == "m_box":
        b = 2 * px * 2 + 2 * px + 4 * e + 2 * px * 5 + 8 * px + 4 * e + 12 * e + 8 * e + 4 * e + px
        return {"bytes": b, "flops": e * ((2 * c["rad"] + 1) ** 2 + 12)}
    area = (2 * c["rad"] + 1) ** 2
    b = 6 * px + 4 * e + 2 * px * (3 + 4 * area) + 2 * px * 4 * area + 8 * e + 4 * e + px
    return {"bytes": b, "flops": e * (4 * area + 10) + 2 * px * area * 10}


# ---------------------------------------------------------------------------
# the same in 64 bits

def _wrap(t, dy, dx):
    """t[y + dy][x + dx], indices wrapped at the borders."""
    return torch.roll(t, (-dy, -dx), (0, 1))


def _tar(w, d, r2l=False):
    x, k = torch.arange(w, device="cuda")[:, None], torch.arange(d, device="cuda")[None, :]
    return (x + k) % w if r2l else (x - k) % w  # [w][d]


def _census(g):
    g = g.to(torch.int32)
    return torch.stack([(g > _wrap(g, dy, dx)) for dy in range(-4, 5) for dx in range(-3, 4)], -1)


def _hamming(a, b, t):
    out = torch.zeros(a.shape[0], *t.shape, dtype=torch.float64, device="cuda")
    for k in range(a.shape[-1]):
        out += a[:, :, k, None] ^ b[:, :, k][:, t]
    return out


def _ad(a, b, t, trunc=None):
    a, b = a.double(), b.double()
    if a.dim() == 2:
        v = (a[:, :, None] - b[:, t]).abs()
    else:
        v = sum((a[:, :, None, k] - b[:, :, k][:, t]).abs() for k in range(3))
    return v if trunc is None else v.clamp(max=trunc)


def _combine(a, b, l1=10.0, l2=10.0):
    return (1 - torch.exp(-a / l1)) + (1 - torch.exp(-b / l2))


def _box(c, r):
    out = torch.zeros_like(c)
    for dy in range(-r, r + 1):
        for dx in range(-r, r + 1):
            out += _wrap(c, dy, dx)
    return out / (2 * r + 1) ** 2


def _arms(rgb, arm=17, tau=20):
    """left, right, up, down: outward while the last pixel seen is within tau, at most arm, inside the picture."""
    h, w, _ = rgb.shape
    c = rgb.to(torch.int32)
    y, x = torch.arange(h, device="cuda")[:, None].expand(h, w), torch.arange(w, device="cuda")[None].expand(h, w)
    got = []
    for dy, dx, room in ((0, -1, x), (0, 1, w - 1 - x), (-1, 0, y), (1, 0, h - 1 - y)):
        n = torch.zeros(h, w, dtype=torch.int64, device="cuda")
        on = torch.ones(h, w, dtype=torch.bool, device="cuda")
        for k in range(1, arm + 1):
            on = on & (room >= k)
            n += on
            on = on & ((c - _wrap(c, dy * k, dx * k)).abs().amax(-1) < tau)
        got.append(n)
    return got


def _cross(pre, al, ar, t):
    """Cross-based means from running sums along the rows."""
    h, w, d = pre.shape
    x = torch.arange(w, device="cuda")[None, :, None]
    l, r, up, dn = (torch.minimum(a[:, :, None], b[:, t]) for a, b in zip(al, ar))
    seg = pre.gather(1, (x + r).clamp(max=w - 1)) - pre.gather(1, (x - l - 1).clamp(min=0))
    zero = torch.zeros(1, w, d, dtype=torch.float64, device="cuda")
    total = torch.cat([zero, seg.cumsum(0)])
    count = torch.cat([zero, (l + r + 1).double().cumsum(0)])
    y = torch.arange(h, device="cuda")[:, None, None]
    hi, lo = y + dn + 1, y - up
    return (total.gather(0, hi) - total.gather(0, lo)) / (count.gather(0, hi) - count.gather(0, lo))


def _weights(lab, r, gp=36.0, gs=7.0):
    h, w, _ = lab.shape
    v = lab.double()
    y, x = torch.arange(h, device="cuda")[:, None], torch.arange(w, device="cuda")[None]
    for dy in range(-r, r + 1):
        for dx in range(-r, r + 1):
            near = math.exp(-math.sqrt(dy * dy + dx * dx) / gp)
            inside = (y + dy >= 0) & (y + dy < h) & (x + dx >= 0) & (x + dx < w)
            yield dy, dx, near * torch.exp(-(v - _wrap(v, dy, dx)).square().sum(-1).sqrt() / gs) * inside


def _aw(cost, llab, rlab, r, t, r2l=False):
    num, den = torch.zeros_like(cost), torch.zeros_like(cost)
    for (dy, dx, a), (_, _, b) in zip(_weights(llab, r), _weights(rlab, r)):
        k = _wrap(a, dy, dx)[:, :, None] * _wrap(b, dy, dx)[:, t] if r2l else a[:, :, None] * b[:, t]
        num += k * _wrap(cost, dy, dx)
        den += k
    return num / den


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("batch", "host") or (kind == "pipe" and not c["cost_out"]):
        return None
    im = _pair(c["w"], c["h"], c["d"], c["scene"], seed)
    t = _tar(c["w"], c["d"], c.get("r2l", False))
    if kind == "m_cross" or (kind == "pipe" and c["aggr"] == "cross"):
        if kind == "pipe" and (c["cost1"], c["cost2"]) != ("ad", "census"):
            return None
        ham = _hamming(_census(im["lgray"]), _census(im["rgray"]), t)
        pre = _combine(_ad(im["lrgb"], im["rrgb"], t, 24.0), ham).cumsum(1)
        fin = _cross(pre, _arms(im["lrgb"]), _arms(im["rrgb"]), t)
        if kind == "pipe":
            return [None, None, None, fin]
        return {"cost1": pre, "cost2": ham, "fin": fin}
    if kind == "pipe":
        if (c["cost1"], c["cost2"]) != ("ad", "census"):
            return None
        cost = _combine(_ad(im["lrgb"], im["rrgb"], t), _hamming(_census(im["lgray"]), _census(im["rgray"]), t))
        fin = _box(cost, c["rad"]) if c["aggr"] == "box" else _aw(cost, _lab(im["lrgb"]), _lab(im["rrgb"]), c["rad"], t)
        return [None, None, None, fin]
    if kind == "m_box":
        def rank(g):
            g = g.to(torch.int32)
            return 1 + sum((_wrap(g, dy, dx) < g).to(torch.int32) for dy in range(-3, 4) for dx in range(-3, 4))

        mask = torch.from_numpy(R.LOG5x5).double().reshape(5, 5)

        def log(g):
            g = g.double()
            v = sum(_wrap(g, dy, dx) * mask[dy + 2, dx + 2].item() for dy in range(-2, 3) for dx in range(-2, 3))
            return v.abs().clamp(max=255)

        ll, lr = log(im["lgray"]), log(im["rgray"])
        cost2 = _ad(ll, lr, t)
        cost1 = _box(_combine(_ad(rank(im["lgray"]), rank(im["rgray"]), t), cost2), c["rad"])
        return {"cost1": cost1, "cost2": cost2, "ll": ll, "lr": lr}
    llab, rlab = _lab(im["lrgb"]), _lab(im["rrgb"])
    cost = _ad(im["lrgb"], im["rrgb"], t) / 3
    fin = _aw(cost, llab, rlab, c["rad"], t, c["r2l"])
    wl, wr = (torch.stack([v for _, _, v in _weights(lab, c["rad"])], -1) for lab in (llab, rlab))
    if c["r2l"]:
        return {"cost1": fin, "wl": wl, "wr": wr}
    return {"cost1": cost, "wl": wl, "wr": wr, "fin": fin}
