"""The work that is timed: template searches, pose scoring and teaching through the public Python operators.

A case is a dict of plain values.  `kind` names the operator:

  find        one FindNccModel call (camera frame in host memory, or already in device memory)
  batch       one FindNccModels call over many frames, several finds in flight
  models      one FindNccModels call with several models
  gradient    NCC and its gradient at many similarity poses
  similarity  Gauss-Newton refinement of many similarity poses
  teach       CreateNccModel from a template, the first search with it, and its release

Inputs are seeded synthetic scenes: a smoothed-noise background, filled rectangles and ellipses, the templates pasted
at known sub-pixel poses by bilinear warping, then additive noise.
"""
import contextlib
import math
import random

import numpy as np
import torch

import mvkit_gb300 as mg

PI = math.pi
DEFAULTS = dict(range_deg=30.0, bits=8, levels=0, min_score=0.7, overlap=0.5, poses=1, memory="host", subpixel=True,
                lowest=1, domain="", candidates=0, images=1, workers=1, sides="")


def listed():
    return [
        # an inspection station's smallest call: one part at a fixed orientation in a VGA frame
        dict(name="find_480x640_t64", kind="find", height=480, width=640, side=64, range_deg=0.0, levels=3,
             min_score=0.8),
        # a small frame of odd size, small rotations, two parts
        dict(name="find_523x701_t47", kind="find", height=523, width=701, side=47, range_deg=10.0, levels=3, poses=2),
        # a 4-megapixel frame from the host, +-30 degrees, five parts: the common robot-guidance call
        dict(name="find_2048_t128", kind="find", height=2048, width=2048, side=128, levels=4, poses=5,
             candidates=1 << 16),
        # the same search over a stream of frames that are already on the GPU, many in flight (throughput)
        dict(name="batch_32x2048_t128", kind="batch", height=2048, width=2048, side=128, levels=4, poses=5,
             images=32, workers=32, memory="device", candidates=1 << 16),
        # any orientation, automatic levels, a low score bound: most candidates have to be refined to be refused
        dict(name="find_1024x1280_t48_360", kind="find", height=1024, width=1280, side=48, range_deg=180.0,
             min_score=0.6, poses=6, candidates=1 << 18),
        # a region of interest inside an odd-sized frame, pixel-accurate poses only
        dict(name="find_1201x1603_t96_roi", kind="find", height=1201, width=1603, side=96, range_deg=20.0, levels=4,
             poses=3, domain="patches", subpixel=False, candidates=1 << 16),
        # several part types in one frame
        dict(name="models_1024x1280_3", kind="models", height=1024, width=1280, sides="48,64,101", range_deg=20.0,
             levels=3, poses=2, candidates=1 << 16),
        # a 12-bit camera, the frame on the GPU
        dict(name="find_2048_u16_t128", kind="find", height=2048, width=2048, side=128, bits=12, levels=4, poses=5,
             min_score=0.6, memory="device", candidates=1 << 16),
        # a large 12-bit frame with a large template over half a circle
        dict(name="find_4096_u16_t256", kind="find", height=4096, width=4096, side=256, bits=12, range_deg=90.0,
             levels=5, min_score=0.5, overlap=0.3, poses=12, memory="device", candidates=1 << 18),
        # scores and gradients of 256 poses of a 26-megapixel frame (a caller's own optimiser)
        dict(name="gradient_5120_t128", kind="gradient", height=5120, width=5120, side=128, range_deg=180.0,
             poses=256, memory="device", levels=3),
        # scaled parts refined in row, column, angle and scale
        dict(name="similarity_3000x4096_t161", kind="similarity", height=3000, width=4096, side=161, range_deg=180.0,
             poses=64, levels=3, candidates=1 << 16),
        # a new part is taught and found once
        dict(name="teach_t128", kind="teach", height=480, width=640, side=128, range_deg=30.0, levels=4),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["find", "find", "find", "find", "batch", "models", "gradient", "similarity", "teach"])
    h, w = log(300, 3000), log(300, 3000)
    side = max(32, min(log(32, 200), min(h, w) // 8))
    levels = 4 if side >= 96 else 3 if side >= 40 else 2
    c = dict(kind=kind, height=h, width=w, side=side, levels=levels, poses=rng.randint(1, 5),
             min_score=round(rng.uniform(0.55, 0.8), 2), memory=rng.choice(["host", "device"]),
             bits=rng.choice([8, 8, 12]), range_deg=round(rng.uniform(5, 45), 1), candidates=1 << 18)
    if kind == "find":
        if rng.random() < 0.2:
            c["range_deg"] = rng.choice([0.0, 180.0])
        if rng.random() < 0.25:
            c["domain"] = "patches"
        if rng.random() < 0.25:
            c["subpixel"] = False
        elif rng.random() < 0.2 and levels > 2:
            c["lowest"] = 2
    elif kind == "batch":
        c["height"], c["width"] = min(h, 1600), min(w, 1600)
        c["images"] = rng.randint(3, 24)
        c["workers"] = rng.choice([4, 8, 16])
    elif kind == "models":
        c["height"], c["width"] = min(h, 1600), min(w, 1600)
        c["sides"] = ",".join(str(max(32, min(log(32, 128), min(h, w) // 10))) for _ in range(rng.randint(2, 4)))
        c["levels"] = 2
        c["range_deg"] = min(c["range_deg"], 20.0)
        c["poses"] = rng.randint(1, 2)
        del c["side"]
    elif kind in ("gradient", "similarity"):
        c["poses"] = log(4, 256)
        c["levels"] = 2
        c["range_deg"] = 180.0
    else:
        c["height"], c["width"] = 480 + h % 160, 640 + w % 160
        c["side"] = min(side, 128)
        c["levels"] = 2 if c["side"] < 40 else 3
    return c


# ------------------------------------------------------------------ inputs
def _full(case):
    return {**DEFAULTS, **case}


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _scene(gen, h, w, maxval, shapes, rng):
    dev = _device()
    unit = (maxval + 1) / 256.0
    v = torch.rand((1, 1, h, w), generator=gen, device=dev)
    for _ in range(3):
        v = torch.nn.functional.avg_pool2d(v, 7, 1, 3, count_include_pad=False)
    v = v[0, 0].double()
    v = (128 + (v - v.mean()) / v.std() * 20) * unit
    for _ in range(shapes):
        cy, cx = rng.randrange(h), rng.randrange(w)
        hy = rng.randint(max(2, h // 64), max(3, h // 8))
        hx = rng.randint(max(2, w // 64), max(3, w // 8))
        val = rng.randint(30, 220) * unit
        r0, r1, c0, c1 = max(0, cy - hy), min(h, cy + hy + 1), max(0, cx - hx), min(w, cx + hx + 1)
        sub = v[r0:r1, c0:c1]
        if rng.random() < 0.5:
            sub[:] = val
        else:
            yy = (torch.arange(r0, r1, device=dev) - cy)[:, None].double() / hy
            xx = (torch.arange(c0, c1, device=dev) - cx)[None, :].double() / hx
            sub[yy * yy + xx * xx <= 1] = val
    return v


def _finish(v, gen, sigma, maxval):
    n = torch.randn(v.shape, generator=gen, device=v.device, dtype=torch.float32)
    return (v + n * sigma).round().clamp(0, maxval)


def _array(v, maxval):
    if maxval < 256:
        return v.to(torch.uint8).cpu().numpy()
    return v.to(torch.int32).cpu().numpy().astype(np.uint16)


def _paste(img, tmpl, row, col, angle, scale):
    t = tmpl.shape[0]
    o = (t - 1) / 2.0
    ca, sa = math.cos(angle), math.sin(angle)
    reach = scale * math.hypot(t, t) / 2 + 2
    r0, r1 = max(0, int(row - reach)), min(img.shape[0], int(row + reach) + 2)
    c0, c1 = max(0, int(col - reach)), min(img.shape[1], int(col + reach) + 2)
    y = torch.arange(r0, r1, device=img.device, dtype=torch.float64)[:, None] - row
    x = torch.arange(c0, c1, device=img.device, dtype=torch.float64)[None, :] - col
    tr, tc = (ca * y + sa * x) / scale + o, (ca * x - sa * y) / scale + o
    ok = (tr >= 0) & (tc >= 0) & (tr <= t - 1) & (tc <= t - 1)
    tr, tc = tr.clamp(0, t - 1), tc.clamp(0, t - 1)
    ri, ci = tr.floor().long().clamp(max=t - 2), tc.floor().long().clamp(max=t - 2)
    fr, fc = tr - ri, tc - ci
    v = (1 - fr) * ((1 - fc) * tmpl[ri, ci] + fc * tmpl[ri, ci + 1]) + \
        fr * ((1 - fc) * tmpl[ri + 1, ci] + fc * tmpl[ri + 1, ci + 1])
    sub = img[r0:r1, c0:c1]
    sub[ok] = v[ok]


def _sides(c):
    return [int(s) for s in c["sides"].split(",")] if c["sides"] else [c["side"]]


def _templates(c, seed):
    rng = random.Random("t%d" % seed)
    gen = torch.Generator(device=_device())
    gen.manual_seed(7919 * seed + 17)
    maxval = (1 << c["bits"]) - 1
    out = []
    for side in _sides(c):
        src = _scene(gen, 2 * side, 2 * side, maxval, 10, rng)
        # the crop a user would teach: the one with most structure of a few
        at = [(rng.randint(0, side), rng.randint(0, side)) for _ in range(12)]
        y, x = max(at, key=lambda p: float(src[p[0]:p[0] + side, p[1]:p[1] + side].std()))
        out.append(_finish(src[y:y + side, x:x + side], gen, 3 * (maxval + 1) / 256, maxval))
    return out


def _frame(c, seed, index, templates):
    """One frame and its pasted poses (template index, row, column, angle, scale; pixel centres)."""
    rng = random.Random("f%d/%d" % (seed, index))
    gen = torch.Generator(device=_device())
    gen.manual_seed(104729 * seed + 31 * index + 5)
    maxval = (1 << c["bits"]) - 1
    h, w = c["height"], c["width"]
    img = _scene(gen, h, w, maxval, 40, rng)
    lim = math.radians(c["range_deg"]) * 0.98
    scaled = c["kind"] in ("gradient", "similarity")
    placed = []
    for k, t in enumerate(templates):
        diag = math.hypot(t.shape[0], t.shape[0]) * (1.05 if scaled else 1)
        margin = diag / 2 + 8
        for _ in range(c["poses"]):
            for _ in range(200):
                row = rng.uniform(margin, max(margin, h - 1 - margin))
                col = rng.uniform(margin, max(margin, w - 1 - margin))
                if all(math.hypot(row - p[1], col - p[2]) > (diag + p[5]) / 2 + 4 for p in placed):
                    scale = rng.uniform(0.96, 1.04) if scaled else 1.0
                    placed.append((k, row, col, rng.uniform(-lim, lim), scale, diag))
                    break
    for k, row, col, angle, scale, _ in placed:
        _paste(img, templates[k].double(), row, col, angle, scale)
    img = _finish(img, gen, 3 * (maxval + 1) / 256, maxval)
    return img, [p[:5] for p in placed], rng


def _domain(c, poses, rng):
    """A reduced domain: a rectangle around each part's rough position and one elsewhere."""
    d = np.zeros((c["height"], c["width"]), dtype=np.uint8)
    for _, row, col, _, _ in poses:
        a, b = rng.randint(20, 90), rng.randint(20, 90)
        d[max(0, int(row) - a):int(row) + a, max(0, int(col) - b):int(col) + b] = 1
    r, k = rng.randrange(c["height"]), rng.randrange(c["width"])
    d[r:r + 150, k:k + 150] = 1
    return d


def _starts(c, poses, rng):
    """Rough similarity poses a caller has before the refinement (several of a part where there are few parts)."""
    return np.array([(r + rng.uniform(-0.6, 0.6), q + rng.uniform(-0.6, 0.6), a + rng.uniform(-0.005, 0.005), 1.0)
                     for _, r, q, a, _ in (poses[i % len(poses)] for i in range(c["poses"]))])


def _image(c, v):
    a = _array(v, (1 << c["bits"]) - 1)
    return mg.DeviceImage(a) if c["memory"] == "device" else a


def _budgets(c):
    if not c["candidates"]:
        return contextlib.nullcontext()
    return mg.extended_budgets(samples=200_000_000, candidates=c["candidates"])


def _range(c):
    a = math.radians(c["range_deg"])
    return -a, min(2 * a, 2 * PI)


def prepare(case, seed):
    c = _full(case)
    maxval = (1 << c["bits"]) - 1
    a0, ext = _range(c)
    templates = _templates(c, seed)
    frames = [_frame(c, seed, i, templates) for i in range(c["images"])]
    s = dict(c=c, images=[_image(c, f[0]) for f in frames])
    arrays = [_array(t, maxval) for t in templates]
    if c["kind"] == "teach":
        s["template"] = arrays[0]
        return s
    levels = c["levels"] or "auto"
    with _budgets(c):
        s["models"] = [mg.create_ncc_model(t, levels, a0, ext, "auto", "use_polarity") for t in arrays]
    img, poses, rng = frames[0]
    s["controls"] = (a0, ext, c["min_score"], c["poses"], c["overlap"], "true" if c["subpixel"] else "false",
                     [c["levels"], c["lowest"]])
    s["domain"] = _domain(c, poses, rng) if c["domain"] else None
    if c["kind"] in ("gradient", "similarity"):
        s["poses"] = _starts(c, poses, rng)
    return s


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind == "gradient":
        return mg.ncc_score_gradient(state["images"][0], state["models"][0], state["poses"])
    if kind == "similarity":
        return mg.ncc_refine_similarity(state["images"][0], state["models"][0], state["poses"])
    with _budgets(c):
        if kind == "find":
            return mg.find_ncc_model(state["images"][0], state["models"][0], *state["controls"],
                                     domain=state["domain"])
        if kind == "batch":
            got = mg.find_ncc_models_batch(state["images"], state["models"], *state["controls"],
                                           workers=c["workers"])
            return [np.concatenate([g[k] for g in got]) for k in range(5)] + [np.array([len(g[0]) for g in got])]
        if kind == "models":
            a0, ext, score, quota, overlap, sub, levels = state["controls"]
            return mg.find_ncc_models(state["images"][0], state["models"], a0, ext, score,
                                      [quota] * len(state["models"]), overlap, sub, levels)
        a0, ext = _range(c)
        model = mg.create_ncc_model(state["template"], c["levels"] or "auto", a0, ext, "auto", "use_polarity")
        out = mg.find_ncc_model(state["images"][0], model, a0, ext, c["min_score"], c["poses"], c["overlap"], "true",
                                c["levels"])
        params = mg.get_ncc_model_params(model)
        model.clear()
        return [*out, np.array(params[:4])]


# ------------------------------------------------------------------- work
def work(case):
    """What any search of this kind does at least: the dense correlation at the top pyramid level with every coarse
    angle, the pyramid's sums, and the image and template read once."""
    c = _full(case)
    bpp = 1 if c["bits"] == 8 else 2
    px = c["height"] * c["width"]
    nbytes, flops = 0.0, 0.0
    for side in _sides(c):
        n = side * side
        if c["kind"] in ("gradient", "similarity"):
            passes = 1 if c["kind"] == "gradient" else 4
            nbytes += c["poses"] * (n * bpp + 32) + n * 12
            flops += c["poses"] * passes * n * 45.0
            continue
        levels = c["levels"] or max(2, int(math.log2(side)) - 2)
        step = 1.0 / (side * math.sqrt(0.5))
        angles = max(1.0, math.radians(2 * c["range_deg"]) / step)
        coarse = max(1.0, angles / 2 ** max(0, levels - 2))
        if c["kind"] == "teach":
            nbytes += angles * n * 12 * 4 / 3
            flops += angles * n * 20 * 4 / 3
        cells = px / 4 ** (levels - 1)
        flops += c["images"] * (2.0 * cells * coarse * n / 4 ** (levels - 1) + 4.0 * px / 3)
        nbytes += n * bpp
    if c["kind"] not in ("gradient", "similarity"):
        nbytes += c["images"] * (px * bpp + (px if c["domain"] else 0))
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ exact
def _moments(img, tmpl, pose):
    """Sums of the bilinear samples q, their derivatives in (row, column, angle, scale) and the template, batched over
    poses (n, 4); float64."""
    t = tmpl.shape[0]
    o = (t - 1) / 2.0
    w = tmpl - tmpl.mean()
    w = (w / w.square().sum().sqrt()).reshape(-1)
    a = torch.arange(t, device=img.device, dtype=torch.float64) - o
    dr, dc = a[:, None].expand(t, t).reshape(-1), a[None, :].expand(t, t).reshape(-1)
    ca, sa = torch.cos(pose[:, 2:3]), torch.sin(pose[:, 2:3])
    u, v, sc = ca * dr - sa * dc, sa * dr + ca * dc, pose[:, 3:4]
    y, x = pose[:, 0:1] + sc * u, pose[:, 1:2] + sc * v
    h, wd = img.shape
    out = ((y < 0) | (x < 0) | (y > h - 1) | (x > wd - 1)).any(1)
    y, x = y.clamp(0, h - 1), x.clamp(0, wd - 1)
    r, q = y.floor().long(), x.floor().long()
    fy, fx = y - r, x - q
    r1, q1 = (r + 1).clamp(max=h - 1), (q + 1).clamp(max=wd - 1)
    va, vb, vd, ve = img[r, q], img[r, q1], img[r1, q], img[r1, q1]
    s = (1 - fy) * ((1 - fx) * va + fx * vb) + fy * ((1 - fx) * vd + fx * ve)
    gy, gx = (1 - fx) * (vd - va) + fx * (ve - vb), (1 - fy) * (vb - va) + fy * (ve - vd)
    g = torch.stack([gy, gx, sc * (gx * u - gy * v), gy * u + gx * v], 2)
    s = s - s.mean(1, keepdim=True)
    g = g - g.mean(1, keepdim=True)
    energy = s.square().sum(1)
    dot = (w * s).sum(1)
    gq = (g * s[:, :, None]).sum(1)
    gw = (g * w[None, :, None]).sum(1)
    gg = g.transpose(1, 2) @ g
    score = torch.where(out | (energy <= 0), torch.full_like(dot, -math.inf), dot / energy.sqrt())
    return score, dot, energy, gq, gw, gg


def _chunks(img, tmpl, pose):
    n = max(1, int(4e6) // tmpl.numel())
    parts = [_moments(img, tmpl, pose[i:i + n]) for i in range(0, len(pose), n)]
    return [torch.cat([p[k] for p in parts]) for k in range(6)]


def _optimum(img, tmpl, pose, axes, lo, hi):
    """Poses of the NCC maximum near `pose`, by Gauss-Newton with halved steps, in float64."""
    for _ in range(40):
        score, dot, energy, gq, gw, gg = _chunks(img, tmpl, pose)
        e = energy[:, None, None]
        m = (gg - gq[:, :, None] * gq[:, None, :] / e) / e
        b = gw / energy.sqrt()[:, None] - (score / energy)[:, None] * gq
        d = torch.zeros_like(pose)
        live = torch.isfinite(score)
        if not live.any():
            break
        d[live, :axes] = torch.linalg.solve(m[live][:, :axes, :axes], b[live][:, :axes])
        limit = torch.tensor([0.75, 0.75, 0.01, 0.01], device=pose.device, dtype=torch.float64)
        d = d * (limit / d.abs().clamp(min=1e-30)).amin(1, keepdim=True).clamp(max=1)
        moved = torch.zeros_like(live)
        for k in range(12):
            trial = pose + d * 0.5 ** k
            trial[:, 2] = trial[:, 2].clamp(lo, hi)
            better = (_chunks(img, tmpl, trial)[0] > score) & ~moved
            pose = torch.where(better[:, None], trial, pose)
            moved |= better
        if not moved.any():
            break
    return pose, _chunks(img, tmpl, pose)[0]


def _edge(pose):
    """The operators' edge-centred row and column."""
    c, s = torch.cos(pose[:, 2]), torch.sin(pose[:, 2])
    return pose[:, 0] + .5 * (1 - c + s), pose[:, 1] + .5 * (1 - c - s)


def exact(case, seed):
    c = _full(case)
    dev = _device()
    templates = [t.double() for t in _templates(c, seed)]
    a0, ext = _range(c)
    if c["kind"] in ("gradient", "similarity"):
        img, poses, rng = _frame(c, seed, 0, [t.float() for t in templates])
        img = img.double()
        p = torch.tensor(_starts(c, poses, rng), device=dev)
        if c["kind"] == "similarity":
            pose, score = _optimum(img, templates[0], p, 4, -math.inf, math.inf)
            return pose.cpu().numpy(), score.cpu().numpy()
        score, dot, energy, gq, gw, _ = _chunks(img, templates[0], p)
        grad = gw / energy.sqrt()[:, None] - (dot / energy ** 1.5)[:, None] * gq
        return score.cpu().numpy(), grad.cpu().numpy()
    if not c["subpixel"] or c["lowest"] > 1:
        return None
    rows = []
    counts = []
    for i in range(c["images"]):
        img, poses, _ = _frame(c, seed, i, [t.float() for t in templates])
        img = img.double()
        found = []
        for k, t in enumerate(templates):
            mine = [p[1:] for p in poses if p[0] == k]
            if not mine:
                continue
            p = torch.tensor(mine, device=dev, dtype=torch.float64)
            p, score = _optimum(img, t, p, 3 if ext > 0 else 2, a0, a0 + ext)
            r, q = _edge(p)
            found += [(float(s), float(a), float(b), float(z), k)
                      for s, a, b, z in zip(score, r, q, p[:, 2]) if s >= c["min_score"]]
        found.sort(key=lambda f: -f[0])
        counts.append(len(found))
        rows += found
    score, row, col, angle = (np.array([f[k] for f in rows]) for k in range(4))
    out = [row, col, angle, score]
    if c["kind"] == "teach":
        return out + [None]
    if c["kind"] == "batch":
        return out + [None, None]
    return out if c["kind"] == "find" else out + [None]
