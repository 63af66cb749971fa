"""Performance cases: the graph cuts a program asks this library for, through jfcut.py.

  image    a segmentation: build the graph from an image (or video, or volume) and seed strokes,
           solve, read the labels.  host=True: numpy in, numpy out (an application that opens a
           file); host=False: image, seeds and labels stay on the GPU (a pipeline stage).
  graph    an explicit graph (what .ef/.c1/.c2 and .mfi files hold) set from device arrays, solved,
           its labels read and their energy computed as the certificate of the flow.
  noalloc  one frame of a real-time loop: the solve that allocates nothing.
  edit     an interactive session: brush strokes on a solved image, re-solved warm, then taken back
           and re-solved warm again (so that a pass leaves the session as it found it).
  batch    an image set: build every image's graph, solve them together, read all labels.
  serve    the request loop: several host images submitted to a server, each edited once after its
           first result, labels read, sessions closed.

Every output is exact by definition (int64 max-flow and the canonical minimum cut, which is unique),
so any correct solver returns the same whole numbers.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("jf-cut_b200"))
import jfcut  # noqa: E402

MODEL = dict(lambda_n=100, z_weight_pct=100, lambda_t=10, k_fg=5, k_bg=5, seed_cap=1000000, kmeans_iters=32)
VIDEO_MODEL = dict(MODEL, z_weight_pct=50)       # temporal links at half the spatial weight
GRAY_MODEL = dict(MODEL, k_fg=2, k_bg=2)
PIXFMT = {"gray": jfcut.PIX_GRAY8, "rgb": jfcut.PIX_RGB8, "i16": jfcut.PIX_I16}
PIXBYTES = {"gray": 1, "rgb": 3, "i16": 2}
DEV = "cuda"


def listed():
    return [
        # a small photograph opened in an editor: call latency, launches and host work count
        dict(name="image_gray_640x480_host", kind="image", pix="gray", w=640, h=480, d=1, host=True),
        # a camera frame of a loop that may not allocate (the reference's images are 600 x 450)
        dict(name="noalloc_600x450", kind="noalloc", w=600, h=450),
        # a graph file of odd size: solve and certify
        dict(name="graph_1023x767", kind="graph", w=1023, h=767, d=1),
        # a full-HD photograph, host to host
        dict(name="image_rgb_1920x1080_host", kind="image", pix="rgb", w=1920, h=1080, d=1, host=True),
        # a scanned page: one channel, both sides odd
        dict(name="image_gray_2999x2011", kind="image", pix="gray", w=2999, h=2011, d=1, host=False),
        # a 12-megapixel photograph, a stage of a GPU pipeline
        dict(name="image_rgb_4096x3072", kind="image", pix="rgb", w=4096, h=3072, d=1, host=False),
        # the largest 2D image (aerial or microscopy mosaics): the headline workload
        dict(name="image_rgb_15000x10000", kind="image", pix="rgb", w=15000, h=10000, d=1, host=False),
        # a CT volume whose sides fit no tile
        dict(name="volume_i16_317x301x181", kind="image", pix="i16", w=317, h=301, d=181, host=False),
        # the largest 3D grid: a 50-frame video
        dict(name="video_rgb_2560x1440x50", kind="image", pix="rgb", w=2560, h=1440, d=50, host=False),
        # correcting strokes in an editing session, and their undo
        dict(name="edit_rgb_4096x4096", kind="edit", pix="rgb", w=4096, h=4096, d=1),
        # an image set of uneven sizes solved together
        dict(name="batch_64_to_1024", kind="batch", count=64, lo=128, hi=1024),
        # a service with a few clients at once, images and volumes
        dict(name="serve_10_to_1024", kind="serve", count=10, lo=256, hi=1024),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def sides(nodes, most=15000):
        a = math.exp(rng.uniform(-0.5, 0.5))
        return max(64, min(most, int(math.sqrt(nodes * a)))), max(64, min(most, int(math.sqrt(nodes / a))))

    kind = rng.choice(["image", "image", "image", "image3", "image3", "graph", "noalloc", "edit", "batch", "serve"])
    if kind == "image":
        host = rng.random() < 0.4
        w, h = sides(log(2e5, 4e6 if host else 1.2e8))
        return dict(kind="image", pix=rng.choice(["gray", "rgb"]), w=w, h=h, d=1, host=host)
    if kind == "image3":
        if rng.random() < 0.5:
            n = log(96 ** 3, 320 ** 3)
            w, h, d = (max(48, int(n ** (1 / 3) * math.exp(rng.uniform(-0.3, 0.3)))) for _ in range(3))
            return dict(kind="image", pix="i16", w=w, h=h, d=d, host=False)
        w = log(320, 1600)
        return dict(kind="image", pix="rgb", w=w, h=int(w * rng.uniform(0.5, 0.8)), d=log(6, 48), host=False)
    if kind == "graph":
        if rng.random() < 0.3:
            return dict(kind="graph", w=log(40, 200), h=log(40, 200), d=log(20, 100))
        w, h = sides(log(1e4, 8e6))
        return dict(kind="graph", w=w, h=h, d=1)
    if kind == "noalloc":
        w = log(96, 1000)
        return dict(kind="noalloc", w=w, h=min(max(64, int(w * rng.uniform(0.5, 1.2))), 480))
    if kind == "edit":
        w, h = sides(log(2.5e5, 1.6e7), 4096)
        return dict(kind="edit", pix="rgb", w=w, h=h, d=1)
    lo = log(100, 256)
    if kind == "batch":
        return dict(kind="batch", count=log(8, 96), lo=lo, hi=log(300, 1024))
    return dict(kind="serve", count=log(3, 12), lo=lo, hi=log(300, 1024))


# ---------------------------------------------------------------- inputs, made on the GPU from the seed
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _noisy(base, sigma, gen):
    """uint8 image: base (float, any shape) plus N(0, sigma) noise."""
    return (base + sigma * torch.randn(base.shape, generator=gen, device=DEV)).round_().clamp_(0, 255).to(torch.uint8)


def _strokes(region_fg, share, gen):
    """Seed bytes of straight strokes of 16-128 pixels that stay inside foreground or background."""
    h, w = region_fg.shape
    count = max(8, int(h * w * share / 60))
    length = 128
    dirs = torch.tensor([[1, 0], [-1, 0], [0, 1], [0, -1], [1, 1], [-1, -1], [1, -1], [-1, 1]], device=DEV)
    x = torch.randint(0, w, (count, 1), generator=gen, device=DEV)
    y = torch.randint(0, h, (count, 1), generator=gen, device=DEV)
    d = dirs[torch.randint(0, 8, (count,), generator=gen, device=DEV)]
    n = torch.randint(16, length + 1, (count, 1), generator=gen, device=DEV)
    s = torch.arange(length, device=DEV)[None]
    px, py = x + d[:, :1] * s, y + d[:, 1:] * s
    ok = (px >= 0) & (px < w) & (py >= 0) & (py < h) & (s < n)
    fg = region_fg[py.clamp(0, h - 1), px.clamp(0, w - 1)]
    ok = (ok & (fg == fg[:, :1])).long().cumprod(1).bool()
    seeds = torch.zeros(h * w, dtype=torch.uint8, device=DEV)
    seeds[(py * w + px)[ok]] = torch.where(fg, 1, 2).to(torch.uint8)[ok]
    for value, where in ((1, region_fg), (2, ~region_fg)):   # both classes have a seed, however small the image
        at = int(where.reshape(-1).to(torch.uint8).argmax())
        if not bool((seeds == value).any()):
            seeds[at] = value
    return seeds.view(h, w)


def _ellipses(w, h, channels, seed):
    """Twenty random overlapping ellipses with colours of their own, noise, strokes over 0.5% of the pixels."""
    r, gen = random.Random(seed), _gen(seed)
    side = min(w, h)
    colour = [[r.randint(0, 255) for _ in range(channels)] for _ in range(21)]
    base = torch.empty(h, w, dtype=torch.uint8, device=DEV).fill_(20)
    xs = torch.arange(w, device=DEV, dtype=torch.float32)[None]
    ys = torch.arange(h, device=DEV, dtype=torch.float32)[:, None]
    for i in range(20):
        cx, cy = r.uniform(0, w), r.uniform(0, h)
        a, b = (r.uniform(max(2, side / 20), max(3, side / 4)) for _ in range(2))
        t = r.uniform(0, math.pi)
        m = max(a, b) + 1
        x0, x1, y0, y1 = int(max(0, cx - m)), int(min(w, cx + m)), int(max(0, cy - m)), int(min(h, cy + m))
        if i == 0:
            x0, x1, y0, y1, cx, cy = 0, w, 0, h, w / 2, h / 2    # one object is always in view
        dx, dy = xs[:, x0:x1] - cx, ys[y0:y1] - cy
        u, v = dx * math.cos(t) + dy * math.sin(t), dy * math.cos(t) - dx * math.sin(t)
        base[y0:y1, x0:x1][(u / a) ** 2 + (v / b) ** 2 <= 1] = i
    img = torch.empty(h, w, channels, dtype=torch.uint8, device=DEV)
    rows = max(1, (1 << 24) // w)
    table = torch.tensor(colour, dtype=torch.float32, device=DEV)
    for y in range(0, h, rows):
        img[y:y + rows] = _noisy(table[base[y:y + rows].long()], 15, gen)
    return img, _strokes((base < 20) & (base % 2 == 0), 0.005, gen)


def _blurred_ellipse(w, h, seed):
    """One channel: a soft bright ellipse on a darker ground, strong noise, a stroke inside and one outside."""
    r, gen = random.Random(seed), _gen(seed)
    cx, cy, a, b = w * r.uniform(0.45, 0.55), h * r.uniform(0.45, 0.55), w * r.uniform(0.2, 0.3), h * r.uniform(0.15, 0.25)
    dx = torch.arange(w, device=DEV, dtype=torch.float32)[None] - cx
    dy = torch.arange(h, device=DEV, dtype=torch.float32)[:, None] - cy
    edge = (1 - ((dx / a) ** 2 + (dy / b) ** 2).sqrt()) * min(a, b) / 2.5
    img = _noisy(80 + 90 * torch.sigmoid(edge * 1.7), 20, gen)
    seeds = torch.zeros(h, w, dtype=torch.uint8, device=DEV)
    seeds[int(cy), int(cx - a / 2):int(cx + a / 2)] = 1
    seeds[h // 12, w // 4:3 * w // 4] = 2
    return img[..., None].contiguous(), seeds


def _video(w, h, d, seed):
    """An ellipse moving 4 pixels a frame over smooth texture; strokes on the first and last frames only."""
    r, gen = random.Random(seed), _gen(seed)
    low = torch.randint(0, 256, (1, 3, h // 32 + 2, w // 32 + 2), generator=gen, device=DEV).float()
    ground = torch.nn.functional.interpolate(low, size=(h, w), mode="bilinear", align_corners=True)[0].permute(1, 2, 0)
    obj = torch.tensor([r.randint(0, 255) for _ in range(3)], dtype=torch.float32, device=DEV)
    a, b, cy = w / 8, h / 6, h * r.uniform(0.4, 0.6)
    img = torch.empty(d, h, w, 3, dtype=torch.uint8, device=DEV)
    seeds = torch.zeros(d, h, w, dtype=torch.uint8, device=DEV)
    xs = torch.arange(w, device=DEV, dtype=torch.float32)[None]
    ys = torch.arange(h, device=DEV, dtype=torch.float32)[:, None]
    for z in range(d):
        cx = w / 4 + 4 * z
        inside = ((xs - cx) / a) ** 2 + ((ys - cy) / b) ** 2 <= 1
        img[z] = _noisy(torch.where(inside[..., None], obj, ground), 10, gen)
        if z in (0, d - 1):
            seeds[z, int(cy), int(cx - a / 2):int(cx + a / 2)] = 1
            seeds[z, h // 12, w // 8:7 * w // 8] = 2
            seeds[z, h - 1 - h // 12, w // 8:7 * w // 8] = 2
    return img, seeds


def _phantom(w, h, d, seed):
    """A CT-like volume: a sphere and a tube beside it, noise; seed cubes in the sphere and in a corner."""
    r, gen = random.Random(seed), _gen(seed)
    x = torch.arange(w, device=DEV, dtype=torch.float32)[None, None]
    y = torch.arange(h, device=DEV, dtype=torch.float32)[None, :, None]
    z = torch.arange(d, device=DEV, dtype=torch.float32)[:, None, None]
    cx, cy, cz = w * r.uniform(0.42, 0.52), h * r.uniform(0.45, 0.55), d * r.uniform(0.45, 0.55)
    rad = min(w, h, d) / 4
    tr = max(2.0, rad / 3)
    v = 10 * torch.randn(d, h, w, generator=gen, device=DEV)
    v += 600 * ((x - (cx + rad + tr + 2)) ** 2 + (y - cy) ** 2 <= tr * tr) + 0 * z
    v[(x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2 <= rad * rad] += 1000
    seeds = torch.zeros(d, h, w, dtype=torch.uint8, device=DEV)
    s = max(1, int(rad / 4))
    seeds[int(cz) - s:int(cz) + s + 1, int(cy) - s:int(cy) + s + 1, int(cx) - s:int(cx) + s + 1] = 1
    seeds[1:2 + s, 1:2 + s, 1:2 + s] = 2
    return v.round_().clamp_(-32768, 32767).to(torch.int16), seeds


def _image(pix, w, h, d, seed):
    """(image, seeds, model) of a case."""
    if pix == "i16":
        return _phantom(w, h, d, seed) + (MODEL,)
    if d > 1:
        return _video(w, h, d, seed) + (VIDEO_MODEL,)
    if pix == "gray":
        return _blurred_ellipse(w, h, seed) + (GRAY_MODEL,)
    return _ellipses(w, h, 3, seed) + (MODEL,)


def _explicit(w, h, d, seed):
    """(excess, capacities) as another program would write them: contrast n-links and intensity t-links of a noisy image."""
    gen = _gen(seed)
    if d > 1:
        v = _phantom(max(w, 48), max(h, 48), max(d, 48), seed)[0][:d, :h, :w].float() / 8
    else:
        v = _blurred_ellipse(w, h, seed)[0][..., 0].float()
    n = v.dim()
    caps = {}
    for axis in range(n):
        diff = v.diff(dim=axis)
        weight = (100 * torch.exp(-diff ** 2 / (2 * (diff ** 2).mean() + 1e-3))).round().to(torch.int32)
        pad = [0, 0] * n
        pad[2 * (n - 1 - axis) + 1] = 1
        caps[axis, 1] = torch.nn.functional.pad(weight, pad).contiguous()     # towards +, 0 on the far side
        pad[2 * (n - 1 - axis):2 * (n - 1 - axis) + 2] = [1, 0]
        caps[axis, -1] = torch.nn.functional.pad(weight, pad).contiguous()
    lo, hi = v.mean() - v.std(), v.mean() + v.std()
    e = ((v - lo) ** 2 - (hi - v) ** 2) / (8 * v.var() + 1e-3) * 10
    e = (e + 4 * torch.randn(v.shape, generator=gen, device=DEV)).round().to(torch.int32).contiguous()
    order = [(1, 1), (0, 1), (0, -1), (1, -1)] if n == 2 else [(2, 1), (1, 1), (0, 1), (0, -1), (1, -1), (2, -1)]
    return e, [caps[k] for k in order]


def _stroke(w, h, share, seed):
    """A hand-drawn stroke: distinct node indices along a wandering brush a few pixels wide."""
    r = np.random.default_rng(seed)
    radius = 3
    steps = max(8, int(w * h * share / (2 * radius + 1)))
    turn = r.normal(0, 0.08, steps).cumsum() + r.uniform(0, 2 * math.pi)
    x = np.abs(r.uniform(0, w) + np.cos(turn).cumsum()) % (2 * w)
    y = np.abs(r.uniform(0, h) + np.sin(turn).cumsum()) % (2 * h)
    x, y = np.minimum(x, 2 * w - 1 - x).clip(0, w - 1), np.minimum(y, 2 * h - 1 - y).clip(0, h - 1)
    off = np.arange(-radius, radius + 1)
    px = np.clip(x[:, None].astype(np.int64) + off, 0, w - 1)
    idx = np.unique(y[:, None].astype(np.int64) * w + px)
    return r.permutation(idx).astype(np.uint32)


def _edit(w, h, share, seed, labels=None, count=6):
    """An edit list of several strokes over distinct nodes: corrections (each stroke the other class than the label where
    it starts) when the labels are known, else object and background in turn."""
    strokes = [_stroke(w, h, share / count, count * seed + k) for k in range(count)]
    marks = [1 + k % 2 if labels is None else (2 if labels[s[0]] else 1) for k, s in enumerate(strokes)]
    idx, first = np.unique(np.concatenate(strokes), return_index=True)
    brush = np.concatenate([np.full(s.size, m, np.uint8) for s, m in zip(strokes, marks)])[first]
    order = np.random.default_rng(seed).permutation(idx.size)
    return idx[order], brush[order]


def _sizes(case, seed):
    r = random.Random(case["count"] * 1000003 + case["lo"] * 1009 + case["hi"])   # sizes belong to the case, contents to the seed
    return [(r.randint(case["lo"], case["hi"]), r.randint(case["lo"], case["hi"]), seed * 131 + i) for i in range(case["count"])]


def _volume(w, h):
    return max(48, w // 4), max(48, h // 4), max(48, h // 10)


def _shape(w, h, d):
    return (h, w) if d == 1 else (d, h, w)


# ---------------------------------------------------------------- the protocol
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case, ctx=jfcut.Context(0))
    if kind in ("image", "edit"):
        w, h, d = case["w"], case["h"], case["d"]
        img, seeds, model = _image(case["pix"], w, h, d, seed)
        s.update(img=img, seeds=seeds, model=jfcut.default_model(**model), g=jfcut.Graph(s["ctx"], _shape(w, h, d)),
                 labels=torch.empty(_shape(w, h, d), dtype=torch.uint8, device=DEV))
        if case.get("host"):
            s.update(img=img.cpu().numpy(), seeds=seeds.cpu().numpy())
        if kind == "edit":
            torch.cuda.synchronize()
            s["g"].build_from_device(img.data_ptr(), seeds.data_ptr(), PIXFMT[case["pix"]], s["model"])
            s["g"].solve()
            labels, seeds = s["g"].labels().reshape(-1), seeds.view(-1).cpu().numpy()
            # other strokes on every pass: the flow of an earlier one is still in the graph where it went
            edits = [_edit(w, h, 0.002, 64 * seed + k, labels) for k in range(48)]
            s.update(edits=[(idx, brush, seeds[idx]) for idx, brush in edits], at=0, undone=torch.empty_like(s["labels"]))
    elif kind in ("graph", "noalloc"):
        w, h, d = case["w"], case["h"], case.get("d", 1)
        e, caps = _explicit(w, h, d, seed)
        s.update(e=e, caps=caps, labels=torch.empty(_shape(w, h, d), dtype=torch.uint8, device=DEV))
        if kind == "graph":
            s["g"] = jfcut.Graph(s["ctx"], _shape(w, h, d))
    elif kind == "batch":
        s["items"], s["batch"] = [], jfcut.Batch(s["ctx"])
        sizes = _sizes(case, seed)
        s["labels"] = torch.empty(sum(w * h for w, h, _ in sizes), dtype=torch.uint8, device=DEV)
        s["model"] = jfcut.default_model(**MODEL)
        at = 0
        for w, h, sd in sizes:
            img, seeds, _ = _image("rgb", w, h, 1, sd)
            s["items"].append((jfcut.Graph(s["ctx"], (h, w)), img, seeds, at))
            at += w * h
        torch.cuda.synchronize()
        for g, img, seeds, _ in s["items"]:      # a batch takes built graphs
            g.build_from_device(img.data_ptr(), seeds.data_ptr(), jfcut.PIX_RGB8, s["model"])
            s["batch"].add(g)
    else:
        s["server"] = jfcut.Server(s["ctx"], 8 << 30)
        s["model"] = jfcut.default_model(**MODEL)
        s["items"] = []
        for i, (w, h, sd) in enumerate(_sizes(case, seed)):
            if i % 10 < 7:
                img, seeds, _ = _image("rgb", w, h, 1, sd)
                idx, brush = _edit(w, h, 0.01, sd)
            else:                                # three in ten are volumes
                img, seeds, _ = _image("i16", *_volume(w, h), sd)
                idx, brush = _edit(img.shape[2], img.shape[1] * img.shape[0], 0.01, sd)
            s["items"].append((img.cpu().numpy(), seeds.cpu().numpy(), jfcut.PIX_RGB8 if i % 10 < 7 else jfcut.PIX_I16,
                               idx, brush))
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "image":
        g = s["g"]
        if s["host"]:
            g.build_from_image(s["img"], s["seeds"], PIXFMT[s["pix"]], s["model"])
            g.solve()
            return [g.flow(), g.labels()]
        g.build_from_device(s["img"].data_ptr(), s["seeds"].data_ptr(), PIXFMT[s["pix"]], s["model"])
        g.solve()
        g.read_labels_device(s["labels"].data_ptr())
        return [g.flow(), s["labels"]]
    if kind == "graph":
        g, caps = s["g"], [c.data_ptr() for c in s["caps"]]
        g.set_device(s["e"].data_ptr(), caps)
        g.solve()
        g.read_labels_device(s["labels"].data_ptr())
        data, smooth = jfcut.energy_device(0, g.shape, s["e"].data_ptr(), caps, s["labels"].data_ptr())
        return [g.flow(), s["labels"], data, smooth]
    if kind == "noalloc":
        flow = jfcut.solve_grid2d_noalloc(s["w"], s["h"], s["e"].data_ptr(), [c.data_ptr() for c in s["caps"]],
                                          s["labels"].data_ptr())
        return [flow, s["labels"]]
    if kind == "edit":
        g, out = s["g"], []
        idx, brush, undo = s["edits"][s["at"] % len(s["edits"])]
        s["at"] += 1
        for mark, labels in ((brush, s["labels"]), (undo, s["undone"])):
            g.edit_seeds(idx, mark)
            g.solve()
            g.read_labels_device(labels.data_ptr())
            out += [g.flow(), labels]
        return out
    if kind == "batch":
        for g, img, seeds, _ in s["items"]:
            g.build_from_device(img.data_ptr(), seeds.data_ptr(), jfcut.PIX_RGB8, s["model"])
        s["batch"].solve()
        for g, _, _, at in s["items"]:
            g.read_labels_device(s["labels"].data_ptr() + at)
        return [np.array([g.flow() for g, _, _, _ in s["items"]], np.int64), s["labels"]]
    server, flows, labels = s["server"], [], []
    sids = [server.submit(img, seeds, pf, s["model"]) for img, seeds, pf, _, _ in s["items"]]
    for sid, (_, _, _, idx, brush) in zip(sids, s["items"]):
        flows.append(server.wait(sid).flow)
        server.edit(sid, idx, brush)
    for sid, (_, seeds, _, _, _) in zip(sids, s["items"]):
        flows.append(server.wait(sid).flow)
        labels.append(server.labels(sid, seeds.shape).reshape(-1))
        server.close_session(sid)
    return [np.array(flows, np.int64), np.concatenate(labels)]


def exact(case, seed):
    """No floating outputs: flows and labels are whole numbers, unique for the inputs."""
    return None


def work(case):
    """Inputs read once and labels written once; integer work only."""
    kind = case["kind"]
    if kind == "image":
        return dict(bytes=case["w"] * case["h"] * case["d"] * (PIXBYTES[case["pix"]] + 2), flops=0)
    if kind == "graph":      # the capacities are read again by the certificate, with the labels
        n = case["w"] * case["h"] * case["d"]
        return dict(bytes=n * (2 * 4 * (5 if case["d"] == 1 else 7) + 2), flops=0)
    if kind == "noalloc":
        return dict(bytes=case["w"] * case["h"] * (4 * 5 + 1), flops=0)
    if kind == "edit":       # two solved states, a label plane each, and the stroke's nodes twice
        n = case["w"] * case["h"]
        return dict(bytes=int(2 * n + 2 * 5 * 0.002 * n), flops=0)
    sizes = _sizes(case, 0)
    if kind == "batch":
        return dict(bytes=sum(w * h for w, h, _ in sizes) * (3 + 2), flops=0)
    return dict(bytes=sum(w * h * (3 + 2) if i % 10 < 7 else math.prod(_volume(w, h)) * (2 + 2)
                          for i, (w, h, _) in enumerate(sizes)), flops=0)
