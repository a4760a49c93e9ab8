"""The work a user of patchtable_b200 has it do, as a fixed list of cases and a generator of more.

Every case goes through the public Python entry points: a table is built of image b, image a is
matched against it, and the nearest-neighbour field (x, y, distance per 8x8 patch, float64) comes
back.  Kinds:

  query   PatchTable.lookup_device: one image already on the GPU against a table the program keeps
  host    PatchTable.lookup with page-locked host buffers, copies included
  video   PatchTable.lookup seeded with the previous frame's field (ann_prev)
  batch   QueryBatch.lookup: several images of uneven sizes in one call
  match   PatchTable(params, b) and one lookup: two images matched from scratch
  atlas   lookup_device against several images packed into one table under an allowed mask
  desc    descriptor mode: lookup_device of caller-supplied descriptor images

Images are value noise with rectangles and a smoothly warped, slightly noisy second view of them
(the generator of patchtable_b200.synth, restated for the GPU so that inputs are made quickly).
"""
import ctypes
import math
import random

import numpy as np
import torch
import torch.nn.functional as F

import patchtable_b200 as ptb

MATCHED = "1/2/1/-1"      # one pass, first jump 2, one pull candidate, no k-coherence: the field is
                          # still better than the reference's, and the fastest schedule that is
DEFAULT = "default"       # the library's schedule: 4 passes, all candidates, k-coherence


def listed():
    return [
        # the smallest call: a thumbnail, the size the tests use; launches and host work are all of it
        dict(name="query_tiny", kind="query", h=48, w=64, bh=48, bw=64, speed=3, schedule=DEFAULT),
        # an odd-sized crop against a 720p-class image, library defaults
        dict(name="query_ragged", kind="query", h=355, w=611, bh=719, bw=1277, speed=3, schedule=DEFAULT),
        # the quality preset (k-coherence 10 on the first sweep, spatial and random search) at 540p
        dict(name="query_540p_speed1", kind="query", h=540, w=960, bh=540, bw=960, speed=1, schedule=DEFAULT),
        # the benchmark's workload: 1080p at the reference's quality, data already on the GPU
        dict(name="query_1080p_matched", kind="query", h=1080, w=1920, bh=1080, bw=1920, speed=3, schedule=MATCHED),
        # the same image pair with the library's defaults: the best field
        dict(name="query_1080p_default", kind="query", h=1080, w=1920, bh=1080, bw=1920, speed=3, schedule=DEFAULT),
        # the same match from and to host memory, as a program without GPU buffers calls it
        dict(name="host_1080p_matched", kind="host", h=1080, w=1920, bh=1080, bw=1920, speed=3, schedule=MATCHED),
        # a frame of a 720p video, seeded with the previous frame's field
        dict(name="video_720p", kind="video", h=720, w=1280, bh=720, bw=1280, speed=3, schedule=DEFAULT),
        # a batch of uneven images (photo collection) against one 1080p table
        dict(name="batch_uneven", kind="batch", n=16, lo=128, hi=1536, bh=1080, bw=1920, speed=3, schedule=MATCHED),
        # two small images matched from scratch: table build and one lookup
        dict(name="match_small", kind="match", h=240, w=320, bh=240, bw=320, speed=3, schedule=DEFAULT),
        # two 1080p images matched from scratch
        dict(name="match_1080p", kind="match", h=1080, w=1920, bh=1080, bw=1920, speed=3, schedule=DEFAULT),
        # one photo against a small collection packed into one table; seams are masked out
        dict(name="atlas_768", kind="atlas", h=768, w=1024, n=6, lo=256, hi=1024, speed=3, schedule=DEFAULT),
        # image-analogy level: descriptors supplied by the caller, 8 channels
        dict(name="desc_540p", kind="desc", h=540, w=960, bh=540, bw=960, channels=8, speed=3, schedule=DEFAULT),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "query", "host", "video", "batch", "match", "atlas", "desc"])
    c = dict(kind=kind, speed=3, schedule=rng.choice([DEFAULT, MATCHED]))
    if kind == "batch":
        lo, hi = 128, _side(rng, 256, 1536)
        return dict(c, n=rng.randint(2, 16), lo=lo, hi=hi, bh=_side(rng, 200, 1080), bw=_side(rng, 200, 1920))
    if kind == "atlas":
        return dict(c, h=_side(rng, 96, 768), w=_side(rng, 96, 1024), n=rng.randint(2, 6), lo=200, hi=_side(rng, 256, 1024))
    if kind == "desc":
        h, w = _side(rng, 48, 540), _side(rng, 64, 960)
        return dict(c, h=h, w=w, bh=h, bw=w, channels=rng.choice([6, 8, 12]))
    h, w = _side(rng, 48, 1080), _side(rng, 64, 1920)
    if kind == "query":
        c["speed"] = rng.choice([3, 3, 6, 1]) if h * w <= 540 * 960 else 3
        if c["speed"] != 3:
            c["schedule"] = DEFAULT
        return dict(c, h=h, w=w, bh=_side(rng, 48, 1080), bw=_side(rng, 64, 1920))
    if kind == "video":
        return dict(c, h=min(h, 720), w=min(w, 1280), bh=min(h, 720), bw=min(w, 1280), schedule=DEFAULT)
    return dict(c, h=h, w=w, bh=h, bw=w)


# ---- inputs -------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7fffffff)


def _image(h, w, g):
    """4 octaves of value noise and 20 rectangles, h x w x 3 in [0, 1]."""
    img = torch.zeros(1, 3, h, w, device="cuda")
    amp, period = 1.0, 64
    for _ in range(4):
        lat = torch.rand(1, 3, h // period + 2, w // period + 2, generator=g, device="cuda")
        up = F.interpolate(lat, scale_factor=period, mode="bilinear", align_corners=False)
        o = period // 2
        img += amp * up[:, :, o:o + h, o:o + w]
        amp, period = amp / 2, period // 2
    img /= 1.875
    r = torch.rand(20, 4, generator=g, device="cuda").cpu().numpy()
    col = torch.rand(20, 3, generator=g, device="cuda")
    side = max(8, min(h, w) // 4)
    for k in range(20):
        x0, y0 = int(r[k, 0] * w), int(r[k, 1] * h)
        rw, rh = 8 + int(r[k, 2] * (side - 7)), 8 + int(r[k, 3] * (side - 7))
        img[0, :, y0:y0 + rh, x0:x0 + rw] = col[k][:, None, None]
    return img.clamp_(0, 1)


def _warp(img, g, most=16.0):
    """A view of img displaced by a smooth flow of at most `most` pixels, with N(0, 0.02) noise."""
    h, w = img.shape[2:]
    lat = torch.randn(1, 2, h // 32 + 4, w // 32 + 4, generator=g, device="cuda")
    flow = F.interpolate(lat, size=(h, w), mode="bicubic", align_corners=True)
    flow *= most / flow.square().sum(1).sqrt().max()
    ys, xs = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    gx = 2 * (xs + flow[0, 0]) / max(1, w - 1) - 1
    gy = 2 * (ys + flow[0, 1]) / max(1, h - 1) - 1
    out = F.grid_sample(img, torch.stack([gx, gy], -1)[None], mode="bilinear", padding_mode="border", align_corners=True)
    return (out + 0.02 * torch.randn(out.shape, generator=g, device="cuda")).clamp_(0, 1)


def _hwc(img):
    return img[0].permute(1, 2, 0).contiguous()


def _crop(img, h, w, r):
    H, W = img.shape[2:]
    y, x = int(r[0] * (H - h + 1)), int(r[1] * (W - w + 1))
    return img[:, :, y:y + h, x:x + w]


def _pair(c, g):
    """Query and table image: views of one scene, each cropped to its size."""
    H, W = max(c["h"], c["bh"]), max(c["w"], c["bw"])
    scene = _image(H, W, g)
    other = _warp(scene, g)
    r = torch.rand(4, generator=g, device="cuda").cpu().numpy()
    return _hwc(_crop(scene, c["h"], c["w"], r[:2])), _hwc(_crop(other, c["bh"], c["bw"], r[2:]))


def _sizes(c):
    """The (h, w) of a case's images, sides uniform in [lo, hi]: the case's own, whatever the seed."""
    r = random.Random("%d %d %d" % (c["n"], c["lo"], c["hi"]))
    return [(r.randint(c["lo"], c["hi"]), r.randint(c["lo"], c["hi"])) for _ in range(c["n"])]


def _params(c, extra=""):
    p = ptb.PatchTableParams("-speed %d -coherence_spatial 4%s" % (c["speed"], extra))
    if c["schedule"] != DEFAULT:
        p.set_schedule([int(v) for v in c["schedule"].split("/")])
    return p


def _table(p, b, seed, allowed=None):
    ctypes.CDLL(None).srand(int(seed) & 0x7fffffff)      # the populate order is drawn from rand()
    return ptb.PatchTable(p, b.cpu().numpy(), allowed_patches=allowed)


def _field(h, w):
    return torch.empty((h - 7, w - 7, 3), dtype=torch.float64, device="cuda")


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def prepare(c, seed):
    g = _gen(seed)
    kind = c["kind"]
    s = dict(kind=kind, case=c, seed=seed)
    if kind == "batch":
        scene = _image(max(c["hi"], c["bh"]), max(c["hi"], c["bw"]), g)
        other = _warp(scene, g)
        r = torch.rand(c["n"] + 1, 4, generator=g, device="cuda").cpu().numpy()
        s["table"] = _table(_params(c), _hwc(_crop(other, c["bh"], c["bw"], r[-1])), seed)
        sizes = _sizes(c)
        s["batch"] = s["table"].batch(sizes)
        s["a"] = torch.cat([_hwc(_crop(scene, h, w, r[i])).reshape(-1) for i, (h, w) in enumerate(sizes)])
        s["ann"] = torch.empty((s["batch"].patches, 3), dtype=torch.float64, device="cuda")
        return s
    if kind == "atlas":
        side = max(c["hi"], c["h"], c["w"])
        scene = _image(side, side, g)
        other = _warp(scene, g)
        r = torch.rand(c["n"] + 1, 4, generator=g, device="cuda").cpu().numpy()
        sizes = _sizes(c)
        cols = max(1, int(math.sqrt(c["n"])))
        cell = max(max(z) for z in sizes)
        rows = -(-c["n"] // cols)
        atlas = torch.zeros(rows * cell, cols * cell, 3, device="cuda")
        allowed = np.zeros((rows * cell - 7, cols * cell - 7), np.int32)
        for i, (h, w) in enumerate(sizes):
            y, x = (i // cols) * cell, (i % cols) * cell
            atlas[y:y + h, x:x + w] = _hwc(_crop(other, h, w, r[i]))
            allowed[y:y + h - 7, x:x + w - 7] = 1
        s["table"] = _table(_params(c), atlas, seed, allowed)
        s["a"] = _hwc(_crop(scene, c["h"], c["w"], r[-1]))
        s["ann"] = _field(c["h"], c["w"])
        return s
    a, b = _pair(c, g)
    if kind == "desc":
        k = torch.randn(c["channels"], 3, 3, 3, generator=g, device="cuda") / math.sqrt(27)

        def feat(x):
            x = F.pad(x.permute(2, 0, 1)[None], (2, 2, 2, 2), mode="replicate")
            taps = [x[:, :, dy:dy + x.shape[2] - 4, dx:dx + x.shape[3] - 4] for dy in (0, 2, 4) for dx in (0, 2, 4)]
            return sum(torch.einsum("kc,nchw->nhwk", k[:, :, i // 3, i % 3], t) for i, t in enumerate(taps))[0].contiguous()
        a, b = feat(a), feat(b)
        s["table"] = _table(_params(c, " -is_descriptor 1"), b, seed)
        s["a"] = a
        s["ann"] = torch.empty((c["h"], c["w"], 3), dtype=torch.float64, device="cuda")
        return s
    if kind == "query":
        s["table"] = _table(_params(c), b, seed)
        s["a"], s["ann"] = a, _field(c["h"], c["w"])
    elif kind == "host":
        s["table"] = _table(_params(c), b, seed)
        s["a"], s["ann"] = _pinned(a.shape, a.dtype).copy_(a), _pinned((c["h"] - 7, c["w"] - 7, 3), torch.float64)
    elif kind == "video":
        s["table"] = _table(_params(c, " -coherence_temporal 0.5"), b, seed)
        before = _hwc(_warp(a.permute(2, 0, 1)[None], g, 3.0))
        s["prev"] = s["table"].lookup(before.cpu().numpy())
        s["a"] = _pinned(a.shape, a.dtype).copy_(a)
        s["ann"] = _pinned((c["h"] - 7, c["w"] - 7, 3), torch.float64)
    else:
        s["a"], s["b"] = a.cpu().numpy(), b.cpu().numpy()
    return s


def run(s):
    c, kind = s["case"], s["kind"]
    if kind in ("query", "atlas", "desc"):
        s["table"].lookup_device(s["a"].data_ptr(), s["a"].shape[0], s["a"].shape[1], s["ann"].data_ptr(),
                                 torch.cuda.current_stream().cuda_stream)
        return s["ann"]
    if kind == "batch":
        s["batch"].lookup(s["a"].data_ptr(), s["ann"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return s["ann"]
    if kind == "host":
        return s["table"].lookup(s["a"].numpy(), out=s["ann"].numpy())
    if kind == "video":
        return s["table"].lookup(s["a"].numpy(), ann_prev=s["prev"], out=s["ann"].numpy())
    ctypes.CDLL(None).srand(int(s["seed"]) & 0x7fffffff)
    table = ptb.PatchTable(_params(c), s["b"])
    ann = table.lookup(s["a"])
    table.close()
    return ann


def exact(c, seed):
    """Every output is a field whose positions are decisions (which candidate was nearest) and whose
    distances belong to those positions, so no value stands on its own in 64 bits."""
    return None


def work(c):
    """Image a and image b read once, one table entry per patch, the field written once; the SSD of
    8x8x3 values (sub, mul, add) of every patch against one candidate per choose and per pull."""
    channels = c.get("channels", 3)
    if c["kind"] == "batch":
        pix = sum(h * w for h, w in _sizes(c))
        patches = sum((h - 7) * (w - 7) for h, w in _sizes(c))
    else:
        pix = c["h"] * c["w"]
        patches = pix if c["kind"] == "desc" else (c["h"] - 7) * (c["w"] - 7)
    if c["kind"] == "atlas":
        bpix = sum(h * w for h, w in _sizes(c))
    else:
        bpix = c["bh"] * c["bw"]
    passes = (2 if c["speed"] == 6 else 4) if c["schedule"] == DEFAULT else int(c["schedule"].split("/")[0])
    nbytes = 4 * channels * (pix + bpix) + 28 * patches
    if c["kind"] == "video":
        nbytes += 24 * patches
    if c["kind"] == "match":
        nbytes += 4e8 + 16 * bpix          # the table's cells (-limit 100) and the k-coherence set, written once
    per = 3 * channels if c["kind"] == "desc" else 3 * 192
    return {"bytes": float(nbytes), "flops": float(patches * 2 * passes * per)}
