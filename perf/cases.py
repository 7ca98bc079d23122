"""The work a user of this package has it do, as cases that can be timed.

Six forms, each through the package's public entry points:

  find    one frame from page-locked host memory to its signal list, as a
          detector worker calls it per frame (`find`)
  series  a short series the per-frame way: `find` and `Labeller.add` frame
          by frame, then the spots and their pixels
  batch   a batch of frames resident in an engine's slot: threshold, ordered
          lists and grouping in one run, and the spots it finished (a 3D
          batch is a wedge that ends with the shutter closed, so each run
          finishes its spots)
  stills  the same for panels of four shapes interleaved, grouped in 2D, with
          the spots and pixels of every series
  stream  a series through the engine's two slots, batch after batch, from
          raw frames or compressed chunks in page-locked memory to spots and
          pixels in page-locked memory, then the series' end
  decode  one compressed chunk into a frame in device memory

Frames are synthetic Eiger frames in the package's benchmark shapes: module
gaps at the masked sentinel, a Poisson background with a diffuse ring, and 3D
Gaussian reflections Poisson-sampled on top, made on the device from the seed
(counts are added as integers, so the order of the additions does not matter).
Results come in the caller's buffers, whole, with the counts of what is in
them: the buffers start as zeros, and what is past a count is not written.
"""

from __future__ import annotations

import math
import random
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import dials_metal_spotfinder_b200 as sf
from dials_metal_spotfinder_b200 import chunk, synth
from dials_metal_spotfinder_b200.engine import Engine
from dials_metal_spotfinder_b200.labeller import Labeller

DEVICE = "cuda"
MIN_SIZE, MAX_SIZE, MAX_SEPARATION = 3, 1000, 2.0  # the grouping's defaults


def listed():
    h4, w4 = synth.EIGER_4M
    h16, w16 = synth.EIGER_16M
    hs, ws = synth.SMALL
    hp, wp = synth.STILL_SHAPES[0]
    return [
        # a region of interest or a small detector: latency and launches
        {"name": "find_small_u16", "kind": "find", "height": hs, "width": ws, "bits": 16},
        # the plain form on the common detector
        {"name": "find_4m_u16", "kind": "find", "height": h4, "width": w4, "bits": 16},
        # 32-bit images (summed or high-dynamic-range data), one panel
        {"name": "find_1m_u32", "kind": "find", "height": hp, "width": wp, "bits": 32},
        # a whole small series the per-frame way, as the command line runs it
        {"name": "series_small", "kind": "series", "height": hs, "width": ws, "frames": 12,
         "bits": 16},
        # one detector frame after another into the labeller
        {"name": "series_4m", "kind": "series", "height": h4, "width": w4, "frames": 4,
         "bits": 16},
        # the headline: a resident 16M batch, threshold and 3D grouping
        {"name": "batch_16m_u16", "kind": "batch", "height": h16, "width": w16, "frames": 16,
         "bits": 16, "masked": False, "two_d": False},
        # the same at 32 bits with intensities up to 2e6
        {"name": "batch_16m_u32", "kind": "batch", "height": h16, "width": w16, "frames": 8,
         "bits": 32, "masked": False, "two_d": False},
        # a 4M series with the detector's pixel mask stamped before every run
        {"name": "batch_4m_u16_mask", "kind": "batch", "height": h4, "width": w4, "frames": 16,
         "bits": 16, "masked": True, "two_d": False},
        # serial stills of four panels at once
        {"name": "stills_uneven", "kind": "stills", "scale": 1.0, "frames": 2},
        # processing a 16M series as it was stored: bslz4 chunks to spots
        {"name": "stream_16m_bslz4", "kind": "stream", "height": h16, "width": w16, "frames": 4,
         "batches": 3, "bits": 16, "source": "bslz4", "graph": False},
        # a live 4M series, one chunk per run, replayed from graphs
        {"name": "live_4m_bslz4", "kind": "stream", "height": h4, "width": w4, "frames": 1,
         "batches": 8, "bits": 16, "source": "bslz4", "graph": True},
        # a stored LZ4 frame decoded into a caller's device buffer
        {"name": "decode_4m_lz4", "kind": "decode", "height": h4, "width": w4, "bits": 16,
         "source": "lz4"},
    ]


def draw(rng: random.Random):
    """Detector sizes from a small region of interest to 16M, odd ones among
    them, and no more pixels in a pass than the largest listed case's."""
    def shape(most):
        h = round(math.exp(rng.uniform(math.log(128), math.log(synth.EIGER_16M[0]))))
        w = round(math.exp(rng.uniform(math.log(128), math.log(synth.EIGER_16M[1]))))
        shrink = min(1.0, math.sqrt(most / (h * w)))
        return max(64, int(h * shrink)), max(64, int(w * shrink))

    kind = rng.choice(["find", "series", "batch", "batch", "stills", "stream", "stream", "decode"])
    bits = rng.choice([16, 16, 32])
    if kind == "find":
        h, w = shape(18e6)
        return {"kind": kind, "height": h, "width": w, "bits": bits}
    if kind == "series":
        h, w = shape(4.5e6)
        return {"kind": kind, "height": h, "width": w, "frames": rng.randint(2, 5), "bits": bits}
    if kind == "batch":
        two_d = rng.random() < 0.3
        frames = rng.randint(1 if two_d else 3, 16)
        h, w = shape(18e6 if bits == 16 else 18e6 * min(1.0, 8 / frames))
        return {"kind": kind, "height": h, "width": w, "frames": frames, "bits": bits,
                "masked": rng.random() < 0.3, "two_d": two_d}
    if kind == "stills":
        return {"kind": kind, "scale": round(rng.uniform(0.2, 1.0), 3),
                "frames": rng.randint(1, 2)}
    if kind == "stream":
        frames, batches = rng.randint(1, 8), rng.randint(2, 4)
        h, w = shape(100e6 / (frames * batches))
        return {"kind": kind, "height": h, "width": w, "frames": frames, "batches": batches,
                "bits": bits, "source": rng.choice(["raw", "bslz4", "bslz4", "lz4"]),
                "graph": rng.random() < 0.5}
    h, w = shape(18e6)
    return {"kind": kind, "height": h, "width": w, "bits": bits,
            "source": rng.choice(["lz4", "bslz4"])}


# -- frames -------------------------------------------------------------------

def still_shapes(case):
    return [(max(64, int(h * case["scale"])), max(64, int(w * case["scale"])))
            for h, w in synth.STILL_SHAPES]


def detector_gaps(h, w):
    rows = (torch.arange(h, device=DEVICE) % 551) >= 514
    cols = (torch.arange(w, device=DEVICE) % 1040) >= 1030
    return rows[:, None] | cols[None, :]


def make_frames(h, w, n, bits, seed, stills=False):
    """n consecutive frames as device tensors of 64-bit integers."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    y = torch.arange(h, device=DEVICE, dtype=torch.float32) + 0.5
    x = torch.arange(w, device=DEVICE, dtype=torch.float32) + 0.5
    r = torch.sqrt((y[:, None] - h / 2) ** 2 + (x[None, :] - w / 2) ** 2)
    small = h * w <= synth.SMALL[0] * synth.SMALL[1]
    if small:
        lam = torch.ones_like(r)
    else:
        lam = 0.3 + 2.0 * torch.exp(-(((r - 0.28 * min(h, w)) / 40.0) ** 2))
    gaps = None if small else detector_gaps(h, w)
    top = (1 << bits) - 1

    # reflections over the series: per frame, as the benchmark series have
    per_mpx = 500.0 if stills else 40.0 if small else 450.0 if h * w < 9e6 else 330.0
    count = max(1, round(per_mpx * h * w / 1e6 * n))
    u = torch.rand((6, count), generator=g, device=DEVICE, dtype=torch.float64)
    cx, cy = u[0] * w, u[1] * h
    cz = torch.floor(u[2] * n)
    sxy = 0.8 + 0.7 * u[3]
    sz = 0.5 + u[4]
    lo, hi = (2000.0, 2000.0) if small else (50.0, 2.0e6 if bits == 32 else 5.0e4)
    inten = lo * (hi / lo) ** u[5]
    off = torch.arange(2 * synth.BOX + 1, device=DEVICE)

    def mass(low, centre, sigma):
        s = math.sqrt(2.0) * sigma
        return 0.5 * (torch.erf((low + 1 - centre) / s) - torch.erf((low - centre) / s))

    frames = []
    for f in range(n):
        img = torch.poisson(lam, generator=g).to(torch.int64).reshape(-1)
        wz = (cz == f).double() if stills else mass(float(f), cz + 0.5, sz)
        k = torch.nonzero(wz > 1e-6).reshape(-1)
        if len(k):
            px = (torch.floor(cx[k]) - synth.BOX).long()[:, None] + off
            py = (torch.floor(cy[k]) - synth.BOX).long()[:, None] + off
            wx = mass(px.double(), cx[k, None], sxy[k, None])
            wy = mass(py.double(), cy[k, None], sxy[k, None])
            mean = (inten[k] * wz[k])[:, None, None] * wy[:, :, None] * wx[:, None, :]
            hits = torch.poisson(mean.clamp_(min=0.0).float(), generator=g).long()
            ok = ((py >= 0) & (py < h))[:, :, None] & ((px >= 0) & (px < w))[:, None, :]
            at = (py.clamp(0, h - 1)[:, :, None] * w + px.clamp(0, w - 1)[:, None, :])
            img.index_add_(0, at.reshape(-1), (hits * ok).reshape(-1))
        img = img.clamp_(max=top - 1).reshape(h, w)
        if gaps is not None:
            img[gaps] = top
        frames.append(img)
    return frames


def pixel_mask(h, w, seed):
    """Dead pixels here and there and a beam stop."""
    rng = np.random.default_rng(seed)
    mask = rng.random((h, w)) < 1e-3
    mask[h // 2 - h // 60:h // 2 + h // 60 + 1, : w // 2] = True
    return mask


def dtype_of(case):
    return np.uint16 if case.get("bits", 16) == 16 else np.uint32


def as_pixels(img, dtype):
    """The device tensor of the frame's pixels (as signed words of the size)."""
    bits = 16 if dtype == np.uint16 else 32
    wrapped = torch.where(img >= 1 << (bits - 1), img - (1 << bits), img)
    return wrapped.to(torch.int16 if bits == 16 else torch.int32).contiguous()


def page_locked(shape, dtype):
    """A page-locked array, kept alive by whoever holds a view of it."""
    nbytes = max(1, math.prod(shape)) * np.dtype(dtype).itemsize
    flat = torch.zeros(nbytes, dtype=torch.uint8, pin_memory=True).numpy().view(dtype)
    return flat[:math.prod(shape)].reshape(shape)


def on_host(img, dtype):
    buf = page_locked(tuple(img.shape), dtype)
    buf[:] = as_pixels(img, dtype).cpu().numpy().view(dtype)
    return buf


def encoded(frames, dtype, algorithm):
    """The frames' chunks in page-locked memory."""
    host = [as_pixels(f, dtype).cpu().numpy().view(dtype) for f in frames]
    with ThreadPoolExecutor(8) as pool:
        chunks = list(pool.map(lambda f: chunk.encode(f, algorithm), host))
    bufs = []
    for c in chunks:
        bufs.append(page_locked((len(c),), np.uint8))
        bufs[-1][:] = c
    return bufs


def spot_capacity(h, w, frames):
    return (frames + 1) * max(500, h * w // 1500)


def pixel_capacity(h, w, frames):
    """Spots close with their pixels of the last few frames."""
    return (frames + 3) * max(4096, h * w // 16)


def signal_capacity(case):
    """What the per-frame list holds: the frame's bytes, 16 to a record."""
    return max(case["height"] * case["width"] * case["bits"] // 8 // 16, 1)


def spot_buffer(h, w, frames):
    return page_locked((spot_capacity(h, w, frames),), sf.SPOT)


def pixel_buffer(h, w, frames):
    return page_locked((pixel_capacity(h, w, frames),), sf.PIXEL)


def frames_of(case, seed):
    frames = make_frames(case["height"], case["width"], case.get("frames", 1)
                         * case.get("batches", 1), case["bits"], seed)
    if case["kind"] == "batch" and not case["two_d"]:  # the closed shutter
        last = frames[-1]
        last[last < (1 << case["bits"]) - 1] = 0
    return frames


# -- a user's program before the call ------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "stills":
        shapes = still_shapes(case)
        made = [make_frames(h, w, case["frames"], 16, seed + 7 * k, stills=True)
                for k, (h, w) in enumerate(shapes)]
        eng = Engine(shapes * case["frames"], np.uint16)
        eng.enable_grouping(two_d=True)
        resident(eng, [made[f % 4][f // 4] for f in range(4 * case["frames"])], np.uint16)
        s["engine"] = eng
        s["out"] = [(spot_buffer(*sh, case["frames"]), pixel_buffer(*sh, case["frames"]))
                    for sh in shapes]
        return s
    h, w, dtype = case["height"], case["width"], dtype_of(case)
    frames = frames_of(case, seed)
    if kind in ("find", "series"):
        s["input"] = [on_host(f, dtype) for f in frames]
        s["list"] = page_locked((signal_capacity(case),), sf.SIGNAL_PIXEL)
        if kind == "series":
            s["out"] = spot_buffer(h, w, len(frames)), pixel_buffer(h, w, len(frames))
    elif kind == "batch":
        eng = Engine([(h, w)] * case["frames"], dtype)
        eng.enable_grouping(two_d=case["two_d"])
        if case["masked"]:
            mask = pixel_mask(h, w, seed)
            for f in range(case["frames"]):
                eng.set_pixel_mask(f, mask)
        resident(eng, frames, dtype)
        s["engine"] = eng
        s["out"] = spot_buffer(h, w, case["frames"])
    elif kind == "stream":
        eng = Engine([(h, w)] * case["frames"], dtype, slots=2)
        eng.enable_grouping()
        eng.use_graph(case["graph"])
        s["engine"] = eng
        s["input"] = ([on_host(f, dtype) for f in frames] if case["source"] == "raw"
                      else encoded(frames, dtype, case["source"]))
        s["out"] = [(spot_buffer(h, w, case["frames"]), pixel_buffer(h, w, case["frames"]))
                    for _ in range(case["batches"] + 1)]
    else:
        s["input"] = encoded(frames, dtype, case["source"])[0]
        s["image"] = torch.empty((h, w), device=DEVICE,
                                 dtype=torch.int16 if case["bits"] == 16 else torch.int32)
    torch.cuda.synchronize()
    return s


def resident(eng, frames, dtype):
    for f, img in enumerate(frames):
        t = as_pixels(img, dtype)
        torch.cuda.synchronize()
        eng.upload_device(0, f, t.data_ptr(), t.shape[1] * t.element_size())
        eng.synchronize()


# -- one pass -------------------------------------------------------------------

def signal_fields(sig):
    return {"index": sig["index"].view(np.int32), "value": sig["value"].view(np.int32),
            "background": sig["background"], "population": sig["population"].view(np.int16)}


def spot_fields(spots):
    return {"bbox": spots["bbox"], "position": spots["position"],
            "variance": spots["variance"], "intensity": spots["intensity"],
            "intensity_variance": spots["intensity_variance"],
            "n_signal": spots["n_signal"].view(np.int32), "first": spots["first"].view(np.int64)}


def spots_and_pixels(out, nspots, npixels):
    """The spots' rows as they lie (13 words of eight bytes), their computed
    fields, and the pixels' rows."""
    spots, pixels = out
    return {"rows": spots.view(np.int64).reshape(-1, 13), "position": spots["position"],
            "variance": spots["variance"], "pixels": pixels.view(np.int32).reshape(-1, 3),
            "n": [nspots, npixels]}


def run(s):
    return {"find": run_find, "series": run_series, "batch": run_batch, "stills": run_stills,
            "stream": run_stream, "decode": run_decode}[s["kind"]](s)


def run_find(s):
    return dict(signal_fields(s["list"]), n=len(sf.find(s["input"][0], out=s["list"])))


def run_series(s):
    lab = Labeller(s["height"], s["width"])
    for z, frame in enumerate(s["input"]):
        lab.add(z, sf.find(frame, out=s["list"]))
    lab.finish()
    spots, pixels = lab.spots(), lab.pixels()
    s["out"][0][:len(spots)] = spots
    s["out"][1][:len(pixels)] = pixels
    counts = lab.counts()
    lab.close()
    return dict(spots_and_pixels(s["out"], len(spots), len(pixels)), counts=counts)


def run_batch(s):
    s["engine"].run(0)
    n = len(s["engine"].spots(out=s["out"]))
    return dict(spot_fields(s["out"]), n=n)


def run_stills(s):
    s["engine"].run(0)
    return [collected(s["engine"], k, out) for k, out in enumerate(s["out"])]


def run_stream(s):
    eng, n = s["engine"], s["frames"]
    got = []
    for b in range(s["batches"]):
        part = s["input"][b * n:(b + 1) * n]
        if s["source"] == "raw":
            for f, img in enumerate(part):
                eng.upload(b & 1, f, img)
        elif n == 1:
            eng.upload_chunk(b & 1, 0, part[0], s["source"])
        else:
            eng.upload_chunks(b & 1, part, algorithm=s["source"])
        if b:
            got.append(collected(eng, 0, s["out"][b - 1]))
        eng.run(b & 1)
    got.append(collected(eng, 0, s["out"][-2]))
    eng.finish()
    got.append(collected(eng, 0, s["out"][-1]))
    return got


def collected(eng, k, out):
    return spots_and_pixels(out, len(eng.spots(k, out=out[0])), len(eng.pixels(k, out=out[1])))


def run_decode(s):
    dtype = np.uint16 if s["bits"] == 16 else np.uint32
    chunk.decode_device(s["input"], (s["height"], s["width"]), dtype,
                        s["image"].data_ptr(), algorithm=s["source"])
    return s["image"]


# -- what a pass cannot do without -------------------------------------------------

SIGNAL_SHARE = 0.035  # of a frame's pixels, in the benchmark series
SPOTS_PER_MPX = 250.0


def work(case):
    kind = case["kind"]
    if kind == "stills":
        px = sum(h * w for h, w in still_shapes(case)) * case["frames"]
    else:
        px = case["height"] * case["width"] * case.get("frames", 1) * case.get("batches", 1)
    pixel = case.get("bits", 16) // 8
    signal = SIGNAL_SHARE * px
    spots = SPOTS_PER_MPX * px / 1e6
    share = 0.3  # of a frame's bytes in its chunk
    out = {"find": 16 * signal, "series": 104 * spots + 12 * signal, "batch": 104 * spots,
           "stills": 104 * spots + 12 * signal, "stream": 104 * spots + 12 * signal,
           "decode": px * pixel}[kind]
    read = px * pixel * (share if case.get("source", "raw") != "raw" else 1.0)
    # the dispersion test's and the Poisson test's operations per pixel
    return {"bytes": read + out, "flops": 0 if kind == "decode" else 12 * px}


# -- the same in 64 bits -------------------------------------------------------------

def box_sum(a, radius):
    """Sums over the (2 radius + 1)^2 window clipped to the frame."""
    for dim in (0, 1):
        n = a.shape[dim]
        c = torch.cumsum(a, dim)
        c = torch.cat([torch.zeros_like(c.narrow(dim, 0, 1)), c], dim)
        at = torch.arange(n, device=a.device)
        a = (c.index_select(dim, (at + radius + 1).clamp(max=n))
             - c.index_select(dim, (at - radius).clamp(min=0)))
    return a


def signal_of(img, bits):
    """(index, value, background, population) of a frame's signal pixels: the
    decisions in the path's own precision, the background in 64 bits."""
    real = torch.float32 if bits == 16 else torch.float64
    valid = img < (1 << bits) - 2
    v = torch.where(valid, img, 0)
    m = box_sum(valid.long(), 3)
    q = box_sum(v * v, 3)
    if bits == 16:
        q &= 0xffffffff
    mf, sm, qf = m.to(real), box_sum(v, 3).to(real), q.to(real)
    lhs = mf * qf - sm * sm
    lhs = lhs - sm * (mf - 1)
    rhs = (sm * 6) * torch.sqrt(2 * (mf - 1))
    dispersed = ((m >= 2) & (lhs > rhs)) | ~valid
    kept = (box_sum((~dispersed).long(), 2) == 0) | ~valid
    ground = valid & ~kept
    n = box_sum(ground.long(), 5)
    s = box_sum(torch.where(ground, img, 0), 5)
    mean = torch.where(n >= 2, s.to(real) / n.clamp(min=1).to(real), torch.zeros_like(mf))
    signal = kept & valid & (img > 0) & (img.to(real) >= mean + 3 * torch.sqrt(mean))
    at = torch.nonzero(signal.reshape(-1)).reshape(-1)
    n, s = n.reshape(-1)[at], s.reshape(-1)[at]
    back = torch.where(n >= 2, s.double() / n.clamp(min=1).double(), 0.0)
    return at, img.reshape(-1)[at], back, n


def components(keys, h, w, two_d):
    """Root position of every pixel; keys = frame * h * w + index, ascending."""
    n = len(keys)
    pos = torch.arange(n, device=keys.device)
    edges = []
    for step, ok in ((1, keys % w != 0), (w, keys % (h * w) >= w),
                     (h * w, torch.full_like(keys, not two_d, dtype=torch.bool))):
        to = torch.searchsorted(keys, keys - step).clamp(max=n - 1)
        hit = ok & (keys[to] == keys - step)
        edges.append(torch.stack([pos[hit], to[hit]]))
    a, b = torch.cat(edges, 1)
    root = pos.clone()
    while True:
        ra, rb = root[a], root[b]
        if torch.equal(ra, rb):
            return root
        root.scatter_reduce_(0, torch.maximum(ra, rb), torch.minimum(ra, rb), "amin")
        while True:
            up = root[root]
            if torch.equal(up, root):
                break
            root = up


def spots_of(frames, bits, two_d):
    """Every accepted spot of the series in order: last frame, position,
    variance and intensity."""
    h, w = frames[0].shape
    found = [signal_of(f, bits)[:2] for f in frames]
    keys = torch.cat([i + z * h * w for z, (i, _) in enumerate(found)])
    value = torch.cat([v for _, v in found]).double()
    if not len(keys):
        none = np.zeros((0, 3))
        return np.zeros(0, np.int64), none, none, np.zeros(0)
    z, index = keys // (h * w), keys % (h * w)
    roots, comp = torch.unique(components(keys, h, w, two_d), return_inverse=True)
    k = len(roots)

    def total(x):
        return torch.zeros(k, dtype=torch.float64, device=x.device).index_add_(0, comp, x)

    def extreme(x, how):
        start = torch.zeros(k, dtype=x.dtype, device=x.device)
        return start.scatter_reduce_(0, comp, x, how, include_self=False)

    size, sum1, sum2 = total(torch.ones_like(value)), total(value), total(value * value)
    first, last = extreme(z, "amin"), extreme(z, "amax")
    at = [index % w + 0.5, index // w + 0.5, z + 0.5]
    mean = [total(value * c) / sum1 for c in at]
    den = sum1 * sum1 - sum2
    var = [torch.where(den > 0, total(value * (c - m[comp]) ** 2) / den, 0.0) + 1.0 / 12.0
           for c, m in zip(at, mean)]
    mean[2] = torch.where(last == first, first + 0.5, mean[2])
    pos = torch.arange(len(keys), device=keys.device)
    peak = extreme(torch.where(value == extreme(value, "amax")[comp], pos, len(keys)), "amin")
    apart = sum((c[peak] - m) ** 2 for c, m in zip(at, mean)).sqrt()
    keep = (size >= MIN_SIZE) & (size <= MAX_SIZE) & (apart <= MAX_SEPARATION)
    order = torch.argsort(last, stable=True)  # components are in order of first pixel
    order = order[keep[order]]
    return (last[order].cpu().numpy(), torch.stack(mean, 1)[order].cpu().numpy(),
            torch.stack(var, 1)[order].cpu().numpy(), sum1[order].cpu().numpy())


def filled(x, rows):
    """x with zeros after it, as the buffers have them."""
    return np.concatenate([x, np.zeros((rows - len(x), *x.shape[1:]))])


def exact_spots(found, pick, rows):
    _, position, variance, _ = (x[pick] for x in found)
    return {"rows": None, "position": filled(position, rows),
            "variance": filled(variance, rows), "pixels": None, "n": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "decode":
        return None
    if kind == "stills":
        out = []
        for k, (h, w) in enumerate(still_shapes(case)):
            frames = make_frames(h, w, case["frames"], 16, seed + 7 * k, stills=True)
            out.append(exact_spots(spots_of(frames, 16, True), slice(None),
                                   spot_capacity(h, w, case["frames"])))
        return out
    h, w, bits, n = case["height"], case["width"], case["bits"], case.get("frames", 1)
    frames = frames_of(case, seed)
    if kind == "find":
        back = signal_of(frames[0], bits)[2].cpu().numpy()
        return {"index": None, "value": None, "background": filled(back, signal_capacity(case)),
                "population": None, "n": None}
    if kind == "batch":
        if case["masked"]:
            mask = torch.from_numpy(pixel_mask(h, w, seed)).to(DEVICE)
            for f in frames:
                f[mask] = (1 << bits) - 1
        found = spots_of(frames, bits, case["two_d"])
        rows = spot_capacity(h, w, n)
        _, position, variance, intensity = (filled(x, rows) for x in found)
        return {"bbox": None, "position": position, "variance": variance,
                "intensity": intensity, "intensity_variance": intensity, "n_signal": None,
                "first": None, "n": None}
    found = spots_of(frames, bits, False)
    if kind == "series":
        return dict(exact_spots(found, slice(None), spot_capacity(h, w, n)), counts=None)
    total = n * case["batches"]
    out = []
    for b in range(case["batches"] + 1):
        # run b finishes what ends before its last frame, finish() the rest
        low = b * n - 1 if b else -1
        high = (b + 1) * n - 1 if b < case["batches"] else total
        out.append(exact_spots(found, (found[0] >= low) & (found[0] < high),
                               spot_capacity(h, w, n)))
    return out
