"""The decision engine's work as its users have it done, as cases that can be timed.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (planes of
seeded content in host memory, an engine, uploaded frames), ``run`` is one pass through the public
Python interface, and what it returns are the decision records themselves (their bytes) -- or, for
the pruner's training step, the gradients, the updated parameters and the loss.

Paths (``case["path"]``):
  frame     one frame through decide_inter / decide_intra, its references new to the engine;
  sequence  the encoder's frame loop: launch with keys, prepare the next source, collect;
  group     leaf frames of a mini-GOP through decide_group, references in the engine by key;
  minigop   a whole mini-GOP (KEY, anchor, mids, leaves) through decide_group, nothing known before;
  batch     launch_group on frames in the engine's store, with or without the learned pruner or
            given keep words;
  multi     launch_multi: one frame each of several streams of uneven size;
  train     one training step of the pruner.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from celv2_b200 import engine as E
from celv2_b200 import gop, pruner
from celv2_b200.pruner.net import SHAPES, Trainer
from celv2_b200.records import DecisionMap

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # The smallest calls, bound by latency: a still or a first frame, KEY, and a small P frame of
        # three references new to the engine (the 416x240 configuration's frames).
        dict(name="key_202x122", path="frame", width=202, height=122, refs=0, depth=8, qindex=120,
             content="natural"),
        dict(name="frame_416x240_r3", path="frame", width=416, height=240, refs=3, depth=10, qindex=120,
             content="natural"),
        # The frame loop of an encoder that decides frame by frame: a ragged small size, and 1080p at
        # seven references.
        dict(name="sequence_641x363_r4", path="sequence", width=641, height=363, refs=4, frames=4, depth=8,
             qindex=160, content="anime"),
        dict(name="sequence_1080p_r7", path="sequence", width=1920, height=1080, refs=7, frames=2, depth=10,
             qindex=130, content="natural"),
        # A KEY frame at full size: intra and partition choice alone.
        dict(name="key_1080p", path="frame", width=1920, height=1080, refs=0, depth=10, qindex=130,
             content="natural"),
        # Mini-GOP leaves, decided as a batch: 720p with few references, 1080p with seven.
        dict(name="leaves_720p_r2", path="group", width=1280, height=720, refs=2, frames=10, depth=8, qindex=100,
             content="natural"),
        dict(name="leaves_1080p_r7", path="group", width=1920, height=1080, refs=7, frames=5, depth=10,
             qindex=130, content="natural"),
        # The headline: a whole 1080p 10-bit mini-GOP, host planes in, every record out.
        dict(name="minigop_1080p_r7", path="minigop", width=1920, height=1080, refs=7, frames=17, depth=10,
             qindex=130, content="natural"),
        # The learned pruner on 1080p leaves, replayed as a CUDA graph.
        dict(name="pruned_1080p_r7", path="batch", width=1920, height=1080, refs=7, frames=5, depth=10,
             qindex=130, content="natural", keep="pruner", graphs=True),
        # 4K animation-like frames with keep words from the caller.
        dict(name="masked_4k_r7", path="batch", width=3840, height=2160, refs=7, frames=1, depth=10, qindex=130,
             content="anime", keep="words", graphs=False),
        # Six streams of uneven size, a frame of each in one batch.
        dict(name="multi_6_streams_r7", path="multi", width=3840, height=2160, refs=7, frames=6, depth=10,
             qindex=130, content="natural"),
        # A training step of the pruner at its training batch.
        dict(name="train_4096", path="train", batch=4096),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["frame", "frame", "sequence", "group", "minigop", "batch", "multi", "train"])
    if path == "train":
        return dict(path="train", batch=size(64, 4096))
    hi = {"frame": 3840, "sequence": 1920, "group": 1920, "minigop": 1920, "batch": 3840, "multi": 3840}[path]
    width = size({"frame": 16, "multi": 256}.get(path, 96), hi)
    height = max(16, min(2160 if hi == 3840 else 1080, int(width * rng.uniform(0.4, 1.0))))
    refs = rng.randint(0, 7) if path == "frame" else rng.randint(1, 7)
    case = dict(path=path, width=width, height=height, refs=refs, depth=rng.choice([8, 10]),
                qindex=rng.randint(60, 220), content=rng.choice(["natural", "anime"]))
    if path == "sequence":
        case["frames"] = rng.randint(2, 4)
    elif path == "group":
        case["frames"] = rng.randint(2, 8)
    elif path == "minigop":
        case["frames"] = rng.randint(5, 17)
        if case["refs"] > case["frames"] - 1:
            case["refs"] = case["frames"] - 1
    elif path == "batch":
        case["frames"] = rng.randint(1, 4) if width <= 1920 else 1
        case["keep"] = rng.choice(["none", "pruner", "words"])
        case["graphs"] = rng.choice([True, False])
    elif path == "multi":
        case["frames"] = rng.randint(2, 6)
    return case


# ---- content -------------------------------------------------------------------------------------
# The seeded content of celv2_b200.synth, rendered on the GPU: natural-like (sinusoids, rectangles,
# regions in affine motion, noise) and animation-like (flat shapes with hard edges in piecewise
# motion, sparse noise).

def _natural(rng, gen, w, h, n):
    ns, nr, gx, gy, motion = 8, 12, 4, 3, 24.0 if w >= 960 else 6.0
    period, angle = rng.uniform(8.0, 64.0, ns), rng.uniform(0.0, np.pi, ns)
    phase, amp = rng.uniform(0.0, 2 * np.pi, ns), rng.uniform(0.3, 1.0, ns)
    amp *= 380.0 / amp.sum()
    kx, ky = np.cos(angle) * 2 * np.pi / period, np.sin(angle) * 2 * np.pi / period
    rw, rh = rng.integers(max(8, w // 16), max(9, w // 4), nr), rng.integers(max(8, h // 16), max(9, h // 4), nr)
    rx, ry, level = rng.uniform(0, w, nr), rng.uniform(0, h, nr), rng.uniform(96.0, 928.0, nr)
    trans = torch.tensor(rng.uniform(-motion, motion, (gx * gy, 2)), dtype=torch.float32, device=DEV)
    rot = torch.tensor(rng.uniform(-0.01, 0.01, gx * gy), dtype=torch.float32, device=DEV)
    zoom = torch.tensor(rng.uniform(-0.01, 0.01, gx * gy), dtype=torch.float32, device=DEV)
    y, x = torch.meshgrid(torch.arange(h, device=DEV), torch.arange(w, device=DEV), indexing="ij")
    ix, iy = (x * gx // w).clamp(max=gx - 1), (y * gy // h).clamp(max=gy - 1)
    reg = iy * gx + ix
    cx, cy = (ix + 0.5) * (w / gx), (iy + 0.5) * (h / gy)
    dx, dy = x - cx, y - cy
    pos = np.zeros((nr, 2))
    for t in range(n):
        a, s = rot[reg] * t, 1.0 + zoom[reg] * t
        sx = (a.cos() * dx - a.sin() * dy) * s + cx - trans[reg, 0] * t
        sy = (a.sin() * dx + a.cos() * dy) * s + cy - trans[reg, 1] * t
        v = torch.full((h, w), 512.0, device=DEV)
        for k in range(ns):
            v += float(amp[k]) * torch.sin(float(kx[k]) * sx + float(ky[k]) * sy + float(phase[k]))
        for k in range(nr):
            x0, y0 = rx[k] + pos[k, 0], ry[k] + pos[k, 1]
            v[(sx >= x0) & (sx < x0 + float(rw[k])) & (sy >= y0) & (sy < y0 + float(rh[k]))] = float(level[k])
        v += 4.0 * torch.randn((h, w), generator=gen, device=DEV)
        pos += np.round(rng.uniform(-motion, motion, (nr, 2)) * 4) / 4
        yield v.clamp(64, 960)


def _anime(rng, gen, w, h, n):
    px, py, shapes = 4, 3, 40
    pal = rng.uniform(64.0, 960.0, int(rng.integers(8, 25)))
    x0, y0 = rng.uniform(-w * 0.2, w * 1.2, shapes), rng.uniform(-h * 0.2, h * 1.2, shapes)
    sw, sh = rng.uniform(w * 0.03, w * 0.3, shapes), rng.uniform(h * 0.03, h * 0.3, shapes)
    colour, oval = rng.integers(0, len(pal), shapes), rng.integers(0, 2, shapes)
    lim = 48.0 if w >= 960 else 12.0
    vel = torch.tensor(rng.uniform(-lim, lim, (px * py, 2)).round(), dtype=torch.float32, device=DEV)
    y, x = torch.meshgrid(torch.arange(h, device=DEV), torch.arange(w, device=DEV), indexing="ij")
    piece = (y * py // h) * px + x * px // w
    for t in range(n):
        sx, sy = x - vel[piece, 0] * t, y - vel[piece, 1] * t
        v = torch.full((h, w), float(pal[0]), device=DEV)
        for k in range(shapes):
            ax, ay, aw, ah = float(x0[k]), float(y0[k]), float(sw[k]), float(sh[k])
            if oval[k]:
                m = ((sx - ax) / aw) ** 2 + ((sy - ay) / ah) ** 2 < 1.0
            else:
                m = (sx >= ax) & (sx < ax + aw) & (sy >= ay) & (sy < ay + ah)
            v = torch.where(m, float(pal[colour[k]]), v)
        noisy = torch.rand((h, w), generator=gen, device=DEV) < 0.005
        yield v + noisy * torch.randn((h, w), generator=gen, device=DEV)


def _planes(case, seed, n, width=None, height=None, pinned=False):
    """n luma planes, padded to multiples of 8 by edge replication, in host memory (uint8 or uint16)."""
    w, h = width or case["width"], height or case["height"]
    pw, ph = (w + 7) & ~7, (h + 7) & ~7
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    out = []
    for v in (_natural if case["content"] == "natural" else _anime)(rng, gen, w, h, n):
        v = v.round().clamp(0, 1023).to(torch.int16)
        if case["depth"] == 8:
            v = ((v + 2) >> 2).clamp(max=255).to(torch.uint8)
        v = torch.cat([v, v[:, -1:].expand(h, pw - w)], 1)
        v = torch.cat([v, v[-1:].expand(ph - h, pw)], 0).cpu().numpy()
        v = v if case["depth"] == 8 else v.view(np.uint16)
        if pinned:
            p = E.host_array(v.shape, v.dtype)
            p[...] = v
            v = p
        out.append(v)
    return out


def _keep_words(rng, nsb):
    """Keep words as a pruner proposes them: some references, the levels from the smallest up, intra
    with a few modes where kept."""
    refs = rng.integers(1, 128, nsb) & rng.integers(1, 128, nsb)
    levels = np.array([0x8, 0xC, 0xE, 0xF])[rng.choice(4, nsb, p=[0.5, 0.25, 0.15, 0.1])] << 8
    modes = np.where(rng.random(nsb) < 0.4, E.KEEP_INTRA | (7 << 16) | (rng.integers(0, 1 << 10, nsb) << 19), 0)
    return (refs | levels | modes).astype(np.uint32)


def _stream_sizes(case):
    """The streams' sizes: the largest given, the others down the usual ladder from it."""
    f = [1.0, 0.5, 0.5, 1 / 3, 0.25, 1 / 6][:case["frames"]]
    return [(max(32, int(case["width"] * k)), max(32, int(case["height"] * k))) for k in f]


# ---- the cases -----------------------------------------------------------------------------------

def prepare(case, seed):
    path = case["path"]
    s = dict(case=case)
    if path == "train":
        return _prepare_train(case, seed)
    if path == "multi":
        s["engines"] = []
        for i, (w, h) in enumerate(_stream_sizes(case)):
            e = E.CudaEngine(w, h)
            for k, p in enumerate(_planes(case, seed * 16 + i, case["refs"] + 1, w, h)):
                e.upload(p, k)
            e.finish()
            s["engines"].append(e)
        return s
    e = s["engine"] = E.CudaEngine(case["width"], case["height"])
    if path == "frame":
        s["src"], *s["refs"] = _planes(case, seed, case["refs"] + 1)
    elif path == "sequence":
        s["planes"] = _planes(case, seed, case["refs"] + case["frames"])
        s["next"] = case["refs"]  # the stream's next frame
    elif path == "group":
        # the leaves lie between their references, as in a mini-GOP
        p = _planes(case, seed, case["refs"] + case["frames"], pinned=True)
        s["srcs"], s["refs"] = p[:case["frames"]], p[case["frames"]:]
    elif path == "minigop":
        s["planes"] = _planes(case, seed, case["frames"], pinned=True)
        s["plan"] = gop.mini_gop_plan(case["frames"], case["refs"])
        s["base"] = 0
    else:  # batch
        n = case["refs"] + case["frames"]
        for k, p in enumerate(_planes(case, seed, n)):
            e.upload(p, k)
        if case["keep"] == "pruner":
            pruner.set_on(e, pruner.load())
        rng = np.random.default_rng(seed)
        s["words"] = [_keep_words(rng, e.sb_cols * e.sb_rows) for _ in range(case["frames"])]
        e.set_config(E.CFG_GRAPHS, int(case["graphs"]))
        e.finish()
    return s


def _bytes(dm):
    return dm.records.view(np.uint8)


def run(s):
    case = s["case"]
    path = case["path"]
    if path == "train":
        t = s["trainer"]
        t.step(s["x"], s["y"], s["w"])
        return {"grads": t.g, "params": t.p, "loss": t.loss}
    q = case["qindex"]
    if path == "multi":
        refs = list(range(1, case["refs"] + 1))
        dms = [DecisionMap() for _ in s["engines"]]
        E.launch_multi([(e, 0, refs) for e in s["engines"]], q, dms=dms)
        for e in s["engines"]:
            e.finish()
        return [_bytes(d) for d in dms]
    e = s["engine"]
    if path == "frame":
        return _bytes(e.decide_inter(s["src"], s["refs"], q) if s["refs"] else e.decide_intra(s["src"], q))
    if path == "sequence":
        # the stream's next frames, each against the ones before it; a picture's key is its number,
        # and the clip plays forwards and backwards in turn
        planes, nr, out = s["planes"], case["refs"], []
        n = len(planes)
        picture = lambda k: planes[k % n if k // n % 2 == 0 else n - 1 - k % n]  # noqa: E731
        for i in range(s["next"], s["next"] + case["frames"]):
            ks = [i - k for k in range(1, nr + 1)]
            dm, gate = DecisionMap(), E.RowGate()
            e.launch(picture(i), [picture(k) for k in ks], q, dm, ks, i)
            e.prepare(picture(i + 1), i + 1)
            e.collect(dm, gate)
            out.append(_bytes(dm))
        s["next"] += case["frames"]
        return out
    if path == "group":
        n, keys = len(s["srcs"]), list(range(len(s["refs"])))
        dms = e.decide_group(s["srcs"], [s["refs"]] * n, q, [keys] * n, pinned=True)
        return [_bytes(d) for d in dms]
    if path == "minigop":
        planes, base, out = s["planes"], s["base"], {}
        s["base"] += len(planes)
        for group in s["plan"]:
            dms = e.decide_group([planes[d] for d, _ in group], [[planes[r] for r in rs] for _, rs in group], q,
                                 [[base + r for r in rs] for _, rs in group], wait=False, pinned=True)
            for (d, _), dm in zip(group, dms):
                out[d] = dm
        e.finish()
        return [_bytes(out[d]) for d in sorted(out)]
    # batch
    n, nr = case["frames"], case["refs"]
    if case["keep"] == "words":
        for j in range(n):
            e.set_keep(j, s["words"][j])
    dms = [DecisionMap() for _ in range(n)]
    e.launch_group(list(range(n)), [list(range(n, n + nr))] * n, q, dms=dms)
    e.finish()
    return [_bytes(d) for d in dms]


# ---- work ----------------------------------------------------------------------------------------

REC = 38872  # bytes of a superblock's record


def _jobs(case):
    """(width, height, references) of every frame a pass decides, and the planes it reads from the host."""
    w, h, path = case["width"], case["height"], case["path"]
    if path == "frame":
        return [(w, h, case["refs"])], case["refs"] + 1
    if path == "sequence":
        return [(w, h, case["refs"])] * case["frames"], case["refs"] + case["frames"]
    if path == "minigop":
        return [(w, h, len(rs)) for g in gop.mini_gop_plan(case["frames"], case["refs"]) for _, rs in g], case["frames"]
    if path == "multi":
        return [(a, b, case["refs"]) for a, b in _stream_sizes(case)], 0
    return [(w, h, case["refs"])] * case["frames"], case["frames"] if path == "group" else 0


def work(case):
    """Bytes: every plane read once (at its sample size where it comes from the host), every record
    written once. Operations (32-bit integer): per 8x8 cell and reference one +-8 whole-pel search
    at each pyramid level (289 SADs of 16 four-sample words, 2 each) and 17 + 8 quarter-pel 8x8
    SATDs (four 4x4 Hadamards of 112); per superblock 29,952 intra Hadamards, and per reference 256
    at each of the 16 vectors a superblock has at the least where its motion is not uniform."""
    if case["path"] == "train":
        b = case["batch"]
        fwd = 2 * (256 * 16 * 9 + 64 * 32 * 144 + 16 * 32 * 288 + 64 * 632 + 24 * 64)
        return {"bytes": 4.0 * (b * (E.PRUNER_FEATURES + 2 * E.PRUNER_OUTPUTS) + 7 * E.PRUNER_PARAMS),
                "flops": 3.0 * fwd * b}
    jobs, planes = _jobs(case)
    byt = planes * case["width"] * case["height"] * (1 if case["depth"] == 8 else 2)
    ops = 0.0
    for w, h, r in jobs:
        nsb, cells = ((w + 63) // 64) * ((h + 63) // 64), ((w + 7) // 8) * ((h + 7) // 8)
        byt += nsb * REC + (w * h * (r + 1) if planes == 0 else 0)
        full = 1.0 if case.get("keep", "none") == "none" else 0.3
        ops += r * cells * (289 * 32 * 1.33 + 25 * 4 * 112 * full)
        ops += nsb * 112 * (29952 + r * 256 * 16) * full
    return {"bytes": float(byt), "flops": float(ops)}


# ---- the pruner's training step ------------------------------------------------------------------

def _samples(case, seed):
    """Features, labels and weights with the training records' ranges, on the GPU."""
    b = case["batch"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    u = lambda *n: torch.rand(n, generator=g, device=DEV)  # noqa: E731
    yy, xx = torch.meshgrid(torch.arange(16.0, device=DEV), torch.arange(16.0, device=DEV), indexing="ij")
    k = (u(b, 1, 1, 3) - 0.5) * 1.6
    img = 0.8 * torch.sin(k[..., 0] * xx + k[..., 1] * yy + 6.28 * k[..., 2])
    img = (img + 0.1 * torch.randn((b, 16, 16), generator=g, device=DEV)).reshape(b, 256)
    img = img - img.mean(1, keepdim=True)
    nrefs = torch.randint(1, 8, (b, 1), generator=g, device=DEV)
    present = (torch.arange(7, device=DEV)[None] < nrefs).float()
    sad = (0.45 + 0.25 * u(b, 7, 1) + 0.15 * u(b, 7, 16)) * present[..., None]
    lam = torch.full((b, 1), 0.5, device=DEV) + 0.1 * u(b, 1)
    x = torch.cat([img, sad.reshape(b, 112), present, lam], 1).contiguous()
    y = (u(b, E.PRUNER_OUTPUTS) < 0.3).float()
    w = 1.0 + 19.0 * u(b, E.PRUNER_OUTPUTS) ** 8
    w[:, 22:] = 0.0
    return x, y, w.contiguous()


def _prepare_train(case, seed):
    x, y, w = _samples(case, seed)
    return dict(case=case, x=x, y=y, w=w, trainer=Trainer(case["batch"], params=pruner.load()["params"]))


def exact(case, seed):
    """The training step in 64 bits: gradients, the parameters after one Adam step, the loss. The
    records of the other cases are whole numbers, the same from any engine."""
    if case["path"] != "train":
        return None
    x, y, w = (t.double() for t in _samples(case, seed))
    p = torch.from_numpy(pruner.load()["params"]).to(DEV).double().requires_grad_(True)
    part, at = {}, 0
    for name, shape in SHAPES:
        n = int(np.prod(shape))
        part[name], at = p[at:at + n].view(shape), at + n

    def conv(a, i, cin, stride):  # a weight's column index is (ky * 3 + kx) * cin + channel
        k = part[f"W{i}"].view(-1, 3, 3, cin).permute(0, 3, 1, 2)
        return torch.relu(torch.nn.functional.conv2d(a, k, part[f"b{i}"], stride=stride, padding=1))

    a = conv(conv(conv(x[:, :256].view(-1, 1, 16, 16), 1, 1, 1), 2, 16, 2), 3, 32, 2)
    h = torch.cat([a.permute(0, 2, 3, 1).reshape(len(x), 512), x[:, 256:]], 1)
    z = torch.relu(h @ part["W4"].T + part["b4"]) @ part["W5"].T + part["b5"]
    loss = (w * torch.nn.functional.binary_cross_entropy_with_logits(z, y, reduction="none")).sum() / len(x)
    g, = torch.autograd.grad(loss, p)
    m, v = 0.1 * g / (1 - 0.9), 0.001 * g * g / (1 - 0.999)
    new = p - 2e-3 * (m / (v.sqrt() + 1e-8) + 1e-4 * p)
    return {"grads": g, "params": new.detach(), "loss": loss.detach().reshape(1)}
