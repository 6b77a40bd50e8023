"""Performance cases of the render backend.

Each case is one call, or one short sequence of calls, that a program using
this framework makes: the render operations on their own (demosaic, warp,
median stack, seam blend of a chunk), whole panoramas through a render plan,
the colour correction and preview export around them, and the learned blend's
inference and training gradients.  Inputs are synthetic, made on the GPU from
the seed alone.
"""
from __future__ import annotations

import ctypes as ct
import math

import numpy as np
import torch
import torch.nn.functional as F

from image360_b200 import COORDS_REFERENCE, B200ComputeBackend, RenderPlan, blendnet, synth

RGGB, BGGR, GRBG, GBRG = 0x94949494, 0x16161616, 0x61616161, 0x49494949
DEV = "cuda"

# (cin, cout, resolution divisor) of the blend network's eight 3x3 convolutions.
NET = [(16, 32, 1), (32, 32, 1), (32, 64, 2), (64, 64, 2), (64, 64, 2), (96, 32, 1), (32, 32, 1), (32, 4, 1)]


def listed() -> list[dict]:
    return [
        # One 24-megapixel frame as a raw converter hands it over: camera white
        # balance and colour matrix, 14-bit RGGB (the panorama workload's frame).
        dict(name="demosaic_6000x4000", kind="demosaic", w=6000, h=4000, filters=RGGB, black=512),
        # One contributor of one 2048 x 2048 output chunk with its exposure gain;
        # the source has odd sides, as cropped frames have.
        dict(name="warp_2048_from_3999x2999", kind="warp", sw=3999, sh=2999, w=2048, h=2048, gain=1.17),
        # MedianStack of an already aligned burst; the odd sides leave rows and
        # the whole image without 4-byte alignment.
        dict(name="median_9x3001x2003", kind="median", n=9, w=3001, h=2003, sigma=2.0),
        # The burst workload: align 16 frames of 4000 x 3000 and stack them.
        dict(name="warp_median_16x4000x3000", kind="warp_median", n=16, w=4000, h=3000, sigma=2.0),
        # The seam blend of a small chunk through the host-buffer entry point: a
        # drop-in caller with a preview-sized chunk, where latency counts.
        dict(name="host_blend_256x256x3", kind="host_blend", w=256, h=256, k=3, bands=5),
        # The seam blend of one full-size chunk whose contributors are on the
        # device, at the corner of four frames, with the reference's band count.
        dict(name="blend_2048x2048x4", kind="blend", w=2048, h=2048, k=4, bands=5),
        # Colour correction of a frame set toward its first frame.
        dict(name="color_correct_6x6000x4000", kind="color", n=6, w=6000, h=4000),
        # The headline workload: 24 raw frames of 6000 x 4000 in a 3 x 8 grid,
        # demosaiced and rendered to 90 tiles (35400 x 9600), 6 bands, exact.
        dict(name="panorama_24x6000x4000", kind="panorama", fw=6000, fh=4000, rows=3, cols=8, tile=2048, bands=6,
             fp16=0),
        # Uneven output tiles with 1-7 contributors each, in the FP16-storage
        # mode (a quarter of the 256-tile batch).
        dict(name="uneven_64_tiles_fp16", kind="uneven", tiles=64, frames=6, fw=6000, fh=4000, kmax=7, layout=3,
             bands=6, fp16=1),
        # The preview composite of a rendered canvas at its full resolution, as
        # the command line exports it.
        dict(name="preview_17700x9600", kind="preview", w=17700, h=9600, tile=2048, maxdim=17700),
        # Learned blend, inference: 64 windows of an output tile (half of them
        # as a second row of windows, the last column partly outside the tile).
        dict(name="net_infer_64", kind="infer", n=64, w=2000, h=2048, k=3),
        # Learned blend, training: loss and every gradient of the documented
        # batch of 64 windows, forward and backward.
        dict(name="net_gradients_64", kind="gradients", n=64, w=2048, h=2048, k=4),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["demosaic", "warp", "median", "warp_median", "host_blend", "blend", "color", "panorama",
                       "uneven", "preview", "infer", "gradients"])
    if kind == "demosaic":
        return dict(kind=kind, w=_log(rng, 500, 6000), h=_log(rng, 400, 4000),
                    filters=rng.choice([RGGB, BGGR, GRBG, GBRG]), black=rng.choice([0, 256, 512, 1024]))
    if kind == "warp":
        return dict(kind=kind, sw=_log(rng, 400, 6000), sh=_log(rng, 300, 4000), w=_log(rng, 128, 2048),
                    h=_log(rng, 128, 2048), gain=rng.choice([1.0, round(rng.uniform(0.7, 1.4), 3)]))
    if kind == "median":
        return dict(kind=kind, n=rng.randint(2, 32), w=_log(rng, 300, 3000), h=_log(rng, 200, 2000),
                    sigma=rng.choice([1.5, 2.0, 3.0]))
    if kind == "warp_median":
        return dict(kind=kind, n=rng.randint(3, 24), w=_log(rng, 400, 4000), h=_log(rng, 300, 3000),
                    sigma=rng.choice([1.5, 2.0, 3.0]))
    if kind == "host_blend":
        return dict(kind=kind, w=_log(rng, 96, 640), h=_log(rng, 96, 640), k=rng.randint(1, 5), bands=5)
    if kind == "blend":
        return dict(kind=kind, w=_log(rng, 256, 2048), h=_log(rng, 256, 2048), k=rng.randint(2, 6),
                    bands=rng.randint(4, 6))
    if kind == "color":
        return dict(kind=kind, n=rng.randint(2, 6), w=_log(rng, 600, 6000), h=_log(rng, 400, 4000))
    if kind == "panorama":
        return dict(kind=kind, fw=_log(rng, 600, 4000), fh=_log(rng, 400, 3000), rows=rng.randint(1, 3),
                    cols=rng.randint(2, 6), tile=rng.choice([512, 1000, 1024, 2048]), bands=rng.randint(4, 6),
                    fp16=rng.choice([0, 0, 1]))
    if kind == "uneven":
        return dict(kind=kind, tiles=_log(rng, 6, 48), frames=4, fw=_log(rng, 1500, 5000), fh=_log(rng, 1000, 3500),
                    kmax=rng.randint(2, 7), layout=rng.randint(1, 10 ** 6), bands=rng.randint(4, 6),
                    fp16=rng.choice([0, 1]))
    if kind == "preview":
        w, h = _log(rng, 2000, 16000), _log(rng, 1000, 9000)
        return dict(kind=kind, w=w, h=h, tile=rng.choice([512, 1000, 1024, 2048]),
                    maxdim=rng.choice([max(w, h), max(w, h), _log(rng, 1024, max(w, h))]))
    if kind == "infer":
        return dict(kind=kind, n=_log(rng, 4, 160), w=_log(rng, 600, 2048), h=_log(rng, 600, 2048),
                    k=rng.randint(2, 4))
    return dict(kind=kind, n=_log(rng, 4, 64), w=_log(rng, 600, 2048), h=_log(rng, 600, 2048), k=rng.randint(2, 4))


# ---- inputs -----------------------------------------------------------------

def _gen(seed: int, salt: int = 0) -> torch.Generator:
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 7919 + salt)
    return g


def _u16(x: torch.Tensor) -> torch.Tensor:
    """Non-negative values below 65536 as uint16 bits in an int16 tensor."""
    return x.round().clamp(0, 65535).to(torch.int32).to(torch.int16)


def _scene(h: int, w: int, seed: int, peak: float = 15000.0) -> torch.Tensor:
    """(h, w, 3) float32: smooth shading, fine texture, hard-edged rectangles."""
    g = _gen(seed, 1)
    img = torch.zeros((1, 3, h, w), device=DEV)
    for cells, amp in ((5, 0.5), (23, 0.25), (141, 0.15)):
        c = torch.rand((1, 3, max(2, cells * h // max(h, w)), max(2, cells * w // max(h, w))), generator=g, device=DEV)
        img += amp * F.interpolate(c, size=(h, w), mode="bilinear", align_corners=True)
    img = img[0].permute(1, 2, 0).contiguous()
    r = np.random.default_rng(seed)
    for _ in range(24):
        rw, rh = int(w * r.uniform(0.01, 0.08)) + 1, int(h * r.uniform(0.01, 0.08)) + 1
        x, y = int(r.integers(0, w)), int(r.integers(0, h))
        img[y:y + rh, x:x + rw] = torch.tensor(r.uniform(0.02, 0.9, 3), dtype=torch.float32, device=DEV)
    return img * peak


def _noisy(img: torch.Tensor, g: torch.Generator, gain: float = 1.0) -> torch.Tensor:
    """One exposure of a scene: gain and photon plus read noise, never (0,0,0)."""
    s = img * gain
    s = s + torch.randn(s.shape, generator=g, device=DEV) * torch.sqrt(s + 9.0)
    return _u16(s.clamp(min=1.0))


def _layers(h: int, w: int, k: int, seed: int):
    """k overlapping exposures of one scene on an h x w chunk (0 outside each
    footprint, a tilted rectangle) and the footprint corners of each."""
    scene = _scene(h, w, seed)
    g = _gen(seed, 2)
    r = np.random.default_rng(seed + 17)
    cols = math.ceil(math.sqrt(k))
    rows = math.ceil(k / cols)
    yy, xx = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float32),
                            torch.arange(w, device=DEV, dtype=torch.float32), indexing="ij")
    out, corners = [], []
    for i in range(k):
        cx, cy = ((i % cols) + 0.5) * w / cols, ((i // cols) + 0.5) * h / rows
        hw, hh = 0.5 * w / cols * r.uniform(1.2, 1.5), 0.5 * h / rows * r.uniform(1.2, 1.5)
        th = math.radians(r.uniform(-1.0, 1.0))
        c, s = math.cos(th), math.sin(th)
        u, v = (xx - cx) * c + (yy - cy) * s, -(xx - cx) * s + (yy - cy) * c
        inside = (u.abs() <= hw) & (v.abs() <= hh)
        out.append(torch.where(inside[..., None], _noisy(scene, g, r.uniform(0.97, 1.03)), 0).to(torch.int16))
        corners.append([(cx + a * hw * c - b * hh * s, cy + a * hw * s + b * hh * c)
                        for a, b in ((-1, -1), (1, -1), (1, 1), (-1, 1))])
    return out, corners


def _backend() -> B200ComputeBackend:
    be = B200ComputeBackend()
    if be.initialize() != 0:
        raise RuntimeError(be.get_last_error())
    return be


def _ok(be, rc):
    if rc != 0:
        raise RuntimeError(be.get_last_error())


CAM_MUL = np.array([1.93, 1.0, 1.61, 1.0], np.float32)
RGB_CAM = np.array([[1.62, -0.47, -0.15, 0.0], [-0.21, 1.49, -0.28, 0.0], [0.02, -0.51, 1.49, 0.0]], np.float32)


def _cfa(h: int, w: int, black: int, seed: int) -> torch.Tensor:
    s = _scene(h, w, seed, 13000.0)
    g = _gen(seed, 3)
    yy, xx = torch.meshgrid(torch.arange(h, device=DEV) % 2, torch.arange(w, device=DEV) % 2, indexing="ij")
    m = torch.where((yy + xx) % 2 == 1, s[..., 1], torch.where(yy == 0, s[..., 0], s[..., 2]))
    m = m + torch.randn(m.shape, generator=g, device=DEV) * torch.sqrt(m + 9.0) + black
    return _u16(m.clamp(0, 16383))


def _near_identity(n: int, w: int, h: int, r) -> np.ndarray:
    """Hand-held burst: rotations of +-0.2 degrees about the centre, shifts of +-3 pixels."""
    out = []
    for _ in range(n):
        t = math.radians(r.uniform(-0.2, 0.2))
        c, s, cx, cy = math.cos(t), math.sin(t), (w - 1) / 2, (h - 1) / 2
        out.append([[c, -s, cx - c * cx + s * cy + r.uniform(-3, 3)], [s, c, cy - s * cx - c * cy + r.uniform(-3, 3)],
                    [0, 0, 1]])
    return np.array(out, np.float32)


def _outliers(img: torch.Tensor, r) -> torch.Tensor:
    """White transient rectangles over about 5 percent of a frame."""
    h, w = img.shape[:2]
    for _ in range(20):
        rw, rh = max(1, int(w * 0.05)), max(1, int(h * 0.05))
        x, y = int(r.integers(0, w - rw + 1)), int(r.integers(0, h - rh + 1))
        img[y:y + rh, x:x + rw] = 15871
    return img


# ---- learned blend ----------------------------------------------------------

def _net_params(seed: int) -> np.ndarray:
    r = np.random.default_rng(seed)
    parts = []
    for cin, cout, _ in NET:
        sd = math.sqrt(2.0 / (9 * cin))
        parts += [r.normal(0, sd, 9 * cin * cout), r.normal(0, 0.02, cout)]
    return np.concatenate(parts).astype(np.float32)


def _windows(case: dict, seed: int):
    """Layers, target and (x, y, width, height) of the windows of one tile."""
    w, h, n = case["w"], case["h"], case["n"]
    layers, corners = _layers(h, w, case["k"], seed)
    r = np.random.default_rng(seed + 5)
    if case["kind"] == "infer":  # the grid of windows of an output tile, as the learned render walks it
        grid = [(x, y) for y in range(0, h, 256) for x in range(0, w, 256)]
        pos = [grid[i % len(grid)] for i in range(n)]
        wins = [(x, y, min(256, w - x), min(256, h - y)) for x, y in pos]
    else:                        # random training windows
        wins = [(int(r.integers(0, w - 255)), int(r.integers(0, h - 255)), 256, 256) for _ in range(n)]
    target = layers[0].clone()
    for q in layers[1:]:
        target = torch.where((target == 0).all(-1, keepdim=True), q, target)
    return layers, corners, target, wins


def _edges(corners, w: int, h: int, x: int, y: int) -> list[float]:
    """The footprint's four edges in window pixels (clamped to the tile)."""
    out = []
    for e in range(4):
        (ax, ay), (bx, by) = corners[e], corners[(e + 1) % 4]
        cl = lambda px, py: (min(max(px, 0.0), w - 1.0) - x, min(max(py, 0.0), h - 1.0) - y)
        out += [float(np.float32(v)) for v in (*cl(ax, ay), *cl(bx, by))]
    return out


def _net_state(case: dict, seed: int) -> dict:
    layers, corners, target, wins = _windows(case, seed)
    w, h, n, k = case["w"], case["h"], case["n"], case["k"]
    net = blendnet.BlendNet(seed=0)
    net.set_params(_net_params(seed))
    # Windows that the grid visits again (batches larger than a tile) write to
    # a tile output of their own.
    per = math.ceil(w / 256) * math.ceil(h / 256)
    outs = [torch.zeros((h, w, 3), dtype=torch.int16, device=DEV)
            for _ in range(math.ceil(n / per) if case["kind"] == "infer" else 0)]
    jobs = (blendnet.BlendJob * n)()
    for j, (x, y, ww, hh) in enumerate(wins):
        off = (y * w + x) * 6
        J = jobs[j]
        for i in range(4):
            J.slot[i] = layers[i].data_ptr() + off if i < k else None
        J.pixStride, J.rowStride, J.width, J.height = 3, 3 * w, ww, hh
        if case["kind"] == "infer":
            J.out, J.outRowStride = outs[j // per].data_ptr() + off, 3 * w
        else:
            J.target, J.targetRowStride = target.data_ptr() + off, 3 * w
        blendnet.set_edges(J, [_edges(corners[i], w, h, x, y) if i < k else None for i in range(4)])
    return dict(net=net, jobs=jobs, n=n, layers=layers, target=target, outs=outs)


# ---- the cases --------------------------------------------------------------

def prepare(case: dict, seed: int):
    st = _prepare(case, seed)
    st["kind"] = case["kind"]
    return st


def _prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    r = np.random.default_rng(seed)
    be = _backend()
    if kind == "demosaic":
        return dict(be=be, cfa=_cfa(case["h"], case["w"], case["black"], seed), case=case,
                    out=torch.zeros((case["h"], case["w"], 3), dtype=torch.int16, device=DEV))
    if kind == "warp":
        sw, sh, w, h = case["sw"], case["sh"], case["w"], case["h"]
        src = _noisy(_scene(sh, sw, seed), _gen(seed, 4))
        t = math.radians(r.uniform(-1.5, 1.5))
        c, s = math.cos(t), math.sin(t)
        # chunk -> frame: the chunk lies about its own size inside or across the frame's edge
        ox, oy = int(r.integers(-w // 4, max(1, sw - 3 * w // 4))), int(r.integers(-h // 4, max(1, sh - 3 * h // 4)))
        H = np.array([[c, -s, 3.3], [s, c, -2.7], [2e-6 * r.uniform(-1, 1), 2e-6 * r.uniform(-1, 1), 1]], np.float32)
        return dict(be=be, src=src, case=case, H=H, off=(ox, oy),
                    out=torch.zeros((h, w, 3), dtype=torch.int16, device=DEV))
    if kind in ("median", "warp_median"):
        w, h, n = case["w"], case["h"], case["n"]
        scene = _scene(h, w, seed)
        g = _gen(seed, 5)
        frames = [_outliers(_noisy(scene, g), r) for _ in range(n)]
        return dict(be=be, frames=frames, case=case, H=_near_identity(n, w, h, r),
                    out=torch.zeros((h, w, 3), dtype=torch.int16, device=DEV))
    if kind == "host_blend":
        bufs = [q.cpu().numpy().view(np.uint16) for q in _layers(case["h"], case["w"], case["k"], seed)[0]]
        return dict(be=be, bufs=bufs, case=case, out=np.zeros((case["h"], case["w"], 3), np.uint16))
    if kind == "blend":
        return dict(be=be, bufs=_layers(case["h"], case["w"], case["k"], seed)[0], case=case,
                    out=torch.zeros((case["h"], case["w"], 3), dtype=torch.int16, device=DEV))
    if kind == "color":
        g = _gen(seed, 6)
        scene = _scene(case["h"], case["w"], seed)
        frames = []
        for i in range(case["n"]):
            tint = torch.tensor(r.uniform(0.8, 1.2, 3), dtype=torch.float32, device=DEV)
            frames.append(_noisy(scene * tint, g, float(r.uniform(0.7, 1.4))))
        return dict(be=be, frames=frames, case=case)
    if kind == "panorama":
        cfg = synth.PanoConfig(frame_w=case["fw"], frame_h=case["fh"], rows=case["rows"], cols=case["cols"],
                               overlap=0.30, focal=0.75 * case["fw"], bits=14, black=512, gain_lo=0.7, gain_hi=1.4,
                               sigma_read=3.0, tile=case["tile"], bands=case["bands"], n_blobs=60, n_gratings=20,
                               n_rects=60, seed=seed)
        pano = synth.make_panorama(cfg, device=DEV)
        cfa = [c.view(torch.int16).contiguous() for c in pano.cfa]
        rgb = [torch.empty((cfg.frame_h, cfg.frame_w, 3), dtype=torch.int16, device=DEV) for _ in cfa]
        frames = [(q.data_ptr(), cfg.frame_w, cfg.frame_h, H, float(gn))
                  for q, H, gn in zip(rgb, pano.to_canvas, (1.0 / pano.gains).astype(np.float32))]
        return dict(be=be, cfa=cfa, rgb=rgb, cfg=cfg, case=case, **_plan(frames, pano.tiles, case))
    if kind == "uneven":
        # the tiles' sides and placements belong to the case, the pixels to the seed
        u = synth.uneven_tiles(case["tiles"], case["frames"], case["fw"], case["fh"], 0.75 * case["fw"],
                               case["layout"], k_max=case["kmax"])
        g = _gen(seed, 7)
        scene = _scene(case["fh"], case["fw"], seed)
        pool = [_noisy(scene, g, float(r.uniform(0.9, 1.1))) for _ in range(case["frames"])]
        frames = [(pool[f].data_ptr(), case["fw"], case["fh"], H, float(r.uniform(0.9, 1.1)))
                  for f, H in zip(u.frame_of, u.to_canvas)]
        return dict(be=be, pool=pool, case=case, **_plan(frames, u.tiles, case))
    if kind == "preview":
        rects = [(x, y, min(case["tile"], case["w"] - x), min(case["tile"], case["h"] - y))
                 for y in range(0, case["h"], case["tile"]) for x in range(0, case["w"], case["tile"])]
        g = _gen(seed, 8)
        px = sum(q[2] * q[3] for q in rects)
        flat = torch.randint(-32768, 32767, (px * 3,), generator=g, device=DEV, dtype=torch.int16)
        chunks, at = [], 0
        for q in rects:
            chunks.append(flat.data_ptr() + at * 6)
            at += q[2] * q[3]
        scale = case["maxdim"] / max(case["w"], case["h"])
        cap = (int(case["w"] * scale) + 2) * (int(case["h"] * scale) + 2) * 3
        return dict(be=be, flat=flat, chunks=chunks, rects=rects, case=case,
                    out=torch.zeros(cap, dtype=torch.uint8, device=DEV))
    return dict(be=be, case=case, **_net_state(case, seed))


def _plan(frames, tiles, case: dict) -> dict:
    """A render plan whose tile outputs are consecutive ranges of one buffer."""
    at = np.cumsum([0] + [w * h * 3 for _, _, w, h, _ in tiles])
    out = torch.zeros(int(at[-1]), dtype=torch.int16, device=DEV)
    plan = RenderPlan(frames, [(x, y, w, h, cs, out.data_ptr() + 2 * int(a)) for (x, y, w, h, cs), a in zip(tiles, at)],
                      case["bands"], COORDS_REFERENCE)
    if case["fp16"]:
        plan.set_precision(1)
    return dict(plan=plan, out=out)


def run(st):
    kind, be = st["kind"], st["be"]
    case = st["case"]
    if kind == "demosaic":
        _ok(be, be.launch_demosaic(st["cfa"].data_ptr(), case["w"], case["h"], case["black"], CAM_MUL, RGB_CAM,
                                   case["filters"], st["out"].data_ptr()))
        return st["out"]
    if kind == "warp":
        _ok(be, be.launch_warp(st["src"].data_ptr(), case["sw"], case["sh"], st["out"].data_ptr(), case["w"],
                               case["h"], st["H"], *st["off"], gain=case["gain"]))
        return st["out"]
    if kind == "median":
        _ok(be, be.launch_median([f.data_ptr() for f in st["frames"]], case["w"], case["h"], st["out"].data_ptr(),
                                 case["sigma"]))
        return st["out"]
    if kind == "warp_median":
        _ok(be, be.launch_warp_median([f.data_ptr() for f in st["frames"]], case["w"], case["h"], st["H"],
                                      st["out"].data_ptr(), case["w"], case["h"], sigma=case["sigma"]))
        return st["out"]
    if kind == "host_blend":
        _ok(be, be.blend_chunk_contributors(st["bufs"], case["w"], case["h"], st["out"], case["bands"]))
        return st["out"]
    if kind == "blend":
        _ok(be, be.launch_blend([b.data_ptr() for b in st["bufs"]], case["w"], case["h"], st["out"].data_ptr(),
                                case["bands"]))
        return st["out"]
    if kind == "color":
        n = case["n"]
        _ok(be, be.launch_color_correct([f.data_ptr() for f in st["frames"]], [case["w"]] * n, [case["h"]] * n, 0))
        return st["frames"]
    if kind == "panorama":
        black, cm, rc, filt = synth.demosaic_params(st["cfg"])
        for c, q in zip(st["cfa"], st["rgb"]):
            _ok(be, be.launch_demosaic(c.data_ptr(), case["fw"], case["fh"], black, cm, rc, filt, q.data_ptr()))
        _ok(be, st["plan"].execute())
        return st["out"]
    if kind == "uneven":
        _ok(be, st["plan"].execute())
        return st["out"]
    if kind == "preview":
        rc, w, h = be.launch_export_preview(st["chunks"], st["rects"], case["w"], case["h"], case["maxdim"],
                                            st["out"].data_ptr(), st["out"].numel())
        _ok(be, rc)
        return st["out"][:w * h * 3]
    if kind == "infer":
        st["net"].infer(st["jobs"], st["n"], 256, 256)
        return st["outs"]
    g, loss = st["net"].gradients(st["jobs"], st["n"], 256, 256)
    return {"gradients": g, "loss": loss}


def work(case: dict) -> dict:
    """Every input read once and every output written once; operations as the
    path's arithmetic needs them (per pixel, multiplies and adds)."""
    kind = case["kind"]
    if kind == "demosaic":
        px = case["w"] * case["h"]
        return dict(bytes=8 * px, flops=30 * px)
    if kind == "warp":
        px = case["w"] * case["h"]
        return dict(bytes=12 * px, flops=45 * px)
    if kind in ("median", "warp_median"):
        px, n = case["w"] * case["h"], case["n"]
        return dict(bytes=px * 6 * (n + 1), flops=px * n * (45 if kind == "warp_median" else 9))
    if kind in ("host_blend", "blend"):
        px = case["w"] * case["h"]
        return dict(bytes=px * 6 * (case["k"] + 1), flops=px * case["k"] * 60)
    if kind == "color":
        px = case["w"] * case["h"] * case["n"]
        return dict(bytes=px * 12, flops=px * 200)
    if kind == "panorama":
        fpx = case["fw"] * case["fh"] * case["rows"] * case["cols"]
        out = int(case["fw"] * (1 + 0.7 * (case["cols"] - 1))) * int(case["fh"] * (1 + 0.7 * (case["rows"] - 1)))
        return dict(bytes=2 * fpx + 6 * out, flops=fpx * 120 + out * 100)
    if kind == "uneven":
        px = int(case["tiles"] * 1177.6 ** 2)  # the mean tile
        return dict(bytes=int(6 * px * (1 + (case["kmax"] + 1) / 2 * 0.8)), flops=px * 200)
    if kind == "preview":
        s = case["maxdim"] / max(case["w"], case["h"])
        return dict(bytes=int(9 * case["w"] * case["h"] * min(1.0, s * s)), flops=0)
    px = case["n"] * 65536
    net = sum(18 * ci * co // (d * d) for ci, co, d in NET) * px
    if kind == "infer":
        return dict(bytes=px * 6 * (case["k"] + 1), flops=net)
    return dict(bytes=px * 6 * (case["k"] + 1), flops=3 * net)


# ---- 64-bit values of the computed (floating) outputs -----------------------

def _exact_mask(e: list[float]) -> torch.Tensor:
    """0.25 + 0.75 min(1, d / 2048), d the distance to the nearest of 4 segments."""
    yy, xx = torch.meshgrid(torch.arange(256, device=DEV, dtype=torch.float64),
                            torch.arange(256, device=DEV, dtype=torch.float64), indexing="ij")
    d2 = torch.full((256, 256), math.inf, dtype=torch.float64, device=DEV)
    for s in range(4):
        ax, ay, bx, by = e[4 * s:4 * s + 4]
        dx, dy = bx - ax, by - ay
        l2 = dx * dx + dy * dy
        t = (((xx - ax) * dx + (yy - ay) * dy) / l2).clamp(0, 1) if l2 > 0 else torch.zeros_like(xx)
        d2 = torch.minimum(d2, (ax + t * dx - xx) ** 2 + (ay + t * dy - yy) ** 2)
    return 0.25 + 0.75 * (d2.sqrt() / 2048.0).clamp(max=1.0)


def exact(case: dict, seed: int):
    if case["kind"] != "gradients":
        return None  # every other output is a whole number
    layers, corners, target, wins = _windows(case, seed)
    w, h, n, k = case["w"], case["h"], case["n"], case["k"]
    flat = torch.from_numpy(_net_params(seed)).to(DEV).double().requires_grad_(True)
    W, B, at = [], [], 0
    for ci, co, _ in NET:
        W.append(flat[at:at + 9 * ci * co].reshape(co, 3, 3, ci).permute(0, 3, 1, 2))
        B.append(flat[at + 9 * ci * co:at + 9 * ci * co + co])
        at += 9 * ci * co + co
    total = 0.0
    for c0 in range(0, n, 4):
        xs, vs, cs, ts = [], [], [], []
        for x, y, _, _ in wins[c0:c0 + 4]:
            x0 = torch.zeros((16, 256, 256), dtype=torch.float64, device=DEV)
            v = torch.zeros((4, 3, 256, 256), dtype=torch.float64, device=DEV)
            cov = torch.zeros((4, 256, 256), dtype=torch.bool, device=DEV)
            for i in range(k):
                q = (layers[i][y:y + 256, x:x + 256].to(torch.int32) & 0xffff).double().permute(2, 0, 1)
                v[i], cov[i] = q, (q != 0).any(0)
                x0[4 * i:4 * i + 3] = q / 32768.0
                x0[4 * i + 3] = torch.where(cov[i], _exact_mask(_edges(corners[i], w, h, x, y)), 0.0)
            xs.append(x0), vs.append(v), cs.append(cov)
            ts.append((target[y:y + 256, x:x + 256].to(torch.int32) & 0xffff).double().permute(2, 0, 1))
        x0, v, cov, t = torch.stack(xs), torch.stack(vs), torch.stack(cs), torch.stack(ts)
        conv = lambda a, i: F.conv2d(a, W[i], B[i], padding=1)
        a2 = conv(conv(x0, 0).relu(), 1).relu()
        a5 = conv(conv(conv(F.avg_pool2d(a2, 2), 2).relu(), 3).relu(), 4).relu()
        up = F.interpolate(a5, scale_factor=2, mode="nearest")
        l = conv(conv(conv(torch.cat([a2, up], 1), 5).relu(), 6).relu(), 7)
        l = torch.where(cov, l, torch.full_like(l, -1e30))
        wts = torch.where(cov, torch.softmax(l, 1), 0.0)
        e = ((wts[:, :, None] * v).sum(1) - t) / 32768.0
        loss = (e * e).sum() / (n * 65536 * 3)
        loss.backward()
        total += float(loss.detach())
    return {"gradients": flat.grad.cpu().numpy(), "loss": total}
