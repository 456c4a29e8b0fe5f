"""The workloads whose speed matters, as calls of the public entry points.

A case is a dict of plain values.  ``prepare`` builds what a stitching program
holds before its frame loop turns (a prepared render or blender, the camera
frames, the output buffers), ``run`` is one pass of that loop, ``work`` the
bytes it cannot do without.  Every output is bytes or 16-bit integers, which
the path defines exactly, so there is no tolerance and no 64-bit reference
here.

Rigs (geometry as in the benchmark rigs of panostitcher_gb300/synth.py):
  fisheye2  two 200 degree full-frame fisheyes back to back
  ricoh     the same two lenses as circular fisheyes in the halves of one
            frame (one source image serves both cameras)
  cube6     six rectilinear cameras, four around, one up, one down
  ring      n rectilinear cameras evenly around the horizon
"""
from __future__ import annotations

import math

import numpy as np
import torch

import panostitcher_gb300 as P
from panostitcher_gb300 import _lib as L
from panostitcher_gb300 import synth as S
from panostitcher_gb300.render import (CudaRicohPanoramaRender, CudaTilingMultibandBlendFast, cvt_bgr32_to_yuv,
                                       cvt_yuv_to_bgr32, render_batch, reproject_to_16s)

PLANAR = {"nv12": L.PS_FMT_NV12, "yuv420p": L.PS_FMT_YUV420P}


def _frame(name, rig, n, sw, sh, dw, levels, hfov=100.0, fin="bgr32", fout="bgr32", host=False, luts=True,
           in_flight=1):
    return {"name": name, "kind": "frame", "rig": rig, "n": n, "sw": sw, "sh": sh, "dw": dw, "levels": levels,
            "hfov": hfov, "fin": fin, "fout": fout, "host": host, "luts": luts, "in_flight": in_flight}


def listed():
    return [
        # the thumbnail of a preview window: the smallest call, all latency
        _frame("thumbnail_256x128", "fisheye2", 2, 160, 120, 256, 5, 200.0, luts=False),
        # a consumer dual-fisheye camera's live preview: one 3-byte frame in, a 3-byte canvas out
        _frame("ricoh_2048x1024", "ricoh", 2, 1920, 960, 2048, 5, 200.0, fin="bgr24", fout="bgr24"),
        # the benchmark rig, one frame at a time: a program that needs each frame before the next
        _frame("cube6_4096x2048", "cube6", 6, 1920, 1080, 4096, 8),
        # the same rig as the benchmark issues it: a frame on each of eight streams
        _frame("cube6_4096x2048_x8", "cube6", 6, 1920, 1080, 4096, 8, in_flight=8),
        # decoder to encoder without leaving the GPU: NV12 frames in, an NV12 canvas out
        _frame("cube6_nv12_device", "cube6", 6, 1920, 1080, 4096, 8, fin="nv12", fout="nv12"),
        # the live-stream task: pinned host NV12 frames up, the NV12 canvas down, frames overlapping
        _frame("cube6_nv12_host", "cube6", 6, 1920, 1080, 4096, 8, fin="nv12", fout="nv12", host=True),
        # the large rig: eight 4K cameras to an 8K canvas, ten levels
        _frame("ring8_7680x3840", "ring", 8, 3840, 2160, 7680, 10, 120.0),
        # one tick of a server: four rigs of uneven size in one launch sequence
        {"name": "batch_four_rigs", "kind": "batch", "rigs": "c3a,c3b,c3c,c3d", "scale": 1},
        # the fast preview mode: feathered linear blend, radius 5% of the width
        {"name": "linear_4096x2048", "kind": "linear", "rig": "cube6", "n": 6, "sw": 1920, "sh": 1080, "dw": 4096,
         "radius": 204, "hfov": 100.0, "fin": "bgr32", "luts": True},
        # the blender alone, fed int16 images warped elsewhere; an odd canvas, partly covered
        {"name": "blender_1999x1001", "kind": "blender", "n": 4, "w": 1999, "h": 1001, "levels": 16, "bits": 16},
        # the remap primitive: one camera into a full-canvas int16 image, as the blender's callers make them
        {"name": "reproject_4096x2048", "kind": "reproject", "sw": 1920, "sh": 1080, "w": 4096, "h": 2048,
         "hfov": 100.0, "fin": "bgr32", "luts": True},
        # the codec handoffs alone: a canvas to encoder planes, decoder planes back to a frame
        {"name": "convert_4096x2048", "kind": "convert", "w": 4096, "h": 2048, "fmt": "nv12"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "batch", "linear", "blender", "reproject", "convert"])
    if kind == "batch":
        rigs = rng.sample(["c1", "c2", "c3a", "c3c", "c3d", "ricoh"], rng.randint(2, 4))
        return {"kind": "batch", "rigs": ",".join(rigs), "scale": rng.randint(2, 16)}
    if kind == "blender":
        w = int(_log(rng, 200, 4000))
        return {"kind": "blender", "n": rng.randint(1, 6), "w": w, "h": max(64, int(w * rng.uniform(0.4, 0.6))),
                "levels": rng.randint(2, 16), "bits": rng.choice([8, 16])}
    if kind == "reproject":
        w = int(_log(rng, 200, 7680))
        sw = int(_log(rng, 160, 3840))
        return {"kind": "reproject", "sw": sw, "sh": max(90, int(sw * rng.uniform(0.5, 0.8))), "w": w, "h": max(64, w // 2),
                "hfov": round(rng.uniform(70, 120), 1), "fin": rng.choice(["bgr24", "bgr32"]),
                "luts": rng.random() < 0.7}
    if kind == "convert":
        w = 2 * int(_log(rng, 100, 3840))
        return {"kind": "convert", "w": w, "h": 2 * max(32, int(w * rng.uniform(0.25, 0.3))),
                "fmt": rng.choice(["nv12", "yuv420p"])}
    rig = rng.choice(["fisheye2", "ricoh", "cube6", "ring"])
    n = {"fisheye2": 2, "ricoh": 2, "cube6": 6, "ring": rng.randint(3, 8)}[rig]
    dw = 4 * int(_log(rng, 64, 1536))                       # canvases of 256 to 6144 pixels across
    sw = max(64, int(dw * rng.uniform(0.3, 0.6)))
    sh = sw // 2 if rig == "ricoh" else max(48, int(sw * rng.uniform(0.55, 1.0)))
    hfov = 200.0 if rig in ("fisheye2", "ricoh") else round(max(90.0, min(130.0, 360.0 / n + rng.uniform(15, 50))), 1)
    fin = rng.choice(["bgr32", "bgr32", "bgr24", "nv12", "yuv420p"])
    fout = rng.choice(["bgr32", "bgr32", "bgr24", "nv12", "yuv420p"])
    if rig == "ricoh" or fin in PLANAR:
        sw, sh = sw // 4 * 4, sh // 2 * 2
    if kind == "linear":
        return {"kind": "linear", "rig": rig, "n": n, "sw": sw, "sh": sh, "dw": dw, "radius": max(2, dw // 20),
                "hfov": hfov, "fin": "bgr24" if fin == "bgr24" else "bgr32", "luts": rng.random() < 0.7}
    if rig == "ricoh":                                       # one 8-bit frame for both cameras
        fin, fout = ("bgr24" if fin == "bgr24" else "bgr32"), ("bgr24" if fout == "bgr24" else "bgr32")
    case = _frame("", rig, n, sw, sh, dw, rng.randint(3, 10), hfov, fin, fout, rng.random() < 0.2, rng.random() < 0.7,
                  rng.choice([1, 1, 1, 4, 8]) if dw <= 3000 else 1)
    if case["host"]:
        case["in_flight"] = 1
    del case["name"]
    return case


# ---- rigs and content -----------------------------------------------------------
def _cams(case):
    rig, n, hfov = case["rig"], case["n"], case["hfov"]
    if rig == "fisheye2":
        return [S.photo_param(1, hfov, 0.0), S.photo_param(1, hfov, 180.0)]
    if rig == "ricoh":
        half = case["sw"] // 2
        return [S.photo_param(3, hfov, 180.0 * k, crop_x=k * half, crop_y=0, crop_width=half, crop_height=case["sh"])
                for k in range(2)]
    if rig == "cube6":
        return ([S.photo_param(0, hfov, y) for y in (0.0, 90.0, 180.0, 270.0)] +
                [S.photo_param(0, hfov, 0.0, 90.0), S.photo_param(0, hfov, 0.0, -90.0)])
    return [S.photo_param(0, hfov, 360.0 * k / n) for k in range(n)]


def _field(gen, h, w, c, amp=10):
    """A smooth field (eight 2-D sinusoids, amplitude 80 around 128) plus integer noise, as uint8 (h, w, c)."""
    p = torch.rand((c, 8, 3), generator=gen, device="cuda")
    x = torch.arange(w, device="cuda") / w
    y = torch.arange(h, device="cuda") / h
    ax = 2 * math.pi * (0.5 + 7.5 * p[:, :, 0, None]) * x
    by = 2 * math.pi * ((0.5 + 7.5 * p[:, :, 1, None]) * y + p[:, :, 2, None])
    f = torch.einsum("cmh,cmw->hwc", by.cos(), ax.sin()) + torch.einsum("cmh,cmw->hwc", by.sin(), ax.cos())
    f = (128 + 10 * f).round_() + torch.randint(-amp, amp + 1, (h, w, c), generator=gen, device="cuda")
    return f.clamp_(0, 255).to(torch.uint8).contiguous()


def _image(gen, h, w, fmt):
    c = 4 if fmt == "bgr32" else 3
    im = _field(gen, h, w, c)
    if c == 4:
        im[..., 3] = 0
    return im


def _planes(gen, h, w, fmt):
    y = _field(gen, h, w, 1)[..., 0].contiguous()
    if fmt == "nv12":
        return [y, _field(gen, h // 2, w // 2, 2).reshape(h // 2, w).contiguous()]
    uv = _field(gen, h // 2, w // 2, 2)
    return [y, uv[..., 0].contiguous(), uv[..., 1].contiguous()]


def _blank(h, w, fmt, host):
    def new(*shape):
        return torch.zeros(shape, dtype=torch.uint8, pin_memory=host, device="cpu" if host else "cuda")
    if fmt == "nv12":
        return [new(h, w), new(h // 2, w)]
    if fmt == "yuv420p":
        return [new(h, w), new(h // 2, w // 2), new(h // 2, w // 2)]
    return new(h, w, 4 if fmt == "bgr32" else 3)


def _host(t):
    """The pinned host array a capture or decode thread would hand over."""
    return t.cpu().pin_memory().numpy()


def _luts(seed, n):
    k = np.random.RandomState(seed & 0x7FFFFFFF).uniform(0.8, 1.2, (n, 3))
    return np.stack([np.stack([S.lut_from_gain(g) for g in row]) for row in k])


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


# ---- what a program holds before its loop ------------------------------------------
def _prepare_frame(case, seed):
    gen, n, sw, sh, dw = _gen(seed), case["n"], case["sw"], case["sh"], case["dw"]
    linear = case["kind"] == "linear"
    fout = "bgr32" if linear else case["fout"]
    fin, host = case["fin"], bool(case.get("host"))
    k = case.get("in_flight", 1)
    r = CudaRicohPanoramaRender() if case["rig"] == "ricoh" else P.CudaPanoramaRender2()
    r.prepare(_cams(case), 0 if linear else 1, case["radius"] if linear else case["levels"], (sw, sh), (dw, dw // 2),
              check=True)
    frames = []
    for _ in range(min(k, 4)):                               # distinct frames of the stream
        if fin in PLANAR:
            f = [_planes(gen, sh, sw, fin) for _ in range(n)]
            f = [[_host(p) for p in ps] for ps in f] if host else f
        else:
            f = [_image(gen, sh, sw, fin) for _ in range(1 if case["rig"] == "ricoh" else n)]
            f = [_host(i) for i in f] if host else f
        frames.append(f)
    outs = [_blank(dw // 2, dw, fout, host) for _ in range(k)]
    if host:
        outs = [[p.numpy() for p in o] if isinstance(o, list) else o.numpy() for o in outs]
    return {"kind": "frame", "r": r, "frames": frames, "outs": outs, "fin": fin, "fout": fout,
            "luts": _luts(seed, n) if case["luts"] else None,
            "streams": [torch.cuda.Stream() for _ in range(k)] if k > 1 else [None]}


def _prepare_batch(case, seed):
    gen, renders, srcs, dsts, luts = _gen(seed), [], [], [], []
    for i, name in enumerate(case["rigs"].split(",")):
        cfg = S.rig(name) if case["scale"] == 1 else S.scaled_rig(S.rig(name), case["scale"])
        r = P.CudaPanoramaRender2()
        r.prepare(cfg.cams, 1, cfg.levels, cfg.src_size, cfg.dst_size, check=True)
        renders.append(r)
        srcs.append([_image(gen, cfg.src_size[1], cfg.src_size[0], "bgr32") for _ in cfg.cams])
        dsts.append(_blank(cfg.dst_size[1], cfg.dst_size[0], "bgr32", False))
        luts.append(_luts(seed + i, cfg.num_cams))
    return {"kind": "batch", "r": renders, "srcs": srcs, "dsts": dsts, "luts": luts}


def _strips(n, w, h):
    """Coverage masks of n overlapping strips with slanted, curved borders; the canvas corners stay uncovered."""
    x, y = np.meshgrid(np.arange(w) / w, np.arange(h) / h)
    bent = x + 0.04 * np.sin(5.0 * y) + 0.03 * y
    lens = ((2 * x - 1) ** 6 + (2 * y - 1) ** 6) < 1.1
    return [(((bent >= (k - 0.35) / n) & (bent < (k + 1.35) / n) & lens) * 255).astype(np.uint8) for k in range(n)]


def _prepare_blender(case, seed):
    gen, n, w, h = _gen(seed), case["n"], case["w"], case["h"]
    masks = _strips(n, w, h)
    b = CudaTilingMultibandBlendFast()
    if not b.prepare(masks, None, case["levels"], 2):
        raise RuntimeError(b.last_error)
    images = []
    for m in masks:
        im = _image(gen, h, w, "bgr32") * (torch.from_numpy(m).cuda() > 0)[..., None]
        images.append(im.to(torch.int16 if case["bits"] == 16 else torch.uint8).contiguous())
    return {"kind": "blender", "b": b, "images": images, "dst": _blank(h, w, "bgr32", False)}


def _prepare_reproject(case, seed):
    gen, sw, sh, w, h = _gen(seed), case["sw"], case["sh"], case["w"], case["h"]
    # the rectilinear view straight ahead on an equirectangular canvas, -1 where the camera does not see
    f = sw / (2 * math.tan(math.radians(case["hfov"]) / 2))
    lon = (torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / w * 2 * math.pi - math.pi
    lat = math.pi / 2 - (torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / h * math.pi
    x = f * torch.tan(lon)[None, :] + (sw - 1) / 2 + 0 * lat[:, None]
    y = (sh - 1) / 2 - f * torch.tan(lat)[:, None] / torch.cos(lon)[None, :]
    ok = (torch.cos(lon)[None, :] > 0) & (x >= 0) & (x < sw) & (y >= 0) & (y < sh)
    xmap, ymap = torch.where(ok, x, -1.0).float().contiguous(), torch.where(ok, y, -1.0).float().contiguous()
    lut = torch.from_numpy(_luts(seed, 1)[0]).cuda() if case["luts"] else None
    return {"kind": "reproject", "src": _image(gen, sh, sw, case["fin"]), "xmap": xmap, "ymap": ymap, "lut": lut,
            "dst": torch.zeros((h, w, 4), dtype=torch.int16, device="cuda")}


def _prepare_convert(case, seed):
    gen, w, h, fmt = _gen(seed), case["w"], case["h"], case["fmt"]
    return {"kind": "convert", "fmt": PLANAR[fmt], "canvas": _image(gen, h, w, "bgr32"),
            "planes_in": _planes(gen, h, w, fmt), "planes_out": _blank(h, w, fmt, False),
            "frame": _blank(h, w, "bgr32", False)}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "linear"):
        return _prepare_frame(case, seed)
    return {"batch": _prepare_batch, "blender": _prepare_blender, "reproject": _prepare_reproject,
            "convert": _prepare_convert}[kind](case, seed)


# ---- one pass ------------------------------------------------------------------
def _render(s, k):
    r, f, out, st = s["r"], s["frames"][k % len(s["frames"])], s["outs"][k], s["streams"][k]
    if s["fin"] in PLANAR:
        if s["fout"] in PLANAR:
            r.render_planar(f, None, s["luts"], PLANAR[s["fin"]], out, PLANAR[s["fout"]], stream=st, check=True)
        else:
            r.render_planar(f, out, s["luts"], PLANAR[s["fin"]], stream=st, check=True)
    elif s["fout"] in PLANAR:
        r.render_yuv(f, out, s["luts"], PLANAR[s["fout"]], stream=st, check=True)
    else:
        r.render(f, out, s["luts"], stream=st, check=True)


def run(state):
    kind = state["kind"]
    if kind == "frame":
        for k in range(len(state["outs"])):
            _render(state, k)
        return state["outs"]
    if kind == "batch":
        render_batch(state["r"], state["srcs"], state["dsts"], state["luts"])
        return state["dsts"]
    if kind == "blender":
        state["b"].blend(state["images"], state["dst"])
        return state["dst"]
    if kind == "reproject":
        reproject_to_16s(state["src"], state["xmap"], state["ymap"], state["dst"], state["lut"])
        return state["dst"]
    cvt_bgr32_to_yuv(state["canvas"], state["planes_out"], state["fmt"])
    cvt_yuv_to_bgr32(state["planes_in"], state["frame"], state["fmt"])
    return [state["planes_out"], state["frame"]]


# ---- what a pass cannot do without ---------------------------------------------------
_BYTES = {"bgr32": 4.0, "bgr24": 3.0, "nv12": 1.5, "yuv420p": 1.5}


def _stitch(n, sw, sh, dw, dh, bin_, bout, frames=1):
    """Camera frames in, canvas out; at least one remapped and blended sample per canvas pixel: the bilinear taps (24
    operations), the pyramid down and up (4/3 of 3 channels x 40) and the accumulation and output (20)."""
    return {"bytes": frames * (n * sw * sh * bin_ + dw * dh * bout), "flops": frames * dw * dh * 204.0}


def work(case):
    kind = case["kind"]
    if kind == "frame":
        n = 1 if case["rig"] == "ricoh" else case["n"]
        return _stitch(n, case["sw"], case["sh"], case["dw"], case["dw"] // 2, _BYTES[case["fin"]],
                       _BYTES[case["fout"]], case["in_flight"])
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for name in case["rigs"].split(","):
            cfg = S.rig(name) if case["scale"] == 1 else S.scaled_rig(S.rig(name), case["scale"])
            w = _stitch(cfg.num_cams, *cfg.src_size, *cfg.dst_size, 4.0, 4.0)
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "linear":
        n = 1 if case["rig"] == "ricoh" else case["n"]
        px = case["dw"] * case["dw"] // 2
        return {"bytes": n * case["sw"] * case["sh"] * _BYTES[case["fin"]] + px * 4.0, "flops": px * 33.0}
    if kind == "blender":
        px = case["w"] * case["h"]
        return {"bytes": px * (case["n"] * (8.0 if case["bits"] == 16 else 4.0) + 4.0), "flops": px * 180.0}
    if kind == "reproject":
        px = case["w"] * case["h"]
        return {"bytes": case["sw"] * case["sh"] * _BYTES[case["fin"]] + px * 16.0, "flops": px * 24.0}
    px = case["w"] * case["h"]
    return {"bytes": px * 11.0, "flops": px * 30.0}
