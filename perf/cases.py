"""What is timed: passes through the public entry points of chaos_gb300, as a
program that uses the framework makes them, from a 256-pixel preview to an 8K
frame.

Each case names a `path` (one way into the framework) and its sizes.  The seed
of a preparation moves the view by a fraction of its span and picks the palette
and the jitter, so that two seeds are two inputs of about the same work.
"""
import atexit
import functools
import math
import os
import random
import sys
from fractions import Fraction

import numpy as np
import torch

# the package lies in chaos-ultra_gb300/ of the repository's root, the working folder
_PKG = os.path.join(os.getcwd(), "chaos-ultra_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import chaos_gb300 as cg  # noqa: E402
from chaos_gb300.palette import default_palette, seeded_palette  # noqa: E402
from chaos_gb300.workloads import deep_zoom_centre  # noqa: E402

# Points on the boundary next to the main cardioid, where zooms go: the ends of
# bisections along seeded rays (chaos_gb300.workloads.boundary_point of seeds 2
# and 11 to 17, maxIter 20000).
BOUNDARY = [
    (0.3004395381261789, -0.5705143370804123), (-0.6496565059452619, -0.3511885889760247),
    (0.32394707824152064, 0.4191877501170017), (0.3672543788913769, -0.35644739925265856),
    (-0.4209536323934241, -0.5717400192728543), (-0.3713113843165885, 0.6288180266652033),
    (0.23326708839601773, 0.5159485646056297), (-0.7152526241535606, -0.22101066431415722),
]
MIXED = (0, 2, 3, 6)  # those around which samples escape within a few thousand steps at every span down to 1e-7
SEAHORSE = (-0.743643887, 0.131825904)  # a valley of the set that a zoom passes through
JULIA_C = (-0.8, 0.156)
BLACK = 0xFF000000
MAX_SAMPLES_DEEP = 640 * 360 * 4  # binary64 samples of the largest deep frame


def listed():
    return [
        # A thumbnail or the first image of an interactive view: the whole set on 256 columns.  Launches and latency.
        {"name": "preview_f32", "path": "frame", "width": 256, "height": 144, "double": False, "arith": "fma",
         "spp": 1, "max_iter": 500, "view": "whole", "span": 3.0, "out": "rgba", "fractal": "mandelbrot"},
        # The plain Mandelbrot configuration: 1024x1024, binary32, span 3, maxIter 1000, counts and smooth counts.
        {"name": "whole_set_f32", "path": "frame", "width": 1024, "height": 1024, "double": False, "arith": "parity",
         "spp": 1, "max_iter": 1000, "view": "whole", "span": 3.0, "out": "counts", "fractal": "mandelbrot"},
        # The binary64 configuration (span 1e-10 at a boundary point, maxIter 20000, 4 jittered samples, palette
        # colours, rounded as the reference): a window of a sixth of its sides.
        {"name": "deep_frame_f64", "path": "frame", "width": 640, "height": 360, "double": True, "arith": "parity",
         "spp": 4, "max_iter": 20000, "view": "b0", "span": 640e-10 / 3840, "out": "rgba", "fractal": "mandelbrot"},
        # renderQuality on the module's default view (maxIter 1600, up to 5 adaptive samples) at full HD.
        {"name": "quality_f32", "path": "quality", "width": 1920, "height": 1080, "double": False,
         "arith": "contracted", "max_iter": 1600, "max_ss": 5.0, "view": "whole", "span": 3.6,
         "fractal": "mandelbrot"},
        # renderQuality of a deep view in binary64, an odd window size.
        {"name": "quality_f64", "path": "quality", "width": 853, "height": 479, "double": True,
         "arith": "contracted", "max_iter": 5000, "max_ss": 4.0, "view": "b2", "span": 1e-6,
         "fractal": "mandelbrot"},
        # renderFast while zooming in at 4K: sample reuse, foveation, adaptive samples in the fovea; then compose.
        {"name": "zoom_4k", "path": "fast", "width": 3840, "height": 2160, "double": False, "arith": "contracted",
         "max_iter": 400, "max_ss": 2.0, "view": "seahorse", "span": 0.02, "zoom": 1.02, "foveation": True,
         "fractal": "mandelbrot"},
        # renderFast on a resting 8K view: every pixel but the border comes from the last frame; then compose.
        {"name": "rest_8k", "path": "fast", "width": 7680, "height": 4320, "double": False, "arith": "contracted",
         "max_iter": 100, "max_ss": 4.0, "view": "whole", "span": 3.0, "zoom": 1.0, "foveation": False,
         "fractal": "mandelbrot"},
        # The deep-zoom configuration: 1920x1080, span 1e-200, maxIter 100000, binary32 differences from an orbit
        # that the program keeps.
        {"name": "perturb_f32", "path": "perturb", "width": 1920, "height": 1080, "double": False,
         "max_iter": 100000, "span_log10": -200.0},
        # One step of a deep zoom to a new centre: its reference orbit and a frame with binary64 differences.
        {"name": "deep_step_f64", "path": "deep_step", "width": 1280, "height": 720, "double": True,
         "max_iter": 100000, "span_log10": -60.0},
        # Many viewports of uneven size and depth in one launch (an atlas, a tile server's backlog).
        {"name": "batch_16", "path": "batch", "viewports": 16, "side_min": 96, "side_max": 768, "iter_min": 500,
         "iter_max": 20000, "rounded": False, "specs": 4},
        # A Newton fractal of the default polynomial, its default view.
        {"name": "newton_f32", "path": "quality", "width": 1920, "height": 1080, "double": False, "arith": "parity",
         "max_iter": 200, "max_ss": 2.0, "view": "origin", "span": 4.0, "fractal": "newton generic"},
        # Zoom sessions of a running server, half shallow, half past binary32: open, a burst of frames, read, close.
        {"name": "serve_8", "path": "serve", "sessions": 8, "frames": 6, "width": 1280, "height": 720,
         "max_iter": 2000, "max_ss": 2.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _shape(rng, lo, hi):
    """Width log-uniform in [lo, hi], any aspect between 1:1 and 2.1:1, odd sizes among them."""
    w = int(_log(rng, lo, hi + 1))
    return w, max(1, int(w / rng.uniform(1.0, 2.1)))


def draw(rng):
    path = rng.choice(["frame", "frame_deep", "quality", "quality_deep", "fast", "fast", "perturb", "deep_step",
                       "batch", "newton", "serve"])
    if path == "frame":
        w, h = _shape(rng, 64, 2048)
        julia = rng.random() < 0.3
        return {"path": "frame", "width": w, "height": h, "double": False, "arith": rng.choice(["fma", "parity"]),
                "spp": rng.choice([1, 1, 2, 4]), "max_iter": int(_log(rng, 100, 2000)),
                "view": "origin" if julia else rng.choice(["whole", "seahorse"]),
                "span": 3.0 if julia else _log(rng, 0.05, 3.0), "out": rng.choice(["rgba", "counts"]),
                "fractal": "julia" if julia else "mandelbrot"}
    if path == "frame_deep":
        spp = rng.choice([1, 2, 4])
        w, h = _shape(rng, 64, int(math.sqrt(MAX_SAMPLES_DEEP / spp)))
        span = _log(rng, 1e-11, 1e-4)
        deep = span < 3e-8  # there only a limit of 20000 lets a sample escape
        return {"path": "frame", "width": w, "height": h, "double": True, "arith": rng.choice(["fma", "parity"]),
                "spp": spp, "max_iter": 20000 if deep else int(_log(rng, 3000, 20000)),
                "view": "b%d" % rng.choice(range(8) if deep else MIXED), "span": span,
                "out": rng.choice(["rgba", "counts"]), "fractal": "mandelbrot"}
    if path == "quality":
        w, h = _shape(rng, 96, 1920)
        julia = rng.random() < 0.3
        return {"path": "quality", "width": w, "height": h, "double": False,
                "arith": rng.choice(["contracted", "parity"]), "max_iter": int(_log(rng, 200, 1600)),
                "max_ss": float(rng.choice([1, 2, 4, 5, 9])), "view": "origin" if julia else "whole",
                "span": 4.0 if julia else 3.6, "fractal": "julia" if julia else "mandelbrot"}
    if path == "quality_deep":
        w, h = _shape(rng, 96, 860)
        return {"path": "quality", "width": w, "height": h, "double": True,
                "arith": rng.choice(["contracted", "parity"]), "max_iter": int(_log(rng, 3000, 5000)),
                "max_ss": float(rng.choice([1, 2, 4])), "view": "b%d" % rng.choice(MIXED),
                "span": _log(rng, 1e-7, 1e-4), "fractal": "mandelbrot"}
    if path == "fast":
        w, h = _shape(rng, 160, 7680)
        zoom = rng.choice([1.0, 1.02, 1.0 / 1.02])
        return {"path": "fast", "width": w, "height": h, "double": False,
                "arith": rng.choice(["contracted", "parity"]), "max_iter": int(_log(rng, 100, 800)),
                "max_ss": float(rng.choice([1, 2, 4])), "view": rng.choice(["seahorse", "whole"]),
                "span": _log(rng, 0.02, 3.0), "zoom": zoom, "foveation": rng.random() < 0.5,
                "fractal": "mandelbrot"}
    if path in ("perturb", "deep_step"):
        w, h = _shape(rng, 160, 1920)
        return {"path": path, "width": w, "height": h, "double": rng.random() < 0.5, "max_iter": 100000,
                "span_log10": -round(rng.uniform(20, 220), 3)}
    if path == "batch":
        return {"path": "batch", "viewports": rng.randint(2, 16), "side_min": 96, "side_max": 768, "iter_min": 500,
                "iter_max": 20000, "rounded": rng.random() < 0.4, "specs": rng.randrange(1000)}
    if path == "newton":
        w, h = _shape(rng, 96, 1920)
        return {"path": "quality", "width": w, "height": h, "double": False, "arith": "parity",
                "max_iter": int(_log(rng, 50, 200)), "max_ss": float(rng.choice([1, 2, 4])), "view": "origin",
                "span": _log(rng, 1.0, 4.0),
                "fractal": rng.choice(["newton wired", "newton generic", "newton colored by iterations"])}
    w, h = _shape(rng, 320, 1280)
    return {"path": "serve", "sessions": rng.randint(1, 8), "frames": rng.randint(2, 6), "width": w, "height": h,
            "max_iter": int(_log(rng, 300, 2000)), "max_ss": float(rng.choice([1, 2]))}


# ---- views ---------------------------------------------------------------------

def _centre(case, seed):
    """The view's centre, moved by the seed: a few columns of a view of the whole set, up to an eighth of the span
    elsewhere."""
    r = random.Random(int(seed) * 7919 + 17)
    view = case["view"]
    if view in ("whole", "origin"):
        cx, cy, f = (-0.5 if view == "whole" else 0.0), 0.0, 0.01
    elif view == "seahorse":
        (cx, cy), f = SEAHORSE, 0.125
    else:
        (cx, cy), f = BOUNDARY[int(view[1:])], 0.125
    return cx + r.uniform(-f, f) * case["span"], cy + r.uniform(-f, f) * case["span"]


def _rect(centre, span, w, h):
    hw, hh = 0.5 * span, 0.5 * span * h / w
    return (centre[0] - hw, centre[1] - hh, centre[0] + hw, centre[1] + hh)


def _dev_palette(host):
    return torch.from_numpy(host.view(np.int32)).cuda()


def _records(w, h):
    """A pitched buffer of 16-byte pixel records, as cudaMallocPitch lays it out."""
    pitch = (16 * w + 511) // 512 * 512
    return torch.zeros((h, pitch // 4), dtype=torch.int32, device="cuda"), pitch


def _image(w, h):
    pitch = (4 * w + 511) // 512 * 512
    return torch.zeros((h, pitch // 4), dtype=torch.int32, device="cuda"), pitch


# ---- prepare -------------------------------------------------------------------

def prepare(case, seed):
    torch.zeros(1, device="cuda")
    return {"frame": _prepare_frame, "quality": _prepare_quality, "fast": _prepare_fast, "perturb": _prepare_perturb,
            "deep_step": _prepare_perturb, "batch": _prepare_batch, "serve": _prepare_serve}[case["path"]](case, seed)


def _prepare_frame(case, seed):
    w, h, n = case["width"], case["height"], case["width"] * case["height"]
    cx, cy = _centre(case, seed)
    jitter = case["spp"] > 1
    desc = cg.FrameDesc(width=w, height=h, max_iterations=case["max_iter"], samples_per_pixel=case["spp"],
                        sample_mode=cg.SAMPLES_JITTER if jitter else cg.SAMPLES_CENTER,
                        tier=cg.TIER_F64 if case["double"] else cg.TIER_F32,
                        arith=cg.ARITH_PARITY if case["arith"] == "parity" else cg.ARITH_FMA,
                        fractal=cg.JULIA if case["fractal"] == "julia" else cg.MANDELBROT, seed=1000 + int(seed),
                        center_x=cx, center_y=cy, pixel_size=case["span"] / w, julia_cx=JULIA_C[0],
                        julia_cy=JULIA_C[1])
    total = torch.zeros(1, dtype=torch.int64, device="cuda")
    if case["out"] == "rgba":
        pal = _dev_palette(seeded_palette(256, seed=int(seed) % (1 << 31)))
        rgba = torch.zeros((h, w), dtype=torch.int32, device="cuda")
        out = cg.FrameOut(rgba=rgba.data_ptr(), palette=pal.data_ptr(), palette_len=256, interior_rgba=BLACK,
                          total_iterations=total.data_ptr())
        bufs = {"rgba": rgba, "total": total}
    else:
        counts = torch.zeros(n * case["spp"], dtype=torch.int32, device="cuda")
        smooth = torch.zeros(n * case["spp"], dtype=torch.float32, device="cuda")
        out = cg.FrameOut(counts=counts.data_ptr(), smooth=smooth.data_ptr(), total_iterations=total.data_ptr())
        bufs, pal = {"counts": counts, "smooth": smooth, "total": total}, None
    return {"path": "frame", "desc": desc, "out": out, "bufs": bufs, "pal": pal, "total": total}


def _module(case):
    m = cg.Module(case["fractal"])
    if case["fractal"] == "julia":
        m.set_custom_params("%r;%r" % JULIA_C)
    return m


def _arith(case):
    return cg.ARITH_CONTRACTED if case["arith"] == "contracted" else cg.ARITH_PARITY


def _prepare_quality(case, seed):
    w, h = case["width"], case["height"]
    out, pitch = _records(w, h)
    rgba, rpitch = _image(w, h)
    pal = default_palette()
    return {"path": "quality", "module": _module(case), "out": out, "pitch": pitch, "rgba": rgba, "rpitch": rpitch,
            "pal": _dev_palette(pal), "pal_len": len(pal), "w": w, "h": h,
            "rect": _rect(_centre(case, seed), case["span"], w, h), "max_iter": case["max_iter"],
            "max_ss": case["max_ss"], "double": case["double"], "arith": _arith(case)}


def _prepare_fast(case, seed):
    w, h = case["width"], case["height"]
    centre = _centre(case, seed)
    rect, old = _rect(centre, case["span"], w, h), _rect(centre, case["span"] * case["zoom"], w, h)
    m = _module(case)
    prev, pitch = _records(w, h)
    out, _ = _records(w, h)
    rgba, rpitch = _image(w, h)
    pal = default_palette()
    arith = _arith(case)
    m.render_main(prev.data_ptr(), pitch, w, h, old, case["max_iter"], 1.0, 0, arith=arith)
    flags = cg.FLAG_ADAPTIVE_SS | cg.FLAG_SAMPLE_REUSE
    if case["zoom"] != 1.0:
        flags |= cg.FLAG_IS_ZOOMING | (cg.FLAG_ZOOMING_IN if case["zoom"] > 1.0 else 0)
    if case["foveation"]:
        flags |= cg.FLAG_FOVEATION
    return {"path": "fast", "module": m, "prev": prev, "out": out, "pitch": pitch, "rgba": rgba, "rpitch": rpitch,
            "pal": _dev_palette(pal), "pal_len": len(pal), "w": w, "h": h, "rect": rect, "old": old,
            "max_iter": case["max_iter"], "max_ss": case["max_ss"], "flags": flags, "arith": arith}


def _deep_offset(case, seed):
    r = random.Random(int(seed) * 104729 + 5)
    span = 10.0 ** case["span_log10"]
    return r.uniform(-0.1, 0.1) * span, r.uniform(-0.1, 0.1) * span


def _prepare_perturb(case, seed):
    w, h = case["width"], case["height"]
    d = deep_zoom_centre()
    bits = int(math.ceil((-case["span_log10"] * math.log2(10) + 400) / 64.0)) * 64
    ox, oy = _deep_offset(case, seed)
    desc = cg.FrameDesc(width=w, height=h, max_iterations=case["max_iter"], samples_per_pixel=1,
                        sample_mode=cg.SAMPLES_CENTER, fractal=cg.MANDELBROT, seed=0, center_x=ox, center_y=oy,
                        tier=cg.TIER_PERTURB_F64 if case["double"] else cg.TIER_PERTURB_F32,
                        pixel_size=10.0 ** case["span_log10"] / w)
    total = torch.zeros(1, dtype=torch.int64, device="cuda")
    if case["path"] == "perturb":
        counts = torch.zeros(w * h, dtype=torch.int32, device="cuda")
        smooth = torch.zeros(w * h, dtype=torch.float32, device="cuda")
        out = cg.FrameOut(counts=counts.data_ptr(), smooth=smooth.data_ptr(), total_iterations=total.data_ptr())
        orbit = cg.Orbit(d["center_x"], d["center_y"], bits, case["max_iter"])
        return {"path": "perturb", "orbit": orbit, "desc": desc, "out": out,
                "bufs": {"counts": counts, "smooth": smooth, "total": total}, "total": total}
    pal = _dev_palette(seeded_palette(256, seed=int(seed) % (1 << 31)))
    rgba = torch.zeros((h, w), dtype=torch.int32, device="cuda")
    out = cg.FrameOut(rgba=rgba.data_ptr(), palette=pal.data_ptr(), palette_len=256, interior_rgba=BLACK,
                      total_iterations=total.data_ptr())
    return {"path": "deep_step", "centre": (d["center_x"], d["center_y"], bits, case["max_iter"]), "desc": desc,
            "out": out, "pal": pal, "bufs": {"rgba": rgba, "total": total}, "total": total}


def _specs(case):
    """The batch's viewports: sides and iteration limits log-uniform in their ranges, spans from 1e-3 to 1e-12."""
    r = random.Random(case["specs"])
    out = []
    for k in range(case["viewports"]):
        side = int(round(_log(r, case["side_min"], case["side_max"]) / 8.0)) * 8
        out.append((side, 10.0 ** r.uniform(-12, -3), int(_log(r, case["iter_min"], case["iter_max"])),
                    BOUNDARY[r.randrange(8)]))
    return out


def _prepare_batch(case, seed):
    r = random.Random(int(seed) * 31337 + 3)
    pal = _dev_palette(seeded_palette(256, seed=int(seed) % (1 << 31)))
    vps, counts, images = [], [], []
    for k, (side, span, max_iter, (cx, cy)) in enumerate(_specs(case)):
        c = torch.zeros((side, side), dtype=torch.int32, device="cuda")
        im = torch.zeros((side, side), dtype=torch.int32, device="cuda")
        counts.append(c)
        images.append(im)
        vps.append(cg.Viewport(width=side, height=side, max_iterations=max_iter, samples_per_pixel=1,
                               sample_mode=cg.SAMPLES_CENTER,
                               tier=cg.TIER_F64_ROUNDED if case["rounded"] else cg.TIER_AUTO, seed=k,
                               center_x=cx + r.uniform(-0.1, 0.1) * span, center_y=cy + r.uniform(-0.1, 0.1) * span,
                               pixel_size=span / side, counts=c.data_ptr(), rgba=im.data_ptr()))
    b = cg.Batch(vps, palette_ptr=pal.data_ptr(), palette_len=256, interior_rgba=BLACK)
    return {"path": "batch", "batch": b, "pal": pal, "bufs": {"counts": counts, "rgba": images}}


_servers = {}


def _server():
    """The running server of this process: it outlives its sessions."""
    if "s" not in _servers:
        _servers["s"] = cg.Server(16 << 30, default_palette())
        atexit.register(lambda: _servers.pop("s").close())
    return _servers["s"]


def _prepare_serve(case, seed):
    r = random.Random(int(seed) * 65537 + 11)
    descs = []
    for k in range(case["sessions"]):
        tx, ty = BOUNDARY[k % 8]
        shallow = k % 2 == 0
        span = 3.0 * r.uniform(0.9, 1.1) if shallow else 1e-4 * r.uniform(0.9, 1.1)
        descs.append(cg.SessionDesc(width=case["width"], height=case["height"], max_iterations=case["max_iter"],
                                    max_super_sampling=case["max_ss"], flags=1 | 4 | 8, fractal=cg.MANDELBROT,
                                    arith=cg.ARITH_FMA, center_x=-0.5 if shallow else tx + 0.1 * span,
                                    center_y=0.0 if shallow else ty, span=span,
                                    target_x=tx, target_y=ty, zoom_per_frame=1.02))
    return {"path": "serve", "server": _server(), "descs": descs, "frames": case["frames"]}


# ---- run -----------------------------------------------------------------------

def run(state):
    return {"frame": _run_frame, "quality": _run_quality, "fast": _run_fast, "perturb": _run_perturb,
            "deep_step": _run_deep_step, "batch": _run_batch, "serve": _run_serve}[state["path"]](state)


def _run_frame(s):
    s["total"].zero_()
    cg.render_frame(s["desc"], s["out"], stream=torch.cuda.current_stream(), sync=False)
    return s["bufs"]


def _run_quality(s):
    w, h, st, m = s["w"], s["h"], torch.cuda.current_stream(), s["module"]
    m.render_main(s["out"].data_ptr(), s["pitch"], w, h, s["rect"], s["max_iter"], s["max_ss"], cg.FLAG_ADAPTIVE_SS,
                  double=s["double"], arith=s["arith"], stream=st)
    m.compose(s["out"].data_ptr(), s["pitch"], s["rgba"].data_ptr(), s["rpitch"], w, h, s["pal"].data_ptr(),
              s["pal_len"], s["max_ss"], stream=st)
    return {"records": s["out"][:, :4 * w], "rgba": s["rgba"][:, :w]}


def _run_fast(s):
    w, h, st, m = s["w"], s["h"], torch.cuda.current_stream(), s["module"]
    m.render_advanced(s["out"].data_ptr(), s["pitch"], w, h, s["rect"], s["max_iter"], s["max_ss"], s["flags"],
                      s["old"], s["prev"].data_ptr(), s["pitch"], (w // 2, h // 2), arith=s["arith"], stream=st)
    m.compose(s["out"].data_ptr(), s["pitch"], s["rgba"].data_ptr(), s["rpitch"], w, h, s["pal"].data_ptr(),
              s["pal_len"], s["max_ss"], stream=st)
    return {"records": s["out"][:, :4 * w], "rgba": s["rgba"][:, :w]}


def _run_perturb(s):
    s["total"].zero_()
    cg.render_frame_perturb(s["desc"], s["orbit"], s["out"], stream=torch.cuda.current_stream(), sync=False)
    return s["bufs"]


def _run_deep_step(s):
    s["total"].zero_()
    orbit = cg.Orbit(*s["centre"])
    cg.render_frame_perturb(s["desc"], orbit, s["out"], stream=torch.cuda.current_stream())
    orbit.close()
    return s["bufs"]


def _run_batch(s):
    s["batch"].launch(stream=torch.cuda.current_stream())
    return s["bufs"]


def _run_serve(s):
    srv = s["server"]
    sids = [srv.open(d) for d in s["descs"]]
    for _ in range(s["frames"]):
        for sid in sids:
            srv.submit(sid)
    srv.drain()
    out = [srv.read(sid) for sid in sids]
    for sid in sids:
        srv.close_session(sid)
    return {"images": [im for im, _ in out], "iterations": [int(n) for _, n in out]}


# ---- work ----------------------------------------------------------------------

# Steps that a sample cannot do without, on average: on a view of the whole set an escaping sample's (5 to 6) and a
# proof of the interior's; next to the boundary about seven tenths of the limit (half of the samples reach it and no
# state repeats); Newton about 12 steps of 40 operations.
STEP_FLOPS = 7


def _steps(case):
    if case["fractal"].startswith("newton"):
        return 12 * 40 / STEP_FLOPS
    if case["view"] in ("whole", "origin"):
        return 10.0
    if case["view"] == "seahorse":
        return 0.25 * case["max_iter"]
    return 0.69 * case["max_iter"]


def work(case):
    path = case["path"]
    if path == "frame":
        n = case["width"] * case["height"]
        out = 4 * n if case["out"] == "rgba" else 8 * n * case["spp"]
        return {"bytes": out, "flops": n * case["spp"] * _steps(case) * STEP_FLOPS}
    if path == "quality":
        n = case["width"] * case["height"]
        return {"bytes": 20 * n, "flops": n * 2 * _steps(case) * STEP_FLOPS}
    if path == "fast":
        n = case["width"] * case["height"]
        return {"bytes": 36 * n, "flops": n * 40.0}
    if path in ("perturb", "deep_step"):
        n = case["width"] * case["height"]
        # an orbit of at most 1000 entries; 9 blocks of 8 operations and 33 plain steps of 16 a sample
        return {"bytes": 8 * n if path == "perturb" else 4 * n, "flops": n * (9 * 16 + 33 * 28.0)}
    if path == "batch":
        pix = [(s * s, it) for s, _, it, _ in _specs(case)]
        return {"bytes": sum(8 * n for n, _ in pix), "flops": sum(n * 0.65 * it * STEP_FLOPS for n, it in pix)}
    n = case["sessions"] * case["frames"] * case["width"] * case["height"]
    return {"bytes": 36 * n, "flops": n * 0.1 * case["max_iter"] * STEP_FLOPS}


# ---- exact ---------------------------------------------------------------------
# Counts, records (votes and thresholds of the path's own arithmetic decide what they hold), images and totals are
# whole numbers and bytes: only the smooth counts have a value in 64 bits.

def exact(case, seed):
    if case["path"] == "frame" and case["out"] == "counts":
        if case["width"] * case["height"] * case["spp"] * case["max_iter"] > 4e9:
            return None
        return {"counts": None, "smooth": _exact_frame(case, seed), "total": None}
    if case["path"] == "perturb":
        return {"counts": None, "smooth": _exact_perturb(case, seed), "total": None}
    return None


def _smooth(i, r2, max_iter):
    nu = (i + 1).double() - torch.log2(0.5 * torch.log2(r2))
    return torch.where(i >= max_iter, torch.full_like(r2, float(max_iter)), nu)


def _mix64(z):
    with np.errstate(over="ignore"):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _exact_frame(case, seed):
    w, h, spp, max_iter = case["width"], case["height"], case["spp"], case["max_iter"]
    cx0, cy0 = _centre(case, seed)
    ps = case["span"] / w
    pix = np.repeat(np.arange(w * h, dtype=np.uint64), spp)
    if spp > 1:  # the frame's jitter: a counter-based hash of (seed, pixel, sample, axis)
        s = np.tile(np.arange(spp, dtype=np.uint64), w * h)
        bits, unit = (np.uint64(11), 2.0 ** -53) if case["double"] else (np.uint64(40), 2.0 ** -24)
        off = [(_mix64(np.uint64(1000 + int(seed)) ^ _mix64((pix << np.uint64(7)) | (s << np.uint64(1)) | np.uint64(a)))
                >> bits).astype(np.float64) * unit for a in (0, 1)]
    else:
        off = [0.5, 0.5]
    px, py = (pix % np.uint64(w)).astype(np.float64), (pix // np.uint64(w)).astype(np.float64)
    zx = torch.from_numpy((px + off[0] - 0.5 * w) * ps + cx0).cuda()
    zy = torch.from_numpy(-(py + off[1] - 0.5 * h) * ps + cy0).cuda()
    n = zx.numel()
    if case["fractal"] == "julia":
        cx, cy = torch.full_like(zx, JULIA_C[0]), torch.full_like(zy, JULIA_C[1])
    else:
        cx, cy, zx, zy = zx, zy, torch.zeros_like(zx), torch.zeros_like(zy)
    out_i = torch.full((n,), max_iter, dtype=torch.int64, device="cuda")
    out_r = torch.full((n,), 16.0, dtype=torch.float64, device="cuda")
    live = torch.arange(n, device="cuda")
    for i in range(max_iter):
        xx, yy = zx * zx, zy * zy
        r2 = xx + yy
        gone = ~(r2 < 4.0) & (out_i[live] == max_iter)
        out_i[live] = torch.where(gone, torch.full_like(live, i), out_i[live])
        out_r[live] = torch.where(gone, r2, out_r[live])
        zy = 2.0 * zx * zy + cy
        zx = xx - yy + cx
        if i % 32 == 31 or i < 8:
            keep = out_i[live] == max_iter
            live, zx, zy, cx, cy = live[keep], zx[keep], zy[keep], cx[keep], cy[keep]
            if live.numel() == 0:
                break
    return _smooth(out_i, out_r, max_iter)


@functools.lru_cache(maxsize=8)
def _orbit64(bits, max_iter):
    d = deep_zoom_centre()

    def fixed(text):
        neg, body = text.startswith("-"), text.lstrip("-")
        ip, frac = body.split(".")
        v = Fraction(int(ip)) + Fraction(int(frac, 16), 16 ** len(frac))
        k = int(v * (1 << bits))
        return -k if neg else k

    cx, cy = fixed(d["center_x"]), fixed(d["center_y"])
    x = y = 0
    zs = [(0.0, 0.0)]
    for _ in range(max_iter):
        x, y = ((x + y) * (x - y) >> bits) + cx, (2 * x * y >> bits) + cy
        fx, fy = x / (1 << bits), y / (1 << bits)
        zs.append((fx, fy))
        if not fx * fx + fy * fy < 4.0:
            break
    return zs


def _exact_perturb(case, seed):
    w, h, max_iter = case["width"], case["height"], case["max_iter"]
    bits = int(math.ceil((-case["span_log10"] * math.log2(10) + 400) / 64.0)) * 64
    zs = torch.tensor(_orbit64(bits, max_iter), dtype=torch.float64, device="cuda")
    last = len(zs) - 1
    ox, oy = _deep_offset(case, seed)
    ps = 10.0 ** case["span_log10"] / w
    pix = torch.arange(w * h, device="cuda")
    cx = ((pix % w).double() + 0.5 - 0.5 * w) * ps + ox
    cy = -((pix // w).double() + 0.5 - 0.5 * h) * ps + oy
    dx, dy = torch.zeros_like(cx), torch.zeros_like(cy)
    m = torch.zeros_like(pix)
    out_i = torch.full((w * h,), max_iter, dtype=torch.int64, device="cuda")
    out_r = torch.full((w * h,), 16.0, dtype=torch.float64, device="cuda")
    live = pix
    for i in range(1, min(max_iter, 20000) + 1):
        wx, wy = 2.0 * zs[m, 0] + dx, 2.0 * zs[m, 1] + dy
        dx, dy = wx * dx - wy * dy + cx, wx * dy + wy * dx + cy
        m = m + 1
        zx, zy = zs[m, 0] + dx, zs[m, 1] + dy
        r2 = zx * zx + zy * zy
        gone = ~(r2 < 4.0) if i < max_iter else torch.zeros_like(r2, dtype=torch.bool)
        if bool(gone.any()):
            out_i[live[gone]] = i
            out_r[live[gone]] = r2[gone]
        # rebase where z is smaller than its difference (compared in units that do not underflow) or the orbit ends
        scale = torch.maximum(dx.abs(), dy.abs()).clamp_min(1e-300)
        back = (m == last) | ((zx / scale) ** 2 + (zy / scale) ** 2 < (dx / scale) ** 2 + (dy / scale) ** 2)
        dx, dy, m = torch.where(back, zx, dx), torch.where(back, zy, dy), torch.where(back, torch.zeros_like(m), m)
        if bool(gone.any()):
            keep = ~gone
            live, dx, dy, cx, cy, m = live[keep], dx[keep], dy[keep], cx[keep], cy[keep], m[keep]
            if live.numel() == 0:
                break
    return _smooth(out_i, out_r, max_iter)
