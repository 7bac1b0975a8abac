"""What the performance of this framework is measured on.

A case is one pass of a user's program through a public entry point of the
Python package: a camera frame through `Pipeline.process`, the frames of many
cameras through `Batch.launch`, a converted image through
`Converter.convert`, the demo's view through `view_compose`. All inputs lie in
device memory, where a capture card, a decoder or the previous stage leaves
them. The serving loop queues the batch's launches and the C++ classes the
same C entry points, so the cases stand for them too.

The ranges (`draw` covers all of them, the listed cases are points of them):

* frames of 64x48 to 24 Mpixel (the largest listed one is 8192x6144), even and
  odd sizes, rows packed or padded to 64 bytes; 8-bit and 16-bit samples, MIPI
  RAW10 and RAW12; the four Bayer patterns; bilinear and Malvar-He-Cutler
  demosaic, with and without sharpening; manual, gray world and white patch
  white balance; no lens shading, one gain plane or four; every tone curve and
  output format; with and without histogram and statistics;
* batches of 2 to 24 such cameras (48 in the listed case);
* conversions between all twelve pixel formats of images of 64x48 to
  3840x2160, same-size, and resized by every mode with and without a
  letterbox or a crop.

Frames are smooth scenes with edges, vignetted, with photon and read noise.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("holoscan-zozo-modules_b200"))  # of the tree it is run in

import isp_b200  # noqa: E402
from isp_b200 import abi, cc, scene  # noqa: E402

PATTERNS = ("RGGB", "BGGR", "GRBG", "GBRG")
RAW_FORMATS = ("u8", "u16", "raw10", "raw12")
OUT_FORMATS = ("rgb8", "rgba8", "rgb16", "rgb32f")
BALANCES = ("manual", "gray_world", "white_patch")
DEMOSAICS = ("bilinear", "malvar")
TONES = ("srgb", "gamma", "linear", "lut")
MODES = ("nearest", "bilinear", "area")
CC_FORMATS = ("nv12", "nv16", "i420", "yuyv", "uyvy", "rgb8", "bgr8", "rgba8", "bgra8", "mono8", "mono16", "rgb16")
EXPOSURE = (10_000_000, 1.5)
CCM = (1.6, -0.3, -0.3, -0.3, 1.6, -0.3, -0.3, -0.3, 1.6)
WB_GAINS = (1.9, 1.0, 1.5)
LSC_SIZE = (17, 13)
# Colour at quad position (y & 1) * 2 + (x & 1): 0 red, 1 green, 2 blue; and the
# channel there: 0 R, 1 green in a red row, 2 green in a blue row, 3 B.
_COLOR = {"RGGB": (0, 1, 1, 2), "BGGR": (2, 1, 1, 0), "GRBG": (1, 0, 2, 1), "GBRG": (1, 2, 0, 1)}
_CHANNEL = {"RGGB": (0, 1, 2, 3), "BGGR": (3, 2, 1, 0), "GRBG": (1, 0, 3, 2), "GBRG": (2, 3, 0, 1)}


def _frame(name, width, height, raw, bits, pattern, **options):
    case = {"kind": "frame", "width": width, "height": height, "raw": raw, "bits": bits, "pattern": pattern,
            "black": 16.0 * 2.0 ** (bits - 8), "balance": "manual", "demosaic": "malvar", "sharpen": 0.0, "shading": 0,
            "tone": "srgb", "table": 0, "out": "rgb8", "histogram": False, "stats": False, "align": 1}
    case.update(options)
    if name:
        case["name"] = name
    return case


def _convert(name, width, height, source, destination, **options):
    case = {"kind": "convert", "width": width, "height": height, "source": source, "destination": destination,
            "out_width": width, "out_height": height, "mode": "nearest", "letterbox": False, "crop": False}
    case.update(options)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # A small machine-vision camera without statistics: latency and launches count.
        _frame("vga_u8", 640, 480, "u8", 8, "RGGB", demosaic="bilinear"),
        # A 1080p camera with manual white balance whose histogram drives exposure.
        _frame("hd_u16_histogram", 1920, 1080, "u16", 12, "RGGB", demosaic="bilinear", shading=4, histogram=True),
        # The full set of stages at 1080p, as the ISP's own benchmark runs them.
        _frame("hd_u16_full", 1920, 1080, "u16", 12, "GBRG", balance="gray_world", sharpen=0.5, shading=4,
               histogram=True, stats=True),
        # A size and rows that no alignment helps, into floats for a network or a measurement.
        _frame("ragged_u16_float", 1366, 768, "u16", 10, "GRBG", balance="white_patch", tone="gamma", out="rgb32f",
               stats=True),
        # A 4K sensor's packed frame through every stage: the framework's headline frame.
        _frame("uhd_raw10_full", 3840, 2160, "raw10", 10, "GRBG", balance="gray_world", sharpen=0.5, shading=4,
               tone="lut", table=1024, out="rgb16", histogram=True, stats=True),
        # The largest frame: a 50 Mpixel sensor for stills and inspection.
        _frame("50mp_raw12_full", 8192, 6144, "raw12", 12, "BGGR", balance="white_patch", sharpen=0.5, shading=4,
               tone="lut", table=4096, out="rgba8", histogram=True, stats=True),
        # A rig of 48 cameras of four kinds, one launch per pass.
        {"name": "batch_48", "kind": "batch", "vga": 16, "hd": 16, "uhd": 12, "large": 4, "mix": 2024},
        # The ISP's 4K output for a video encoder.
        _convert("uhd_rgb8_nv12", 3840, 2160, "rgb8", "nv12"),
        # A decoded 1080p video frame for display.
        _convert("hd_nv12_rgb8", 1920, 1080, "nv12", "rgb8"),
        # A decoded frame scaled for a preview.
        _convert("hd_nv12_rgba8_720p", 1920, 1080, "nv12", "rgba8", out_width=1280, out_height=720, mode="bilinear"),
        # A decoded 4K frame reduced without aliasing for inference.
        _convert("uhd_nv12_rgb8_area", 3840, 2160, "nv12", "rgb8", out_width=1280, out_height=720, mode="area"),
        # The demo's raw and processed pictures side by side.
        {"name": "view_uhd_raw10", "kind": "view", "width": 3840, "height": 2160, "raw": "raw10", "bits": 10,
         "pattern": "GRBG", "black": 64.0, "align": 1},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _draw_size(rng, low, high):
    """Width and height of `low` to `high` pixels, over the logarithm; one in three odd somewhere."""
    pixels = _log_int(rng, low, high)
    aspect = rng.choice((4 / 3, 16 / 9, 3 / 2, 1.0, 9 / 16, 2.39))
    w = max(64, min(8192, int(math.sqrt(pixels * aspect))))
    h = max(48, min(8192, int(pixels / w)))
    odd = rng.randrange(6)
    w = w | 1 if odd in (0, 2) else (w + 7) // 8 * 8 if odd in (3, 4) else w & ~1
    h = h | 1 if odd in (1, 2) else h & ~1
    return w, h


def draw(rng):
    kind = rng.choice(("frame",) * 6 + ("convert",) * 4 + ("batch", "view"))
    raw = rng.choice(RAW_FORMATS)
    bits = {"u8": 8, "u16": rng.choice((10, 12, 14, 16)), "raw10": 10, "raw12": 12}[raw]
    pattern = rng.choice(PATTERNS)
    align = rng.choice((1, 64))
    if kind == "frame":
        w, h = _draw_size(rng, 64 * 48, 24_000_000)
        tone = rng.choice(TONES)
        return _frame(None, w, h, raw, bits, pattern, balance=rng.choice(BALANCES), demosaic=rng.choice(DEMOSAICS),
                      sharpen=rng.choice((0.0, 0.5, 1.25)), shading=rng.choice((0, 1, 4)), tone=tone,
                      table=rng.choice((256, 1024, 4096)) if tone == "lut" else 0, out=rng.choice(OUT_FORMATS),
                      histogram=rng.random() < 0.6, stats=rng.random() < 0.6, align=align)
    if kind == "batch":
        return {"kind": "batch", "vga": rng.randrange(1, 9), "hd": rng.randrange(1, 9), "uhd": rng.randrange(0, 6),
                "large": rng.randrange(0, 3), "mix": rng.randrange(1, 10_000)}
    if kind == "view":
        w, h = _draw_size(rng, 320 * 240, 12_000_000)
        return {"kind": "view", "width": w, "height": h, "raw": raw, "bits": bits, "pattern": pattern,
                "black": 16.0 * 2.0 ** (bits - 8), "align": align}
    w, h = _draw_size(rng, 64 * 48, 3840 * 2160)
    w, h = min(w, 3840), min(h, 3840)
    source, destination = rng.choice(CC_FORMATS), rng.choice(CC_FORMATS)
    packed_pairs = ("yuyv", "uyvy")  # whole pixel pairs only
    if rng.random() < 0.5:
        return _convert(None, w & ~1 if source in packed_pairs or destination in packed_pairs else w, h, source,
                        destination)
    scale = math.exp(rng.uniform(math.log(0.2), math.log(1.5)))
    w = w & ~1 if source in packed_pairs else w
    ow, oh = max(16, int(w * scale)), max(16, int(h * scale * rng.choice((1.0, 0.8, 1.2))))
    ow = ow & ~1 if destination in packed_pairs else ow
    return _convert(None, w, h, source, destination, out_width=ow, out_height=oh, mode=rng.choice(MODES),
                    letterbox=rng.random() < 0.4, crop=rng.random() < 0.3)


# ---- Inputs ----------------------------------------------------------------

_stream = None


def _launch_stream():
    """The stream that a program gives its frames to, one for all."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


def _scene(width, height, seed):
    """Linear RGB [3, H, W] in [0, 1]: a gradient, blobs and rectangles."""
    rng = np.random.default_rng(np.random.PCG64(seed))
    ys = torch.arange(height, dtype=torch.float32, device="cuda")[:, None]
    xs = torch.arange(width, dtype=torch.float32, device="cuda")[None, :]
    img = torch.empty((3, height, width), dtype=torch.float32, device="cuda")
    for c in range(3):
        base, gx, gy = rng.uniform(0.05, 0.35), rng.uniform(-0.25, 0.25) / width, rng.uniform(-0.25, 0.25) / height
        img[c] = base + gx * xs + gy * ys
    for _ in range(6):
        cx, cy, sigma = rng.uniform(0, width), rng.uniform(0, height), rng.uniform(0.03, 0.15) * max(width, height)
        blob = torch.exp((ys - cy) ** 2 / (-2 * sigma * sigma)) * torch.exp((xs - cx) ** 2 / (-2 * sigma * sigma))
        for c in range(3):
            img[c] += float(rng.uniform(0.05, 0.5)) * blob
    for _ in range(48):
        w, h = int(rng.uniform(0.02, 0.2) * width) + 1, int(rng.uniform(0.02, 0.2) * height) + 1
        x0, y0 = int(rng.uniform(0, width - w + 1)), int(rng.uniform(0, height - h + 1))
        for c in range(3):
            img[c, y0:y0 + h, x0:x0 + w] = float(rng.uniform(0.0, 1.0))
    return img.clamp_(0.0, 1.0)


def _counts(case, seed):
    """Raw counts [H, W] int32 of the mosaicked, vignetted, noisy scene."""
    w, h, bits = case["width"], case["height"], case["bits"]
    img = _scene(w, h, seed)
    ys = torch.arange(h, dtype=torch.float32, device="cuda")[:, None] - (h - 1) / 2
    xs = torch.arange(w, dtype=torch.float32, device="cuda")[None, :] - (w - 1) / 2
    tan2 = math.tan(math.acos(0.5 ** 0.25)) ** 2
    vignette = (1 + tan2 * (ys * ys + xs * xs) / (((w - 1) ** 2 + (h - 1) ** 2) / 4)) ** -2  # cos^4
    mosaic = torch.empty((h, w), dtype=torch.float32, device="cuda")
    for q, c in enumerate(_COLOR[case["pattern"]]):
        mosaic[q >> 1::2, q & 1::2] = img[c, q >> 1::2, q & 1::2]
    full = (1 << bits) - 1
    dn = mosaic * vignette * (full - case["black"])
    noise = torch.randn((h, w), generator=torch.Generator("cuda").manual_seed(seed), device="cuda")
    dn += noise * torch.sqrt(0.5 * dn + 9.0 * 4.0 ** (bits - 12))
    return (dn + case["black"]).round_().clamp_(0, full).to(torch.int32)


def _pack(counts, raw, align):
    """Rows of `counts` in the sensor's format, [H, pitch] bytes."""
    h, w = counts.shape
    if raw == "u8":
        rows = counts.to(torch.uint8)
    elif raw == "u16":
        rows = torch.stack((counts & 255, counts >> 8), dim=2).to(torch.uint8).reshape(h, 2 * w)
    else:
        per = 4 if raw == "raw10" else 2
        c = torch.nn.functional.pad(counts, (0, -w % per)).reshape(h, -1, per)
        low = c & (3 if raw == "raw10" else 15)
        last = sum(low[:, :, k] << (8 // per * k) for k in range(per))
        rows = torch.cat((c >> (2 if raw == "raw10" else 4), last[:, :, None]), dim=2).to(torch.uint8).reshape(h, -1)
    return torch.nn.functional.pad(rows, (0, -rows.shape[1] % align)).contiguous()


def _raw_view(case, rows):
    return abi.RawViewC(rows.data_ptr(), case["width"], case["height"], rows.shape[1], RAW_FORMATS.index(case["raw"]),
                        case["bits"], PATTERNS.index(case["pattern"]))


def _shading(width, height, channels):
    """Gains [13, 17, channels] that undo the vignette, the colours a little apart."""
    gw, gh = LSC_SIZE
    gains = 1.0 / scene.vignette(width, height, np.arange(gw) * (width - 1) / (gw - 1),
                                 np.arange(gh) * (height - 1) / (gh - 1))
    tint = np.array((1.02, 1.0, 1.0, 0.98))[:channels] if channels == 4 else np.ones(1)
    return np.maximum(gains[:, :, None] * tint, 1.0).astype(np.float32)


def _table(case):
    return scene.srgb_table(case["table"]) if case["table"] <= 1024 else scene.filmic_table(case["table"])


def _params(case):
    shading = None
    if case["shading"]:
        g = _shading(case["width"], case["height"], case["shading"])
        shading = abi.LensShading(LSC_SIZE[0], LSC_SIZE[1], case["shading"], np.ascontiguousarray(g.ravel()))
    return abi.IspParams(black_level=case["black"], lens_shading=shading,
                         white_balance=BALANCES.index(case["balance"]), wb_gains=WB_GAINS,
                         white_patch_percentile=0.995, demosaic=DEMOSAICS.index(case["demosaic"]), ccm=CCM,
                         tone_curve=TONES.index(case["tone"]), lut=_table(case) if case["tone"] == "lut" else None,
                         sharpen=case["sharpen"])


def _image(case):
    """The output rows, packed: [H, W, channels] of the format's type."""
    fmt = OUT_FORMATS.index(case["out"])
    # 16-bit codes as int16, the type of that size that torch computes with: the same bits.
    kind = {"rgb16": torch.int16, "rgb32f": torch.float32}.get(case["out"], torch.uint8)
    return torch.empty((case["height"], case["width"], abi.output_channels(fmt)), dtype=kind, device="cuda")


def _cameras(case):
    """The batch's cameras, each a frame case: settings by the mix's seed, sizes as in the mixed workload."""
    rng = np.random.default_rng(np.random.PCG64(case["mix"]))
    kinds = (("vga", 640, 480, "u8", 8, "RGGB"), ("hd", 1920, 1080, "u16", 12, "GBRG"),
             ("uhd", 3840, 2160, "raw10", 10, "GRBG"), ("large", 4096, 3072, "u16", 16, "BGGR"))
    cameras = []
    for key, w, h, raw, bits, pattern in kinds:
        for _ in range(case[key]):
            cameras.append(_frame(None, w, h, raw, bits, pattern, balance=BALANCES[int(rng.integers(3))],
                                  demosaic=DEMOSAICS[int(rng.integers(2))], shading=4, tone="lut", table=1024,
                                  histogram=True, stats=True))
    return cameras


def _cc_planes(fmt, width, height, seed):
    """A packed image of the scene in one of the converter's formats, as bytes."""
    rgb = (_scene(width, height, seed) ** (1 / 2.2) * 255.0)
    noise = torch.randn((height, width), generator=torch.Generator("cuda").manual_seed(seed), device="cuda")
    rgb = (rgb + 2.0 * noise).clamp_(0.0, 255.0)
    y = 0.299 * rgb[0] + 0.587 * rgb[1] + 0.114 * rgb[2]
    u8 = lambda v: v.round().clamp(0, 255).to(torch.uint8)  # noqa: E731
    if fmt in ("rgb8", "bgr8", "rgba8", "bgra8"):
        c = [u8(rgb[k]) for k in ((0, 1, 2) if fmt.startswith("rgb") else (2, 1, 0))]
        if len(fmt) == 5:
            c.append(u8(128.0 + 20.0 * noise))
        return torch.stack(c, dim=2).reshape(-1)
    if fmt in ("mono8", "mono16", "rgb16"):
        if fmt == "mono8":
            return u8(y).reshape(-1)
        v = ((y[None] if fmt == "mono16" else rgb) * 257.0).round().clamp(0, 65535).to(torch.int32).permute(1, 2, 0)
        return torch.stack((v & 255, v >> 8), dim=3).to(torch.uint8).reshape(-1)
    down = 2 if fmt in ("nv12", "i420") else 1
    even = torch.nn.functional.pad(torch.stack((rgb[2] - y, rgb[0] - y)), (0, -width % 2, 0, -height % down),
                                   mode="replicate") if width % 2 or height % down else torch.stack((rgb[2] - y, rgb[0] - y))
    chroma = torch.nn.functional.avg_pool2d(even[None], (down, 2))[0]
    cb, cr = u8(128.0 + 0.5 * chroma[0]), u8(128.0 + 0.6 * chroma[1])
    luma = u8(16.0 + y * (219.0 / 255.0))
    if fmt in ("nv12", "nv16"):
        return torch.cat((luma.reshape(-1), torch.stack((cb, cr), dim=2).reshape(-1)))
    if fmt == "i420":
        return torch.cat((luma.reshape(-1), cb.reshape(-1), cr.reshape(-1)))
    pairs = torch.nn.functional.pad(luma, (0, -width % 2)).reshape(height, -1, 2)
    order = (pairs[:, :, 0], cb, pairs[:, :, 1], cr) if fmt == "yuyv" else (cb, pairs[:, :, 0], cr, pairs[:, :, 1])
    rows = torch.stack(order, dim=2).reshape(height, -1)
    row_bytes = cc.plane_size(CC_FORMATS.index(fmt), width, height, 0)[0]
    return rows[:, :row_bytes].reshape(-1)


def _crop(case):
    """The central three quarters, at even coordinates."""
    w, h = case["width"], case["height"]
    return (w // 8 & ~1, h // 8 & ~1, max(2, w * 3 // 4 & ~1), max(2, h * 3 // 4 & ~1)) if case["crop"] else None


def _prepare_frame(case, seed):
    rows = _pack(_counts(case, seed), case["raw"], case["align"])
    image = _image(case)
    out = {"image": image}
    if case["histogram"]:
        out["histogram"] = torch.empty((abi.HISTOGRAM_CHANNELS, abi.HISTOGRAM_BINS), dtype=torch.int32, device="cuda")
    if case["stats"]:
        out["stats"] = torch.empty(abi.STATS_SIZE, dtype=torch.float32, device="cuda")
    return {"case": case, "pipe": isp_b200.Pipeline(_params(case)), "rows": rows, "out": out,
            "raw_view": _raw_view(case, rows),
            "rgb_view": abi.RgbViewC(image.data_ptr(), image.stride(0) * image.element_size(), OUT_FORMATS.index(case["out"]))}


def _prepare_batch(case, seed):
    cameras = _cameras(case)
    images = torch.empty(sum(c["width"] * c["height"] * 3 for c in cameras), dtype=torch.uint8, device="cuda")
    histograms = torch.empty((len(cameras), 4, 256), dtype=torch.int32, device="cuda")
    stats = torch.empty((len(cameras), abi.STATS_SIZE), dtype=torch.float32, device="cuda")
    batch, kept, at = isp_b200.Batch(len(cameras)), [], 0
    for i, c in enumerate(cameras):
        rows = _pack(_counts(c, seed * 1000 + i), c["raw"], c["align"])
        pipe = isp_b200.Pipeline(_params(c))
        batch.add(pipe, _raw_view(c, rows), abi.RgbViewC(images.data_ptr() + at, c["width"] * 3, abi.RGB8),
                  histograms[i].data_ptr(), stats[i].data_ptr(), EXPOSURE)
        kept.append((rows, pipe))
        at += c["width"] * c["height"] * 3
    return {"case": case, "batch": batch, "kept": kept,
            "out": {"images": images, "histograms": histograms, "stats": stats}}


def _prepare_convert(case, seed):
    src = _cc_planes(case["source"], case["width"], case["height"], seed)
    sf, df = CC_FORMATS.index(case["source"]), CC_FORMATS.index(case["destination"])
    dst = torch.empty(cc.packed_size(df, case["out_width"], case["out_height"]), dtype=torch.uint8, device="cuda")
    return {"case": case, "converter": cc.Converter(), "src": src, "out": {"image": dst},
            "source": cc.packed_view(src.data_ptr(), sf, case["width"], case["height"]),
            "destination": cc.packed_view(dst.data_ptr(), df, case["out_width"], case["out_height"]),
            "params": cc.params(cc.BT709, mode=MODES.index(case["mode"]), crop=_crop(case),
                                letterbox=case["letterbox"], fill_rgb=(114, 114, 114))}


def _prepare_view(case, seed):
    rows = _pack(_counts(case, seed), case["raw"], case["align"])
    rgb = (_scene(case["width"], case["height"], seed + 1).permute(1, 2, 0) * 255.0).to(torch.uint8).contiguous()
    view = torch.empty((case["height"], 2 * case["width"], 3), dtype=torch.uint8, device="cuda")
    return {"case": case, "rows": rows, "rgb": rgb, "out": {"view": view}, "raw_view": _raw_view(case, rows)}


def prepare(case, seed):
    make = {"frame": _prepare_frame, "batch": _prepare_batch, "convert": _prepare_convert, "view": _prepare_view}
    state = make[case["kind"]](case, seed)
    state["stream"] = _launch_stream()
    torch.cuda.synchronize()
    return state


def run(state):
    case, out = state["case"], state["out"]
    if case["kind"] == "frame":
        state["pipe"].process(state["raw_view"], state["rgb_view"],
                              out["histogram"].data_ptr() if "histogram" in out else 0,
                              out["stats"].data_ptr() if "stats" in out else 0, EXPOSURE, state["stream"])
    elif case["kind"] == "batch":
        state["batch"].launch(state["stream"], True)
    elif case["kind"] == "convert":
        state["converter"].convert(state["source"], state["destination"], state["params"], state["stream"])
    else:
        view = out["view"]
        isp_b200.view_compose(state["raw_view"], case["black"], state["rgb"].data_ptr(), 3 * case["width"],
                              view.data_ptr(), 6 * case["width"], state["stream"])
    return out


def work(case):
    """Inputs read once, outputs written once; the operations of the definitions, counted per pixel."""
    if case["kind"] == "batch":
        parts = [work(c) for c in _cameras(case)]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    if case["kind"] == "convert":
        sf, df = CC_FORMATS.index(case["source"]), CC_FORMATS.index(case["destination"])
        source = cc.packed_size(sf, case["width"], case["height"])
        crop = _crop(case)
        if crop:
            source = source * crop[2] * crop[3] // (case["width"] * case["height"])
        outputs = case["out_width"] * case["out_height"]
        if case["mode"] == "nearest" and outputs * 4 < case["width"] * case["height"]:
            source = min(source, outputs * 6)
        taps = {"nearest": 0, "bilinear": 32, "area": 8 * max(1.0, case["width"] * case["height"] / outputs)}
        resized = (case["out_width"], case["out_height"]) != (case["width"], case["height"])
        return {"bytes": source + cc.packed_size(df, case["out_width"], case["out_height"]),
                "flops": outputs * (24 + (taps[case["mode"]] if resized else 0))}
    pixels = case["width"] * case["height"]
    raw = abi.raw_row_bytes(RAW_FORMATS.index(case["raw"]), case["width"]) * case["height"]
    if case["kind"] == "view":
        return {"bytes": raw + 9 * pixels, "flops": 8 * pixels}
    fmt = OUT_FORMATS.index(case["out"])
    ops = 4 + (5 if case["shading"] else 0) + (20 if case["demosaic"] == "malvar" else 6) + 15 + 9 + 6
    ops += (45 if case["sharpen"] > 0 else 0) + (6 if case["stats"] else 0) + (8 if case["histogram"] else 0)
    ops += 6 if case["balance"] != "manual" else 0
    return {"bytes": raw + pixels * abi.output_channels(fmt) * abi.output_channel_bytes(fmt)
            + (4096 if case["histogram"] else 0) + (48 if case["stats"] else 0), "flops": ops * pixels}


# ---- The same in 64 bits ---------------------------------------------------


def _exact_linear(case, counts):
    """Linear samples [H, W] before white balance."""
    h, w = counts.shape
    full = float((1 << case["bits"]) - 1)
    v = ((counts.double() - case["black"]) / (full - case["black"])).clamp_min_(0.0)
    if case["shading"]:
        grid = torch.from_numpy(_shading(w, h, case["shading"])).double().cuda()
        gw, gh = LSC_SIZE
        fx = torch.arange(w, device="cuda", dtype=torch.float64) * ((gw - 1) / (w - 1))
        fy = torch.arange(h, device="cuda", dtype=torch.float64) * ((gh - 1) / (h - 1))
        ix, iy = fx.long().clamp_max(gw - 2), fy.long().clamp_max(gh - 2)
        tx, ty = fx - ix, fy - iy
        for q in range(4):
            plane = grid[:, :, _CHANNEL[case["pattern"]][q] if case["shading"] == 4 else 0]
            xs, ys = slice(q & 1, None, 2), slice(q >> 1, None, 2)
            across = plane[:, ix[xs]] + (plane[:, ix[xs] + 1] - plane[:, ix[xs]]) * tx[xs]
            top, bottom = across[iy[ys]], across[iy[ys] + 1]
            v[ys, xs] *= top + (bottom - top) * ty[ys, None]
    return v


def _exact_gains(case, counts, linear):
    """The white balance that the frame is processed with."""
    if case["balance"] == "manual":
        return list(WB_GAINS)
    h, w = counts.shape
    qh, qw = h // 2 * 2, w // 2 * 2
    quad = [counts[q >> 1:qh:2, q & 1:qw:2] for q in range(4)]
    ok = torch.stack([q < (1 << case["bits"]) - 1 for q in quad]).all(dim=0)
    values = [[], [], []]
    for q, c in enumerate(_COLOR[case["pattern"]]):
        values[c].append(linear[q >> 1:qh:2, q & 1:qw:2][ok].clamp_max(4.0))
    levels = []
    for c in range(3):
        if case["balance"] == "gray_world":
            levels.append(float(sum(v.sum() for v in values[c])) / max(1, sum(v.numel() for v in values[c])))
            continue
        bins = sum(torch.bincount((v * 1024.0).long().clamp_max(1023), minlength=1024) for v in values[c]).cpu().numpy()
        target, below = 0.995 * float(bins.sum()), np.cumsum(bins)
        b = int(np.argmax((below >= target) & (bins > 0)))
        levels.append((b + (target - float(below[b] - bins[b])) / float(bins[b])) / 1024.0)
    if min(levels) <= 0.0:
        return list(WB_GAINS)
    return [min(max(levels[1] / levels[c], 0.0625), 16.0) if c != 1 else 1.0 for c in range(3)]


def _exact_demosaic(case, mosaic):
    """RGB [3, H + 2, W + 2] of every pixel and its one-pixel ring."""
    h, w = mosaic.shape
    m = torch.nn.functional.pad(mosaic[None, None], (4, 4, 4, 4), mode="reflect")[0, 0]
    rgb = torch.empty((3, h + 2, w + 2), dtype=torch.float64, device="cuda")
    for q in range(4):
        # Ring rows start at image row -1: quad row q >> 1 begins at ring row (q >> 1) ^ 1.
        y0, x0 = (q >> 1) ^ 1, (q & 1) ^ 1
        n = lambda dy, dx: m[y0 + 3 + dy:y0 + 3 + dy + h + 2 - y0:2, x0 + 3 + dx:x0 + 3 + dx + w + 2 - x0:2]  # noqa: E731
        c, at = n(0, 0), rgb[:, y0::2, x0::2]
        channel = _CHANNEL[case["pattern"]][q]
        vertical, horizontal = n(-1, 0) + n(1, 0), n(0, -1) + n(0, 1)
        corners = n(-1, -1) + n(-1, 1) + n(1, -1) + n(1, 1)
        if case["demosaic"] == "malvar":
            v2, h2 = n(-2, 0) + n(2, 0), n(0, -2) + n(0, 2)
            green = ((4 * c + 2 * (vertical + horizontal) - v2 - h2) / 8).clamp(0, 1)
            diagonal = ((6 * c + 2 * corners - 1.5 * (v2 + h2)) / 8).clamp(0, 1)
            across = ((5 * c + 4 * horizontal - h2 - corners + 0.5 * v2) / 8).clamp(0, 1)
            down = ((5 * c + 4 * vertical - v2 - corners + 0.5 * h2) / 8).clamp(0, 1)
        else:
            green, diagonal, across, down = (vertical + horizontal) / 4, corners / 4, horizontal / 2, vertical / 2
        if channel in (0, 3):
            at[1] = green
            at[channel // 3 * 2], at[2 - channel // 3 * 2] = c, diagonal
        else:
            at[1] = c
            at[(channel - 1) * 2], at[2 - (channel - 1) * 2] = across, down
    return rgb


def _exact_frame(case, seed):
    counts = _counts(case, seed)
    linear = _exact_linear(case, counts)
    gains = _exact_gains(case, counts, linear)
    for q, c in enumerate(_COLOR[case["pattern"]]):
        linear[q >> 1::2, q & 1::2] *= float(np.float32(gains[c])) if case["balance"] == "manual" else gains[c]
    rgb = _exact_demosaic(case, linear.clamp_max_(1.0))
    del linear
    if case["sharpen"] > 0:
        for c in range(3):
            x = rgb[c]
            blur = (4 * x[1:-1, 1:-1] + 2 * (x[:-2, 1:-1] + x[2:, 1:-1] + x[1:-1, :-2] + x[1:-1, 2:])
                    + x[:-2, :-2] + x[:-2, 2:] + x[2:, :-2] + x[2:, 2:]) / 16
            x[1:-1, 1:-1] = (x[1:-1, 1:-1] + case["sharpen"] * (x[1:-1, 1:-1] - blur)).clamp(0, 1)
    rgb = rgb[:, 1:-1, 1:-1]
    ccm = np.array(CCM, np.float32).astype(np.float64).reshape(3, 3)
    lit = [sum(float(ccm[k, j]) * rgb[j] for j in range(3)).clamp(0, 1) for k in range(3)]
    del rgb
    image = None
    if case["out"] == "rgb32f":
        if case["tone"] == "lut":
            lut = _table(case).astype(np.float64)
        else:
            x = np.arange(4097) / 4096.0
            lut = {"linear": x, "gamma": x ** (1.0 / float(np.float32(2.2))),
                   "srgb": np.where(x <= 0.0031308, 12.92 * x, 1.055 * x ** (1 / 2.4) - 0.055)}[case["tone"]]
        lut = torch.from_numpy(np.append(lut, lut[-1])).cuda()
        image = torch.empty((*lit[0].shape, 3), dtype=torch.float64, device="cuda")
        for k in range(3):
            f = lit[k] * (lut.numel() - 2)
            i = f.long()
            image[:, :, k] = lut[i] + (f - i) * (lut[i + 1] - lut[i])
    stats = None
    if case["stats"]:
        mean = [float(v.mean()) for v in lit]
        luma = 0.2126 * mean[0] + 0.7152 * mean[1] + 0.0722 * mean[2]
        ev = min(max(math.log2(float(np.float32(0.18)) / luma), -8.0), 8.0) if luma > 0 else 8.0
        wanted = EXPOSURE[0] * EXPOSURE[1] * 2.0 ** (0.5 * ev)
        exposure = min(max(wanted, 10_000.0), 33_000_000.0)
        saturated = float((counts >= (1 << case["bits"]) - 1).sum()) / counts.numel()
        stats = np.array(mean + [luma, ev, 2.0 ** (0.5 * ev), exposure, min(max(wanted / exposure, 1.0), 16.0)]
                         + list(gains) + [saturated])
    return image, stats


def exact(case, seed):
    if case["kind"] == "frame":
        if case["out"] != "rgb32f" and not case["stats"]:
            return None
        image, stats = _exact_frame(case, seed)
        out = {"image": image}
        if case["histogram"]:
            out["histogram"] = None
        if case["stats"]:
            out["stats"] = stats
        return out
    if case["kind"] == "batch":
        stats = [_exact_frame(c, seed * 1000 + i)[1] for i, c in enumerate(_cameras(case))]
        return {"images": None, "histograms": None, "stats": np.stack(stats)}
    return None  # bytes
