"""The tile and statistics passes where their set-up differs from frame to
frame: rows that no 16-byte alignment helps (boxes filled without TMA), output
rows of every alignment, lens shading grids too dense for a tile's table, and
the frames of several cameras in turn on one stream, whose kernels overlap.
Everything against the C oracle, bit for bit.
"""
import numpy as np
import pytest

import isp_b200
import oracle
from gpu_support import DeviceFrame, same_bits, torch_cuda
from isp_b200 import abi, scene

pytestmark = pytest.mark.gpu

EXPOSURE = (10_000_000, 1.5)
BITS = {abi.U8: 8, abi.U16: 12, abi.RAW10: 10, abi.RAW12: 12}


def _raw(width, height, fmt, pattern, seed, pitch=None):
    bits = BITS[fmt]
    black = float(1 << (bits - 4))
    counts = scene.mosaic_counts(width, height, pattern, black, (1 << bits) - 1, bits, seed)
    counts[:: 7, :: 5] = (1 << bits) - 1  # saturated samples everywhere
    data, pitch = scene.pack(counts, fmt, pitch)
    return abi.RawFrame(data, width, height, pitch, fmt, bits, pattern), black


def _params(black, width, height, balance, demosaic, sharpen, grid=None, smoothing=0.25):
    lsc = scene.lens_shading_grid(width, height, *(grid or (17, 13)))
    return abi.IspParams(black_level=black, lens_shading=lsc, white_balance=balance, wb_gains=(1.9, 1.0, 1.5),
                         awb_smoothing=smoothing, demosaic=demosaic, ccm=scene.CCM, sharpen=sharpen)


def _same(got, exp, what):
    assert same_bits(got.image, exp.image), f"{what}: image"
    assert np.array_equal(got.histogram, exp.histogram), f"{what}: histogram"
    assert same_bits(got.stats, exp.stats), f"{what}: {got.stats} vs {exp.stats}"


@pytest.mark.parametrize("rows", [64, 32])
@pytest.mark.parametrize("fmt,offset,extra", [(abi.U8, 1, 0), (abi.U8, 0, 3), (abi.U8, 4, 0), (abi.U16, 2, 0),
                                              (abi.U16, 4, 4), (abi.U16, 0, 2), (abi.RAW10, 3, 1), (abi.RAW10, 8, 0),
                                              (abi.RAW12, 1, 2), (abi.RAW12, 4, 4)])
@pytest.mark.parametrize("size", [(131, 67), (198, 130), (66, 5)])
def test_rows_without_alignment(fmt, offset, extra, size, rows):
    torch = torch_cuda()
    w, h = size
    pitch = abi.raw_row_bytes(fmt, w) + extra
    if fmt == abi.U16:
        pitch += pitch % 2
    raw, black = _raw(w, h, fmt, abi.GBRG, 5, pitch)
    params = _params(black, w, h, abi.WHITE_PATCH, abi.MALVAR, 0.5 if rows == 64 else 0.0)
    pipe, ref = isp_b200.Pipeline(params), oracle.OraclePipeline(params)
    pipe.set_tile_rows(rows)
    frame = DeviceFrame(raw, abi.RGB8)
    # The frame's bytes `offset` into a buffer that ends right behind them.
    moved = torch.empty(offset + raw.data.size, dtype=torch.uint8, device="cuda")
    moved[offset:] = frame.raw
    frame.raw = moved[offset:]
    for f in range(2):
        frame.run(pipe, EXPOSURE)
        _same(frame.result(), ref.process(raw, abi.RGB8, True, EXPOSURE), f"frame {f}")
    assert pipe.device_status() == 0


@pytest.mark.parametrize("fmt", [abi.RGB8, abi.RGBA8, abi.RGB16, abi.RGB32F])
@pytest.mark.parametrize("extra", [0, 1, 2, 3])
def test_output_rows_of_every_alignment(fmt, extra):
    w, h = 135, 66
    raw, black = _raw(w, h, abi.RAW10, abi.RGGB, 9)
    params = _params(black, w, h, abi.GRAY_WORLD, abi.BILINEAR, 0.0)
    cb = abi.output_channel_bytes(fmt)
    pitch = (w * abi.output_channels(fmt) + extra) * cb
    frame = DeviceFrame(raw, fmt, out_pitch=pitch)
    frame.run(isp_b200.Pipeline(params), EXPOSURE)
    _same(frame.result(), oracle.OraclePipeline(params).process(raw, fmt, True, EXPOSURE), "frame")
    row = w * abi.output_channels(fmt) * cb
    assert np.all(frame.out.cpu().numpy().reshape(h, pitch)[:, row:] == 0xAB), "padding bytes were written"


@pytest.mark.parametrize("channels", [1, 4])
@pytest.mark.parametrize("grid", [(64, 64), (9, 40), (200, 3), (2, 2)])
def test_lens_shading_grids(grid, channels):
    """Grid cells of a few rows (no table), of a row or two per tile row, and one cell for the frame."""
    w, h = 190, 150
    raw, black = _raw(w, h, abi.RAW12, abi.BGGR, 3)
    params = _params(black, w, h, abi.GRAY_WORLD, abi.MALVAR, 0.75, (*grid, channels))
    rng = np.random.default_rng(1)
    params.lens_shading.gains = rng.uniform(0.5, 3.0, params.lens_shading.gains.shape).astype(np.float32)
    frame = DeviceFrame(raw, abi.RGB16)
    frame.run(isp_b200.Pipeline(params), EXPOSURE)
    _same(frame.result(), oracle.OraclePipeline(params).process(raw, abi.RGB16, True, EXPOSURE), "frame")


@pytest.mark.parametrize("between", [False, True])
def test_cameras_in_turn_on_one_stream(between):
    """Four cameras (manual, gray world, white patch; sharpened or not), five
    frames each, queued in turn on one stream and never waited for, each camera
    into one output buffer; with `between`, other work on the stream as well.
    The first four frames' results are copied out on the stream."""
    torch = torch_cuda()
    stream = torch.cuda.Stream()
    cameras = []
    for i, (balance, demosaic, sharpen, size) in enumerate(((abi.MANUAL, abi.BILINEAR, 0.0, (640, 480)),
                                                            (abi.GRAY_WORLD, abi.MALVAR, 0.5, (322, 250)),
                                                            (abi.WHITE_PATCH, abi.MALVAR, 0.0, (700, 130)),
                                                            (abi.MANUAL, abi.MALVAR, 0.5, (64, 48)))):
        raws = [_raw(*size, abi.U16, abi.GRBG, 10 * i + f) for f in range(5)]
        params = _params(raws[0][1], *size, balance, demosaic, sharpen)
        frames = [DeviceFrame(r, abi.RGB8) for r, _ in raws]
        for f in frames[1:]:
            f.out, f.hist, f.stats = frames[0].out, frames[0].hist, frames[0].stats
        cameras.append((params, isp_b200.Pipeline(params), [r for r, _ in raws], frames, []))
    filler = torch.zeros(1 << 20, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for f in range(5):
            for params, pipe, raws, frames, kept in cameras:
                frames[f].run(pipe, EXPOSURE, stream.cuda_stream)
                if between or f < 4:
                    kept.append((frames[f].out.clone(), frames[f].hist.clone(), frames[f].stats.clone()))
                if between:
                    filler += 1.0
    torch.cuda.synchronize()
    for c, (params, pipe, raws, frames, kept) in enumerate(cameras):
        ref = oracle.OraclePipeline(params)
        for f in range(5):
            exp = ref.process(raws[f], abi.RGB8, True, EXPOSURE)
            if f < len(kept):
                frames[f].out, frames[f].hist, frames[f].stats = kept[f]
            _same(frames[f].result(), exp, f"camera {c} frame {f}")
        assert pipe.device_status() == 0


def test_cameras_back_to_back_without_a_copy_between():
    """Twelve frames of three cameras back to back on one stream, each into buffers of its own."""
    torch = torch_cuda()
    stream = torch.cuda.Stream()
    queued, cameras = [], []
    for i, (balance, sharpen) in enumerate(((abi.MANUAL, 0.0), (abi.WHITE_PATCH, 0.0), (abi.GRAY_WORLD, 1.0))):
        raws = [_raw(450, 333, abi.RAW10, abi.RGGB, 20 * i + f) for f in range(4)]
        params = _params(raws[0][1], 450, 333, balance, abi.MALVAR, sharpen)
        cameras.append((params, isp_b200.Pipeline(params), [(r, DeviceFrame(r, abi.RGB16)) for r, _ in raws]))
    torch.cuda.synchronize()
    for f in range(4):
        for params, pipe, frames in cameras:
            frames[f][1].run(pipe, EXPOSURE, stream.cuda_stream)
    torch.cuda.synchronize()
    for c, (params, pipe, frames) in enumerate(cameras):
        ref = oracle.OraclePipeline(params)
        for f, (raw, frame) in enumerate(frames):
            _same(frame.result(), ref.process(raw, abi.RGB16, True, EXPOSURE), f"camera {c} frame {f}")
        pipe.close()
