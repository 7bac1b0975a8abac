"""Batches with enough tiles that both passes deal part of them out through
their queues: claimed ranges that cross frames and end in frames of one tile,
with and without a sharpening camera, at both tile heights and under very uneven
cost weights. Every frame must get the bytes the single-frame path gives it."""
import numpy as np
import pytest

import isp_b200
from gpu_support import DeviceFrame, first_mismatch, same_bits, torch_cuda
from isp_b200 import abi, scene

pytestmark = pytest.mark.gpu

# (width, height, raw format, bits, black, pattern, demosaic, wb, out)
BIG = [
    (2626, 2050, abi.U16, 12, 256.0, abi.GBRG, abi.MALVAR, abi.WHITE_PATCH, abi.RGB8),
    (2560, 2000, abi.RAW10, 10, 64.0, abi.RGGB, abi.BILINEAR, abi.GRAY_WORLD, abi.RGB8),
    (2700, 1930, abi.U8, 8, 16.0, abi.BGGR, abi.BILINEAR, abi.GRAY_WORLD, abi.RGB16),
]
TINY = [
    (64, 40, abi.U8, 8, 16.0, abi.RGGB, abi.BILINEAR, abi.GRAY_WORLD, abi.RGB8),
    (35, 67, abi.RAW12, 12, 256.0, abi.GRBG, abi.MALVAR, abi.MANUAL, abi.RGBA8),
    (200, 150, abi.U16, 12, 256.0, abi.GRBG, abi.MALVAR, abi.WHITE_PATCH, abi.RGB8),
]
MIX = TINY[:1] + BIG + BIG + TINY[1:2] + BIG[:1] + TINY


def _raw(spec, seed):
    w, h, fmt, bits, black, pattern = spec[:6]
    data, pitch = scene.pack(scene.mosaic_counts(w, h, pattern, black, (1 << bits) - 1, bits, seed), fmt,
                             abi.raw_row_bytes(fmt, w))
    return abi.RawFrame(data, w, h, pitch, fmt, bits, pattern)


@pytest.fixture(scope="module")
def raws():
    made = {}
    for spec in BIG + TINY:
        made[spec] = _raw(spec, len(made))
    return [made[spec] for spec in MIX]


def _camera(spec, index, sharpen):
    w, h, _, _, black, _, dem, wb, _ = spec
    return isp_b200.Pipeline(abi.IspParams(
        black_level=black, lens_shading=scene.lens_shading_grid(w, h), white_balance=wb,
        wb_gains=(1.0 + 0.1 * index, 1.0, 1.7), demosaic=dem, ccm=scene.CCM, tone_curve=abi.LUT,
        lut=scene.srgb_table(1024), sharpen=sharpen if index % 3 == 1 else 0.0))


@pytest.mark.parametrize("sharpen,rows,weights,use_graph", [
    (0.0, 64, (1.0, 1.0, 1.0, 1.0), True),
    (0.7, 64, (1.0, 1.5, 2.0, 2.5), False),
    (0.7, 32, (1.0, 1e30, 1e-30, float("inf")), True),
    (0.0, 32, (1.0, 100.0, 1.0, 1.0), False),
])
def test_claimed_ranges_match_single_frames(raws, sharpen, rows, weights, use_graph):
    torch = torch_cuda()
    cams = [_camera(spec, i, sharpen) for i, spec in enumerate(MIX)]
    alone = [_camera(spec, i, sharpen) for i, spec in enumerate(MIX)]
    batch = isp_b200.Batch(len(MIX))
    batch.set_tile_rows(rows)
    batch.set_tuning(weights, 1)
    stream = torch.cuda.Stream()
    for _ in range(2):
        frames = [DeviceFrame(raw, spec[8], True) for raw, spec in zip(raws, MIX)]
        batch.clear()
        for cam, f in zip(cams, frames):
            rv, ov = f.views()
            batch.add(cam, rv, ov, f.hist.data_ptr(), f.stats.data_ptr(), (8_000_000, 1.5))
        batch.launch(stream.cuda_stream, use_graph)
        torch.cuda.synchronize()
        for i, (f, cam, one) in enumerate(zip(frames, cams, alone)):
            got = f.result()
            assert cam.device_status() == 0, "a kernel gave up a bounded wait"
            g = DeviceFrame(raws[i], MIX[i][8], True)
            g.run(one, (8_000_000, 1.5))
            want = g.result()
            what = f"frame {i} {MIX[i][:3]}"
            assert same_bits(got.image, want.image), f"{what}: {first_mismatch(got.image, want.image)}"
            assert np.array_equal(got.histogram, want.histogram), f"{what}: histogram"
            assert same_bits(got.stats, want.stats), f"{what}: stats"
            assert np.array_equal(cam.awb()[0], one.awb()[0]), f"{what}: white balance"
    batch.close()
