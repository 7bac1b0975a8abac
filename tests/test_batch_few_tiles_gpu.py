"""Batches of a few tiles per CTA, whose ranges are reordered: one more and one
less than the CTAs, a tile or two each, with and without a statistics pass, and
cost weights that leave CTAs without work."""
import numpy as np
import pytest

import isp_b200
from gpu_support import DeviceFrame, same_bits, torch_cuda
from isp_b200 import abi, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("balance", [abi.MANUAL, abi.GRAY_WORLD])
@pytest.mark.parametrize("sizes,weights", [
    ([(64, 40)], (1.0, 1.0, 1.0, 1.0)),
    ([(1920, 1080), (35, 67)], (1.0, 1.0, 1.0, 1.0)),
    ([(640, 480), (640, 480), (200, 150)], (1.0, 1.0, 1.0, 1.0)),
    ([(1792, 1030), (640, 480), (200, 150)], (1.0, 3.0, 1.0, 1.0)),
    ([(1000, 700), (1920, 1080)], (1e-30, float("inf"), 1.0, 1.0)),
])
def test_few_tiles(balance, sizes, weights):
    torch = torch_cuda()
    raws = []
    for i, (w, h) in enumerate(sizes):
        data, pitch = scene.pack(scene.mosaic_counts(w, h, abi.GBRG, 256.0, 4095, 12, i), abi.U16)
        raws.append(abi.RawFrame(data, w, h, pitch, abi.U16, 12, abi.GBRG))

    def cameras():
        return [isp_b200.Pipeline(abi.IspParams(
            black_level=256.0, white_balance=balance, wb_gains=(1.9, 1.0, 1.5),
            demosaic=abi.MALVAR if i % 2 else abi.BILINEAR, lens_shading=scene.lens_shading_grid(r.width, r.height),
            ccm=scene.CCM)) for i, r in enumerate(raws)]

    cams, alone, batch = cameras(), cameras(), isp_b200.Batch(len(raws))
    batch.set_tuning(weights, 0)
    for _ in range(2):
        frames = [DeviceFrame(raw, abi.RGB8) for raw in raws]
        batch.clear()
        for cam, f in zip(cams, frames):
            rv, ov = f.views()
            batch.add(cam, rv, ov, f.hist.data_ptr(), f.stats.data_ptr(), (8_000_000, 1.5))
        torch.cuda.synchronize()
        batch.launch(0, True)
        torch.cuda.synchronize()
        for i, (raw, f, one) in enumerate(zip(raws, frames, alone)):
            g = DeviceFrame(raw, abi.RGB8)
            g.run(one, (8_000_000, 1.5))
            want, got = g.result(), f.result()
            assert same_bits(got.image, want.image), i
            assert np.array_equal(got.histogram, want.histogram), i
            assert same_bits(got.stats, want.stats), i
    batch.close()
