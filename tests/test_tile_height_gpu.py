"""Frames whose tile height the pipeline chooses by itself, on both sides of its
lines (tiles as many as SMs, sharpened or not), and small frames at the height it
would not choose: the same bytes as the oracle's at either height."""
import numpy as np
import pytest

import isp_b200
import oracle
from gpu_support import DeviceFrame, same_bits, torch_cuda
from isp_b200 import abi, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sharpen", [0.0, 0.5])
@pytest.mark.parametrize("tiles", [(1, 1, 0), (0, 1, -3), (0, 1, 1), (0, 2, 1), (2, 2, 5)])
def test_chosen_height_gives_the_same_bytes(sharpen, tiles):
    """tiles: half the columns' share of the SMs or one, rows of tiles, and rows beyond a whole number of them."""
    torch = torch_cuda()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    across = tiles[0] or (sms // tiles[1])
    rows = 64 if sharpen else 32
    w, h = 64 * across - 1, max(5, rows * tiles[1] + tiles[2])
    counts = scene.mosaic_counts(w, h, abi.GBRG, 256.0, 4095, 12, w + h)
    data, pitch = scene.pack(counts, abi.U16)
    raw = abi.RawFrame(data, w, h, pitch, abi.U16, 12, abi.GBRG)
    params = abi.IspParams(black_level=256.0, lens_shading=scene.lens_shading_grid(w, h), white_balance=abi.GRAY_WORLD,
                           wb_gains=(1.9, 1.0, 1.5), demosaic=abi.MALVAR, ccm=scene.CCM, sharpen=sharpen)
    want = oracle.OraclePipeline(params).process(raw, abi.RGB16, True, (10_000_000, 1.5))
    for height in (0, 64, 32):
        pipe = isp_b200.Pipeline(params)
        pipe.set_tile_rows(height)
        frame = DeviceFrame(raw, abi.RGB16)
        frame.run(pipe, (10_000_000, 1.5))
        got = frame.result()
        assert same_bits(got.image, want.image), height
        assert np.array_equal(got.histogram, want.histogram), height
        assert same_bits(got.stats, want.stats), height
