"""Frames of one pipeline that follow each other on one stream at different
sizes: a frame's kernels may start under the previous frame's end, so nothing
that the frames share (the counter by which tiles are claimed among it) may be
touched before that frame is done."""
import numpy as np
import pytest

import isp_b200
from gpu_support import DeviceFrame, same_bits, torch_cuda
from isp_b200 import abi, scene

pytestmark = pytest.mark.gpu


def _raw(w, h, seed):
    data, pitch = scene.pack(scene.mosaic_counts(w, h, abi.GRBG, 256.0, 4095, 12, seed), abi.U16)
    return abi.RawFrame(data, w, h, pitch, abi.U16, 12, abi.GRBG)


@pytest.mark.parametrize("sharpen", [0.0, 0.5])
@pytest.mark.parametrize("balance", [abi.MANUAL, abi.GRAY_WORLD])
def test_sizes_in_turn_on_one_stream(balance, sharpen):
    """A frame of fewer tiles than CTAs fit leaves room for the next one's to start at once."""
    torch = torch_cuda()
    sizes = [(512, 640), (3008, 2112), (640, 70), (2624, 1984)]
    raws = [_raw(w, h, i) for i, (w, h) in enumerate(sizes)]

    def params(w, h):
        return abi.IspParams(black_level=256.0, lens_shading=scene.lens_shading_grid(w, h), white_balance=balance,
                             wb_gains=(1.9, 1.0, 1.5), awb_smoothing=0.25, ccm=scene.CCM, sharpen=sharpen)

    pipe, alone = (isp_b200.Pipeline(params(3008, 2112)) for _ in range(2))
    order = [0, 1, 0, 3, 2, 1, 2, 3] * 3
    frames = [DeviceFrame(raws[k], abi.RGB8) for k in order]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for f in frames:
        f.run(pipe, (0, 0.0), stream.cuda_stream)
    torch.cuda.synchronize()
    assert pipe.device_status() == 0
    for i, (k, f) in enumerate(zip(order, frames)):
        one = DeviceFrame(raws[k], abi.RGB8)
        one.run(alone, (0, 0.0))
        want, got = one.result(), f.result()  # waits: every frame alone
        assert same_bits(got.image, want.image), i
        assert np.array_equal(got.histogram, want.histogram), i
        assert same_bits(got.stats, want.stats), i
