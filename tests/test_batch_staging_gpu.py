"""Launches of one batch whose staged ranges differ in number although its graph
stays the same: cost weights that move work between the CTAs' own ranges and the
queue from launch to launch, and fewer cameras in between."""
import numpy as np
import pytest

import isp_b200
from gpu_support import DeviceFrame, same_bits, torch_cuda
from isp_b200 import abi, scene

pytestmark = pytest.mark.gpu


def _raw(w, h, seed):
    data, pitch = scene.pack(scene.mosaic_counts(w, h, abi.GBRG, 256.0, 4095, 12, seed), abi.U16)
    return abi.RawFrame(data, w, h, pitch, abi.U16, 12, abi.GBRG)


@pytest.mark.parametrize("use_graph", [True, False])
def test_ranges_of_any_number(use_graph):
    torch = torch_cuda()
    raws = [_raw(2560, 2048, 1), _raw(640, 480, 2), _raw(2564, 1990, 3)]

    def cameras():
        return [isp_b200.Pipeline(abi.IspParams(
            black_level=256.0, white_balance=abi.GRAY_WORLD, demosaic=abi.MALVAR if i else abi.BILINEAR,
            lens_shading=scene.lens_shading_grid(r.width, r.height), ccm=scene.CCM)) for i, r in enumerate(raws)]

    cams, alone = cameras(), cameras()
    batch, stream = isp_b200.Batch(3), torch.cuda.Stream()
    for weights, used in (((1.0, 1.0, 1.0, 1.0), (0, 1, 2)), ((1.0, 40.0, 1.0, 1.0), (0, 1, 2)), ((1.0, 1.0, 1.0, 1.0), (1,)),
                          ((50.0, 1.0, 1.0, 1.0), (2, 0, 1)), ((1.0, 1.0, 1.0, 1.0), (0, 1, 2))):
        batch.clear()
        batch.set_tuning(weights, 1)
        frames = [DeviceFrame(raw, abi.RGB8) for raw in raws]
        for i in used:
            rv, ov = frames[i].views()
            batch.add(cams[i], rv, ov, frames[i].hist.data_ptr(), frames[i].stats.data_ptr(), (8_000_000, 1.5))
        torch.cuda.synchronize()
        batch.launch(stream.cuda_stream, use_graph)
        torch.cuda.synchronize()
        for i in used:
            one = DeviceFrame(raws[i], abi.RGB8)
            one.run(alone[i], (8_000_000, 1.5))
            want, got = one.result(), frames[i].result()
            assert same_bits(got.image, want.image), (weights, i)
            assert np.array_equal(got.histogram, want.histogram), (weights, i)
            assert same_bits(got.stats, want.stats), (weights, i)
    batch.close()
