"""A pipeline's frame whose raw samples are the image of a no-alloc frame queued
just before it: the no-alloc frame's kernels let dependents start early, so the
frame must not start under them as it may start under another pipeline's frame."""
import numpy as np
import pytest

import isp_b200
from gpu_support import DeviceFrame, same_bits, torch_cuda
from isp_b200 import abi, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("balance", [abi.GRAY_WORLD, abi.MANUAL])
def test_raw_samples_from_a_noalloc_frame(balance):
    torch = torch_cuda()
    w, h = 704, 1536  # its RGB16 image: a mosaic of 2112x1536
    first = abi.IspParams(black_level=256.0, white_balance=abi.MANUAL, ccm=scene.CCM)
    second = abi.IspParams(black_level=1024.0, white_balance=balance, wb_gains=(1.9, 1.0, 1.5), awb_smoothing=0.25,
                           lens_shading=scene.lens_shading_grid(3 * w, h), ccm=scene.CCM)
    raws = []
    for seed in (1, 2, 3):
        data, pitch = scene.pack(scene.mosaic_counts(w, h, abi.RGGB, 256.0, 4095, 12, seed), abi.U16)
        raws.append(abi.RawFrame(data, w, h, pitch, abi.U16, 12, abi.RGGB))
    empty = abi.RawFrame(np.zeros(6 * w * h, np.uint8), 3 * w, h, 6 * w, abi.U16, 16, abi.GRBG)
    inputs = [DeviceFrame(raw, abi.RGB16) for raw in raws]
    stream = torch.cuda.Stream()

    def frames(pipe, wait):
        results = [DeviceFrame(empty, abi.RGB8) for _ in range(6)]
        shared = torch.zeros_like(results[0].raw)
        for f in results:
            f.raw = shared
        torch.cuda.synchronize()
        for i, f in enumerate(results):
            raw, _ = inputs[i % 3].views()
            isp_b200.process_noalloc(first, raw, abi.RgbViewC(shared.data_ptr(), 6 * w, abi.RGB16), stream=stream.cuda_stream)
            if wait:
                torch.cuda.synchronize()
            f.run(pipe, stream=stream.cuda_stream)
            if wait:
                torch.cuda.synchronize()
        return [f.result() for f in results]

    want = frames(isp_b200.Pipeline(second), True)
    got = frames(isp_b200.Pipeline(second), False)
    for i, (a, b) in enumerate(zip(got, want)):
        assert same_bits(a.image, b.image), i
        assert np.array_equal(a.histogram, b.histogram), i
