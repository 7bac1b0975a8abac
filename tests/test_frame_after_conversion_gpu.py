"""A frame whose raw samples a conversion on the same stream has just written:
the conversion's kernel signals its dependents early, so the frame must not
start under it as it may start under another frame."""
import numpy as np
import pytest

import isp_b200
from gpu_support import DeviceFrame, same_bits, torch_cuda
from isp_b200 import abi, cc, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("balance", [abi.GRAY_WORLD, abi.MANUAL])
def test_raw_frames_written_by_conversions(balance):
    torch = torch_cuda()
    w, h = 2048, 1536
    params = abi.IspParams(black_level=4096.0, lens_shading=scene.lens_shading_grid(w, h), white_balance=balance,
                           wb_gains=(1.9, 1.0, 1.5), awb_smoothing=0.25, ccm=scene.CCM)
    raws = []
    for seed in (1, 2):
        data, pitch = scene.pack(scene.mosaic_counts(w, h, abi.RGGB, 4096.0, 65535, 16, seed), abi.U16)
        raws.append(abi.RawFrame(data, w, h, pitch, abi.U16, 16, abi.RGGB))
    alone = isp_b200.Pipeline(params)
    want = []
    for i in range(8):
        f = DeviceFrame(raws[i % 2], abi.RGB8)
        f.run(alone, (0, 0.0))
        want.append(f.result())
    pipe, converter, stream = isp_b200.Pipeline(params), cc.Converter(), torch.cuda.Stream()
    frames = [DeviceFrame(raws[i % 2], abi.RGB8) for i in range(8)]
    sources = [f.raw.clone() for f in frames[:2]]
    shared = torch.zeros_like(frames[0].raw)  # every frame's raw samples, rewritten for each
    for f in frames:
        f.raw = shared
    torch.cuda.synchronize()
    copy = cc.params(cc.BT709, mode=cc.NEAREST)
    for i, f in enumerate(frames):
        converter.convert(cc.packed_view(sources[i % 2].data_ptr(), cc.MONO16, w, h), cc.packed_view(shared.data_ptr(), cc.MONO16, w, h),
                          copy, stream.cuda_stream)
        f.run(pipe, (0, 0.0), stream.cuda_stream)
    for i, (f, exp) in enumerate(zip(frames, want)):
        got = f.result()
        assert same_bits(got.image, exp.image), i
        assert np.array_equal(got.histogram, exp.histogram), i
