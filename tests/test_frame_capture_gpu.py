"""Frames captured into a graph, beside frames queued on the same stream."""
import numpy as np
import pytest

import isp_b200
from gpu_support import DeviceFrame, same_bits, torch_cuda
from isp_b200 import abi, cc, scene

pytestmark = pytest.mark.gpu

W, H = 1024, 768


def params(balance=abi.GRAY_WORLD):
    return abi.IspParams(black_level=4096.0, lens_shading=scene.lens_shading_grid(W, H), white_balance=balance,
                         wb_gains=(1.9, 1.0, 1.5), awb_smoothing=0.25, ccm=scene.CCM)


def raw_frame(seed):
    data, pitch = scene.pack(scene.mosaic_counts(W, H, abi.RGGB, 4096.0, 65535, 16, seed), abi.U16)
    return abi.RawFrame(data, W, H, pitch, abi.U16, 16, abi.RGGB)


def alone(raws, balance=abi.GRAY_WORLD):
    """The frames' results one after the other, each waited for."""
    pipe, results = isp_b200.Pipeline(params(balance)), []
    for raw in raws:
        f = DeviceFrame(raw, abi.RGB8)
        f.run(pipe)
        results.append(f.result())
    return results


def same(frame, want, what):
    got = frame.result()
    assert same_bits(got.image, want.image), what
    assert np.array_equal(got.histogram, want.histogram), what
    assert same_bits(got.stats, want.stats), what


def capture(stream, queue):
    torch = torch_cuda()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        queue()
    return graph


@pytest.mark.parametrize("balance", [abi.MANUAL, abi.GRAY_WORLD])
def test_frames_can_be_captured(balance):
    """Two frames of a camera in one graph; each replay processes the raw samples of the moment."""
    torch = torch_cuda()
    want = alone([raw_frame(i) for i in (1, 2, 3, 4)], balance)
    pipe, stream = isp_b200.Pipeline(params(balance)), torch.cuda.Stream()
    frames = [DeviceFrame(raw_frame(0), abi.RGB8) for _ in range(2)]
    torch.cuda.synchronize()
    graph = capture(stream, lambda: [f.run(pipe, stream=stream.cuda_stream) for f in frames])
    for k in (0, 2):
        for i, f in enumerate(frames):
            f.raw.copy_(torch.from_numpy(raw_frame(1 + k + i).data))
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        for i, f in enumerate(frames):
            same(f, want[k + i], k + i)


def test_a_captured_frame_is_not_waited_for_by_others():
    """Another camera's next frame follows its own work on the stream, not the captured frame's event."""
    torch = torch_cuda()
    raws = [raw_frame(i) for i in range(3)]
    want, captured_want = alone(raws), alone(raws[:1])
    camera, other, captured = (isp_b200.Pipeline(params()) for _ in range(3))
    frames, inside = [DeviceFrame(raw, abi.RGB8) for raw in raws], DeviceFrame(raws[0], abi.RGB8)
    beside, stream = DeviceFrame(raws[0], abi.RGB8), torch.cuda.Stream()
    torch.cuda.synchronize()
    frames[0].run(camera, stream=stream.cuda_stream)
    beside.run(other, stream=stream.cuda_stream)
    torch.cuda.synchronize()
    graph = capture(stream, lambda: inside.run(captured, stream=stream.cuda_stream))
    frames[1].run(camera, stream=stream.cuda_stream)
    with torch.cuda.stream(stream):
        graph.replay()
    frames[2].run(camera, stream=stream.cuda_stream)
    for i, f in enumerate(frames):
        same(f, want[i], i)
    same(inside, captured_want[0], "captured")


@pytest.mark.parametrize("balance", [abi.MANUAL, abi.GRAY_WORLD])
def test_captured_cameras_in_turn(balance):
    """Frames of two cameras in one graph, each behind the other's."""
    torch = torch_cuda()
    raws = [raw_frame(i) for i in range(3)]
    want = alone(raws + raws, balance)
    pipes, stream = [isp_b200.Pipeline(params(balance)) for _ in range(2)], torch.cuda.Stream()
    frames = [[DeviceFrame(raw, abi.RGB8) for raw in raws] for _ in pipes]
    torch.cuda.synchronize()
    graph = capture(stream, lambda: [f[i].run(pipe, stream=stream.cuda_stream) for i in range(3)
                                     for f, pipe in zip(frames, pipes)])
    for k in (0, 3):
        with torch.cuda.stream(stream):
            graph.replay()
        for camera in frames:
            for i, f in enumerate(camera):
                same(f, want[k + i], k + i)


@pytest.mark.parametrize("balance", [abi.MANUAL, abi.GRAY_WORLD])
def test_a_captured_frame_waits_for_the_conversion_before_it(balance):
    """frame, conversion into the raw samples of the next, frame: in one graph, replayed with changing sources."""
    torch = torch_cuda()
    raws = [raw_frame(i) for i in range(4)]
    want = alone([raws[i] for i in (0, 1, 2, 3)], balance)
    pipe, converter, stream = isp_b200.Pipeline(params(balance)), cc.Converter(), torch.cuda.Stream()
    sources = [torch.zeros_like(DeviceFrame(raws[0], abi.RGB8).raw) for _ in range(2)]
    frames = [DeviceFrame(raws[0], abi.RGB8) for _ in range(2)]
    copy = cc.params(cc.BT709, mode=cc.NEAREST)

    def queue():
        for source, f in zip(sources, frames):
            converter.convert(cc.packed_view(source.data_ptr(), cc.MONO16, W, H),
                              cc.packed_view(f.raw.data_ptr(), cc.MONO16, W, H), copy, stream.cuda_stream)
            f.run(pipe, stream=stream.cuda_stream)

    torch.cuda.synchronize()
    graph = capture(stream, queue)
    for k in (0, 2):
        for i, source in enumerate(sources):
            source.copy_(torch.from_numpy(raws[k + i].data))
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        for i, f in enumerate(frames):
            same(f, want[k + i], k + i)
