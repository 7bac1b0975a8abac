"""A camera's frame on its stream waits for no work of another camera on another
stream, whatever that camera did on this one before."""
import pytest

import isp_b200
from gpu_support import DeviceFrame, torch_cuda
from isp_b200 import abi, scene

pytestmark = pytest.mark.gpu

W, H = 640, 480


def _frame(seed):
    data, pitch = scene.pack(scene.mosaic_counts(W, H, abi.RGGB, 16.0, 255, 8, seed), abi.U8)
    return DeviceFrame(abi.RawFrame(data, W, H, pitch, abi.U8, 8, abi.RGGB), abi.RGB8)


@pytest.mark.parametrize("work", ["batch", "check"])
def test_work_of_another_camera_on_another_stream(work):
    torch = torch_cuda()
    params = abi.IspParams(black_level=16.0, white_balance=abi.GRAY_WORLD, ccm=scene.CCM)
    a, b = isp_b200.Pipeline(params), isp_b200.Pipeline(params)
    frames = [_frame(i) for i in range(4)]
    here, there = torch.cuda.Stream(), torch.cuda.Stream()
    batch = isp_b200.Batch(1)
    raw, out = frames[2].views()

    def beside():
        if work == "batch":
            batch.clear()
            batch.add(a, raw, out)
            batch.launch(there.cuda_stream)
        else:
            a.check_bounded_wait(16, there.cuda_stream)

    beside()  # everything loaded and set up
    torch.cuda.synchronize()
    frames[0].run(b, stream=here.cuda_stream)
    frames[1].run(a, stream=here.cuda_stream)  # the last frame of `here`
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    with torch.cuda.stream(there):
        torch.cuda._sleep(400_000_000)  # a fifth of a second
    beside()
    done.record(there)
    frames[3].run(b, stream=here.cuda_stream)
    here.synchronize()
    assert not done.query(), "the frame waited for the other stream"
    torch.cuda.synchronize()
    batch.close()
