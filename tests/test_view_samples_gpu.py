"""The view's gray codes where they come from a table and where they do not:
samples beyond the bit depth, frames of one run per thread and of several."""
import numpy as np
import pytest

import isp_b200
import oracle
from isp_b200 import abi, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,bits,top", [(abi.U8, 8, 8), (abi.U8, 5, 8), (abi.U16, 9, 16), (abi.U16, 12, 16), (abi.U16, 13, 16),
                                          (abi.RAW10, 10, 10), (abi.RAW10, 7, 10), (abi.RAW12, 12, 12)])
@pytest.mark.parametrize("size", [(48, 6), (35, 9), (2048, 1700)])
def test_samples_beyond_the_bit_depth(fmt, bits, top, size):
    import torch

    w, h = size
    rng = np.random.default_rng(w + bits)
    data, pitch = scene.pack(rng.integers(0, 1 << top, (h, w)).astype(np.uint16), fmt)
    raw = abi.RawFrame(data, w, h, pitch, fmt, bits, abi.RGGB)
    rgb = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    d_raw, d_rgb = torch.from_numpy(data).cuda(), torch.from_numpy(rgb.reshape(-1)).cuda()
    out = torch.full((h * 6 * w + 16,), 0xAB, dtype=torch.uint8, device="cuda")
    isp_b200.view_compose(raw.view(d_raw.data_ptr()), 3.0, d_rgb.data_ptr(), 3 * w, out.data_ptr(), 6 * w)
    torch.cuda.synchronize()
    assert np.array_equal(out[:-16].cpu().numpy().reshape(h, 2 * w, 3), oracle.view_compose(raw, 3.0, rgb))
    assert bool((out[-16:] == 0xAB).all())


@pytest.mark.parametrize("fmt,bits", [(abi.U8, 8), (abi.U16, 14), (abi.RAW10, 10), (abi.RAW12, 12)])
@pytest.mark.parametrize("w,h", [(1, 3), (513, 5), (1030, 7), (515, 4), (528, 3)])
def test_rows_at_every_byte(fmt, bits, w, h):
    """Raw, RGB and view rows that start at any byte; what surrounds the view's rows stays."""
    import torch

    rng = np.random.default_rng(w * h + bits)
    counts = rng.integers(0, 1 << bits, (h, w)).astype(np.uint16)
    rgb = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    for shift in range(4):
        data, pitch = scene.pack(counts, fmt, abi.raw_row_bytes(fmt, w) + shift)
        raw = abi.RawFrame(data, w, h, pitch, fmt, bits, abi.RGGB)
        d_raw = torch.zeros(data.size + 4, dtype=torch.uint8, device="cuda")
        d_raw[shift:shift + data.size] = torch.from_numpy(data.reshape(-1).view(np.uint8)).cuda()
        rows = torch.zeros((h, 3 * w + 3 - shift), dtype=torch.uint8, device="cuda")
        rows[:, :3 * w] = torch.from_numpy(rgb.reshape(h, -1)).cuda()
        out = torch.full((16 + h * (6 * w + shift) + 16,), 0xAB, dtype=torch.uint8, device="cuda")
        isp_b200.view_compose(raw.view(d_raw.data_ptr() + shift), 3.0, rows.data_ptr(), 3 * w + 3 - shift,
                              out.data_ptr() + 5 + shift, 6 * w + shift)
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        body = got[5 + shift:5 + shift + h * (6 * w + shift)].reshape(h, -1)
        assert np.array_equal(body[:, :6 * w].reshape(h, 2 * w, 3), oracle.view_compose(raw, 3.0, rgb)), shift
        assert (body[:, 6 * w:] == 0xAB).all() and (got[:5 + shift] == 0xAB).all() and (got[body.size + 5 + shift:] == 0xAB).all()
