"""The converter's resample kernel where its routes part: area footprints of
whole pixels (summed as integers) and of any other size, planes and rows whose
words can be read whole or not, alpha carried or constant, groups of four
pixels cut by a letterbox or the image's edge. Byte for byte against the C
oracle, as tests/test_cc_gpu.py.
"""
from __future__ import annotations

import pytest

from isp_b200 import cc
from oracle import cc as occ
from test_cc_gpu import expect_same

pytestmark = pytest.mark.gpu

EIGHT_BIT = (cc.NV12, cc.NV16, cc.I420, cc.YUYV, cc.UYVY, cc.RGB8, cc.BGR8, cc.RGBA8, cc.BGRA8, cc.MONO8)
DESTS = (cc.RGB8, cc.NV12, cc.UYVY, cc.BGRA8, cc.MONO16)


@pytest.mark.parametrize("across,down", [(2, 2), (3, 3), (4, 4), (3, 1), (2, 7), (4, 3), (5, 5)])
@pytest.mark.parametrize("src", EIGHT_BIT)
def test_area_of_whole_pixels(src, across, down):
    for dw, dh, pad in ((36, 10, 0), (22, 5, 0), (24, 6, 4), (24, 6, 1)):
        w, h = dw * across, dh * down
        img = occ.noise(src, w, h, 7 * across + down)
        for dst in DESTS:
            p = cc.params(cc.BT709, mode=cc.AREA)
            assert expect_same(img, src, w, h, dst, dw, dh, p, pads=(pad, 0)) == 0, (dw, dh, pad, dst)


@pytest.mark.parametrize("src", (cc.NV12, cc.RGB8, cc.BGRA8))
def test_whole_pixels_under_a_letterbox_or_a_crop(src):
    w, h = 96, 48
    img = occ.noise(src, w, h, 3)
    for dw, dh, box, crop in ((32, 32, True, None), (40, 16, True, None), (50, 24, True, None), (30, 14, False, (3, 3, 90, 42)),
                              (16, 8, False, (32, 16, 48, 24)), (48, 24, False, (0, 0, 96, 48))):
        for dst in (cc.RGBA8, cc.NV12):
            p = cc.params(cc.BT709, mode=cc.AREA, crop=crop, letterbox=box, fill_rgb=(200, 30, 90))
            assert expect_same(img, src, w, h, dst, dw, dh, p) == 0, (dw, dh, box, crop, dst)


@pytest.mark.parametrize("mode", (cc.NEAREST, cc.BILINEAR, cc.AREA))
@pytest.mark.parametrize("src", cc.ALL_FORMATS)
def test_every_alignment_and_scale(src, mode):
    """Scales on both sides of the area tap counts, offsets and paddings that allow whole words or forbid them."""
    w, h = 92, 41
    img = occ.noise(src, w, h, 11)
    for dw, dh, offset, pad in ((70, 33, 0, 0), (37, 17, 0, 0), (26, 12, 2, 2), (19, 8, 1, 3), (13, 5, 4, 0), (150, 60, 3, 1),
                                (4, 41, 0, 4), (92, 3, 0, 0)):
        for dst in (cc.RGB8, cc.I420, cc.BGRA8, cc.RGB16):
            p = cc.params(cc.BT601, cc.FULL, mode)
            assert expect_same(img, src, w, h, dst, dw, dh, p, offsets=(offset, offset), pads=(pad, 0)) == 0, (dw, dh, offset, dst)


@pytest.mark.parametrize("src", (cc.NV12, cc.RGB8, cc.RGBA8, cc.MONO16))
def test_footprints_of_thousands_of_pixels(src):
    """Whole and broken footprints on both sides of the size from which alpha is summed."""
    w, h = 640, 300
    img = occ.noise(src, w, h, 2)
    for dw, dh in ((10, 5), (9, 7), (5, 2), (3, 1), (1, 1)):
        for dst in (cc.RGBA8, cc.NV12):
            assert expect_same(img, src, w, h, dst, dw, dh, cc.params(cc.BT709, mode=cc.AREA)) == 0, (dw, dh, dst)


def test_a_chain_of_conversions_on_one_stream():
    """Conversions queued back to back, each reading what the one before wrote."""
    import numpy as np
    import torch

    w, h = 322, 242
    stream = torch.cuda.Stream()
    img = occ.noise(cc.RGB8, w, h, 5)
    hops = ((cc.NV12, w, h, cc.NEAREST), (cc.RGBA8, 161, 121, cc.AREA), (cc.YUYV, 400, 200, cc.BILINEAR), (cc.RGB8, 200, 100, cc.AREA),
            (cc.BGR8, 200, 100, cc.NEAREST), (cc.MONO8, 77, 91, cc.BILINEAR))
    want, size, fmt = img, (w, h), cc.RGB8
    source = torch.from_numpy(img).cuda()
    buffers = [torch.empty(cc.packed_size(f, a, b), dtype=torch.uint8, device="cuda") for f, a, b, _ in hops]
    torch.cuda.synchronize()
    for _ in range(20):
        at, at_size, at_fmt = source, (w, h), cc.RGB8
        for (f, a, b, mode), out in zip(hops, buffers):
            cc.Converter().convert(cc.packed_view(at.data_ptr(), at_fmt, *at_size), cc.packed_view(out.data_ptr(), f, a, b),
                                   cc.params(cc.BT709, mode=mode), stream.cuda_stream)
            at, at_size, at_fmt = out, (a, b), f
    for f, a, b, mode in hops:
        want = occ.convert(want, fmt, *size, f, a, b, cc.params(cc.BT709, mode=mode))
        size, fmt = (a, b), f
    torch.cuda.synchronize()
    assert np.array_equal(buffers[-1].cpu().numpy(), want)
