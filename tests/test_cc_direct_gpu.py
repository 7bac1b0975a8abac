"""The converter's direct kernel where its routes part: rows that start at any
byte (whole words shifted together on the way in, and between neighbouring lanes
on the way out), groups of four pixels cut by the right edge, a letterbox or a
crop, chroma from mid-pair, last rows without a partner. Byte for byte against
the C oracle, as tests/test_cc_gpu.py.
"""
from __future__ import annotations

import pytest

from isp_b200 import cc
from oracle import cc as occ
from test_cc_gpu import expect_same

pytestmark = pytest.mark.gpu

PACKED = (cc.YUYV, cc.UYVY)  # whole pixel pairs only


@pytest.mark.parametrize("src", cc.ALL_FORMATS)
def test_every_pair_at_every_alignment(src):
    for w, h, offset, pad in ((261, 3, 0, 0), (518, 5, 1, 3), (134, 2, 2, 1), (127, 4, 3, 2), (132, 3, 0, 1), (4, 1, 1, 0), (7, 2, 0, 0)):
        even = w & ~1
        imgs = {width: occ.noise(src, width, h, width) for width in (w, even) if not (src in PACKED and width & 1)}
        for dst in cc.ALL_FORMATS:
            width = even if src in PACKED or dst in PACKED else w
            p = cc.params(cc.BT709, mode=cc.NEAREST)
            assert expect_same(imgs[width], src, width, h, dst, width, h, p, offsets=(offset, 3 - offset), pads=(pad, 3 - pad)) == 0, \
                (width, h, offset, pad, dst)


@pytest.mark.parametrize("src", cc.ALL_FORMATS)
def test_crops_and_letterboxes_of_the_same_size(src):
    w, h = 150, 9
    img = occ.noise(src, w, h, 5)
    for crop in ((2, 1, 131, 6), (3, 2, 130, 5), (1, 0, 133, 9), (8, 4, 128, 4)):
        for dst in (cc.NV12, cc.RGB8, cc.RGBA8, cc.UYVY, cc.I420, cc.MONO16):
            dw = crop[2] & ~1 if dst in PACKED else crop[2]
            p = cc.params(cc.BT601, cc.FULL, cc.BILINEAR, crop=(crop[0], crop[1], dw, crop[3]))
            assert expect_same(img, src, w, h, dst, dw, crop[3], p, offsets=(1, 2)) == 0, (crop, dst)
            boxed = cc.params(cc.BT709, mode=cc.AREA, crop=(crop[0], crop[1], dw, crop[3]), letterbox=True, fill_rgb=(20, 200, 90))
            assert expect_same(img, src, w, h, dst, dw, crop[3] + 7, boxed) == 0, (crop, dst, "bars above and below")
            assert expect_same(img, src, w, h, dst, dw + 14, crop[3], boxed, offsets=(0, 1)) == 0, (crop, dst, "bars at the sides")
