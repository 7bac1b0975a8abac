"""Bands of a batch's statistics pass that share a lens shading table: the rule
(compiled with g++, without a GPU), and batches whose grids overrun the table in a
long band, and in a single tile, against the oracle."""
import os
import subprocess

import numpy as np
import pytest

import isp_b200
import oracle
from isp_b200 import abi, scene

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_band_fits_its_table(tmp_path):
    exe = str(tmp_path / "bands_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror",
                    "-I", os.path.join(ROOT, "holoscan-zozo-modules_b200", "csrc"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "bands_check.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("balance", [abi.GRAY_WORLD, abi.WHITE_PATCH])
def test_grids_that_overrun_the_table(balance):
    """2048x2046 cameras in turn with 13, 33 and 256 grid rows."""
    from gpu_support import DeviceFrame, same_bits, torch_cuda

    torch = torch_cuda()
    w, h, exposure = 2048, 2046, (8_000_000, 1.5)
    data, pitch = scene.pack(scene.mosaic_counts(w, h, abi.GRBG, 256.0, 4095, 12, 5), abi.U16)
    raw = abi.RawFrame(data, w, h, pitch, abi.U16, 12, abi.GRBG)
    params = []
    for rows in (13, 33, 256):
        rng = np.random.default_rng(rows)
        gains = rng.uniform(1.0, 2.0, rows * 9 * 4).astype(np.float32)
        params.append(abi.IspParams(black_level=256.0, lens_shading=abi.LensShading(9, rows, 4, gains),
                                    white_balance=balance, demosaic=abi.BILINEAR, ccm=scene.CCM))
    want = [oracle.OraclePipeline(p).process(raw, abi.RGB8, True, exposure) for p in params]
    cameras = [isp_b200.Pipeline(params[i % 3]) for i in range(6)]
    frames = [DeviceFrame(raw, abi.RGB8, True) for _ in cameras]
    batch = isp_b200.Batch(len(cameras))
    for camera, f in zip(cameras, frames):
        rv, ov = f.views()
        batch.add(camera, rv, ov, f.hist.data_ptr(), f.stats.data_ptr(), exposure)
    batch.launch(0)
    torch.cuda.synchronize()
    for i, f in enumerate(frames):
        got = f.result()
        assert same_bits(got.stats, want[i % 3].stats), i
        assert same_bits(got.image, want[i % 3].image), i
        assert np.array_equal(got.histogram, want[i % 3].histogram), i
    batch.close()
