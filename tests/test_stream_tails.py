"""The register of each stream's last frame, which decides whether a frame may
start under the end of the one before it: compiled with g++ and run without a GPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_register_of_last_frames(tmp_path):
    exe = str(tmp_path / "tails_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-pthread",
                    "-I", os.path.join(ROOT, "holoscan-zozo-modules_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "tails_check.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout
