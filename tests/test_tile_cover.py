"""CPU: the plan's tiles, slabs, scratch points and copies (tile_cover_check.cpp)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sympygr_b200", "csrc")


def test_tiles_cover_blocks_and_copies_stay_inside(tmp_path):
    exe = str(tmp_path / "tile_cover_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, os.path.join(HERE, "tile_cover_check.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout
