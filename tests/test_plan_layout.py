"""CPU: how plans cut blocks into slabs and chunks, and the scratch they need (plan_layout_check.cpp)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def layout_check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("layout") / "plan_layout_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-I", os.path.join(REPO, "sympygr_b200", "csrc"), "-I", os.path.join(REPO, "include"),
                    os.path.join(HERE, "plan_layout_check.cpp"), "-o", exe], check=True)
    return exe


# limits: no plan is refused whose slabs of the depth asked for (48 planes by default) fit, none is
# accepted whose slabs do not; points: tiles and algebra tasks agree on every point's scratch point;
# strips: the same with planes larger than the scratch; whole: blocks that fit a chunk are not split;
# memory: scratch buffers hold no more points than asked for, the tiles' padding among them
@pytest.mark.parametrize("check", ["limits", "points", "strips", "whole", "memory"])
def test_plan_layout(layout_check, check):
    res = subprocess.run([layout_check, check], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout
