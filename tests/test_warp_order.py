"""A warp's digit ranks hold whatever order its lanes run in between the
points where the code makes them meet: the step is compiled for the host, its
lanes taking turns there."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def warp(tmp_path_factory):
    exe = tmp_path_factory.mktemp("warp") / "digit_ranks"
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", str(ROOT / "neslgpu_gb300" / "csrc"),
                    str(ROOT / "tests" / "warp" / "digit_ranks.cpp"), "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("order", ["drawn", "descending"])
@pytest.mark.parametrize("digits", [1, 2, 5, 40, 256])
def test_digit_ranks_in_any_order_of_the_lanes(warp, digits, order):
    out = subprocess.run([str(warp), str(digits), order], capture_output=True, text=True, check=True, timeout=120)
    assert int(out.stdout) == 0
