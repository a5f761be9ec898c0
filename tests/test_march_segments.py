"""How the velocity march cuts the x axis, from the rule's own source compiled for the host: the count of the least cost,
found without trying every count, and never more blocks than a launch may have."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_the_segments_are_those_of_the_least_cost(tmp_path):
    exe = tmp_path / "march_segments_check"
    build = subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "plume_b200" / "csrc"), "-o", str(exe),
                            str(ROOT / "tests" / "native" / "march_segments_check.cpp")], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    differ, blocks, ms = (float(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert differ == 0
    assert blocks <= 65535
    assert ms < 400  # 100 calls at 2^22 planes: about 4000 lengths each, against a million counts
