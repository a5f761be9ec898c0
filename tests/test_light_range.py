"""The light march reads without a clamp only where a rule says that every sample lies inside the grid. The rule's own
source is compiled for the host and held to the sample points as the kernel computes them."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_sample_read_without_a_clamp_is_inside(tmp_path):
    exe = tmp_path / "light_range_check"
    build = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "plume_b200" / "csrc"), "-o",
                            str(exe), str(ROOT / "tests" / "native" / "light_range_check.cpp")], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    bad, with_runs, marches = (int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert marches > 500_000 and with_runs > marches // 4
    assert bad == 0, f"{bad} of {with_runs} marches read outside the grid"
