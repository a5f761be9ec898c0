"""A kernel's shared memory limit belongs to the device that was current when it was set: the fused marches set theirs on
every device they run on, through a helper whose own source is compiled here for the host."""

import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_device_is_set_up_once(tmp_path):
    exe = tmp_path / "once_per_device_check"
    build = subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", str(ROOT / "plume_b200" / "csrc"), "-o", str(exe),
                            str(ROOT / "tests" / "native" / "once_per_device_check.cpp")], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == ""


def test_the_marches_remember_their_set_up_by_device():
    source = (ROOT / "plume_b200" / "csrc" / "advect.cu").read_text()
    flags = re.findall(r"static (\w+) configured\[", source)
    assert flags and set(flags) == {"OncePerDevice"}
