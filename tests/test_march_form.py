"""Which form of the velocity march a call takes, from the rule's own source compiled for the host: a time step that is
infinite or no number never reaches the forms that index on-chip memory by a trace of zero velocity."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_steps_that_are_not_finite_take_the_long_form(tmp_path):
    exe = tmp_path / "march_form_check"
    build = subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "plume_b200" / "csrc"), "-o", str(exe),
                            str(ROOT / "tests" / "native" / "march_form_check.cpp")], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    cells = [(38, 48, 38), (128, 192, 128), (1, 2, (1 << 22) - 1), ((1 << 22) - 2, 1, 1)]
    calls = [(*c, dt, chosen) for c in cells for dt in ("inf", "-inf", "nan", "0.5", "-1e30", "3e38") for chosen in (0, 1, 2, 3)]
    forms = subprocess.run([str(exe), *(str(x) for call in calls for x in call)], capture_output=True, text=True, check=True).stdout
    for (n0, n1, n2, dt, chosen), form in zip(calls, forms.split(), strict=True):
        by_size = 2 if n0 * n1 * n2 >= 2_000_000 else 1
        long_form = dt in ("inf", "-inf", "nan") or max(n0, n1, n2) >= (1 << 22) - 1
        assert int(form) == (3 if long_form else chosen or by_size), (n0, n1, n2, dt, chosen)
