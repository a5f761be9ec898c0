"""The one-launch pressure solve divides by a coupling sum (or a cell volume) as a product with its double
reciprocal. That this is the IEEE quotient is a property of the arithmetic, checked here on the host CPU with the
same operations; the device kernel is held to the same floats by the solver's parity tests."""

import shutil
import subprocess
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent / "native" / "quotient_check.c"


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_the_product_with_a_double_reciprocal_is_the_ieee_quotient(tmp_path):
    exe = tmp_path / "quotient_check"
    flags = ["-O2", "-ffp-contract=off", "-fno-fast-math"]
    build = subprocess.run(["gcc", *flags, "-mfma", "-o", str(exe), str(SOURCE), "-lm"], capture_output=True, text=True)
    if build.returncode != 0:  # a host without FMA instructions still has a correctly rounded libm fma
        build = subprocess.run(["gcc", *flags, "-o", str(exe), str(SOURCE), "-lm"], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    bad, bad_subnormal, checked = (int(x) for x in out)
    assert checked > 150_000_000
    assert bad == 0, f"{bad} of {checked} quotients differ from IEEE division"
    assert bad_subnormal == 0, f"{bad_subnormal} of {checked} subnormal quotients differ from IEEE division"
