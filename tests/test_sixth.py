"""The exact form's division by six (host build of the device code) against the IEEE one."""
import subprocess
from pathlib import Path

import pytest


@pytest.mark.parametrize("numb", ["double", "float"])
def test_sixth_is_the_division_bit_for_bit(numb, tmp_path):
    """float: every positive bit pattern; double: every exponent with 60,000 mantissas, among them
    the neighbours of rounding boundaries, both signs, subnormals, infinities and NaN."""
    root = Path(__file__).resolve().parents[1]
    exe = tmp_path / "sixth"
    flags = ["-DUCB_NUMB_F32"] if numb == "float" else []
    subprocess.run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", *flags,
                    f"-I{root / 'u-cuda_b200' / 'csrc' / 'kernels'}", str(root / "tests" / "sixth_driver.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.stdout == "same\n" and out.returncode == 0, out.stdout
