"""The peak finder that decides a chunk of samples at a time (host build of the device code)
against the reference's loop over the whole series."""
import subprocess
from pathlib import Path

import pytest


@pytest.mark.parametrize("numb", ["double", "float"])
def test_chunked_peaks_equal_the_whole_series(numb, tmp_path):
    """Lengths across several chunk edges; smooth, noisy, alternating and flat series,
    plateaus that span chunks, differences at the threshold, infinities and NaN."""
    root = Path(__file__).resolve().parents[1]
    exe = tmp_path / "peak_chunks"
    flags = ["-DNUMB=float"] if numb == "float" else []
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", *flags,
                    f"-I{root / 'u-cuda_b200' / 'csrc' / 'kernels'}", str(root / "tests" / "peak_chunks_driver.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert int(out.stdout) == 130 * 8 * 20
