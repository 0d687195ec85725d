"""The period count of a 2-D bifurcation cell: the device's sorted form of the reference's
per-cell dbscan against its scans, on the host."""
import subprocess
from pathlib import Path

import pytest


@pytest.mark.parametrize("numb", ["double", "float"])
def test_sorted_dbscan_equals_the_scans(numb, tmp_path):
    """Sorted ranges with the visits replayed on bit sets against the scans over all peaks:
    sizes around warps and words and up to the cap, repeats, chains, distances at eps,
    signed zeros, infinities and NaN."""
    root = Path(__file__).resolve().parents[1]
    exe = tmp_path / "dbscan1d"
    flags = ["-DNUMB=float", "-DUCB_NUMB_F32"] if numb == "float" else []
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", *flags,
                    f"-I{root / 'u-cuda_b200' / 'csrc' / 'kernels'}", str(root / "tests" / "dbscan1d_driver.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), "7"], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert int(out.stdout) == 600 * 7
