"""The clustering's parts of a square's extent (csrc/heavy_parts.h): every coordinate of the extent has
a part of [0, 16), whatever its width, on the host and through a whole clustering."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import oracle as O

DRIVER = r"""
#include <cmath>
#include <cstdio>
#include "heavy_parts.h"
int main() {
    using namespace ucbbr;
    const double widths[] = {0.0, 5e-324, 1e-323, 1e-310, 2.2250738585072014e-308, 8.9002954340288055e-308, 8.91e-308,
                             1e-300, 1e-100, 0.35, 1.0, 1e130};
    int n = 0;
    for (double w : widths) {
        const double s = part_scale(w);
        int last = 0;
        for (int k = 0; k <= 64; ++k) {
            const double offset = k == 64 ? w : w * (k / 64.0);
            const int i = part_index(offset, s);
            if (i < 0 || i >= kSub || i < last) return std::printf("width %g offset %g: part %d\n", w, offset, i), 1;
            last = i;
            ++n;
        }
        if (s > 0 && last != kSub - 1) return std::printf("width %g: the far end in part %d\n", w, last), 1;
        if (!(s >= 0 && std::isfinite(s))) return std::printf("width %g: scale %g\n", w, s), 1;
    }
    std::printf("%d\n", n);
}
"""


def test_every_coordinate_has_a_part(tmp_path):
    src = tmp_path / "parts.cpp"
    src.write_text(DRIVER)
    csrc = Path(__file__).resolve().parents[1] / "u-cuda_b200" / "csrc"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{csrc}", str(src), "-o", str(tmp_path / "parts")], check=True)
    out = subprocess.run([str(tmp_path / "parts")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert int(out.stdout) == 12 * 65


@pytest.mark.gpu
@pytest.mark.parametrize("width", [0.0, 5e-324, 1e-310, 1e-307, 1e-300])
@pytest.mark.parametrize("gap", [1.0 - 1e-6, 1.02])
@pytest.mark.parametrize("axis", [0, 1])
def test_spot_of_subnormal_width(width, gap, axis):
    """Half of the cells rest within `width` of the origin, the others on an arc about eps around it:
    heavy pairs of squares, one of them narrower than its parts' scale can say."""
    import ucb

    n, eps = 40, 0.5
    m = n * n
    rng = np.random.default_rng(7)
    phi = rng.uniform(0, 2 * np.pi, m)
    arc = np.arange(m) % 2 == 1
    r = gap * eps * (1 + 1e-3 * rng.random(m))
    f = [np.where(arc, r * np.cos(phi), 0.0), np.where(arc, r * np.sin(phi), 0.0)]
    f[axis] = np.where(arc, f[axis], width * rng.random(m))
    f[axis][0], f[axis][2] = 0.0, width
    cls = np.ones(m, dtype=np.int32)
    eng = ucb.Engine(0)
    lab, _ = eng.run_basins_recluster("x", 3, n, eps, f[0], f[1], cls, opt=ucb.options(precision=ucb.PREC_F64))
    eng.close()
    np.testing.assert_array_equal(lab, O.dbscan_cells(f[0], f[1], cls, eps, "f64"))
