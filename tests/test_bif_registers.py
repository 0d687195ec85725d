"""max_registers reaches a diagram's kernel, also where two warps share 32 points: read from the
compiler's own report, in a child process with a fresh CUBIN cache."""
import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CODE = f"""
import sys
sys.path.insert(0, {str(ROOT / 'u-cuda_b200')!r}); sys.path.insert(0, {str(ROOT / 'tests')!r})
import ucb
from helpers import HYPER_ROSSLER, rk4_body
n, block, cap = map(int, sys.argv[1:])
ucb.precompile(ucb.Engine.bif1d_request(rk4_body(HYPER_ROSSLER), 4, (-10.0, -6.0, 0.0, 10.0), (0, 0.25, 0.05), n_pts=n,
                                        param_index=1, param_lo=0.24, param_hi=0.26, h=0.01, t_max=10.0,
                                        opt=ucb.options(precision=ucb.PREC_F64, block_threads=block,
                                                        max_registers=cap)))
"""


def registers(cache, n, block, cap):
    env = dict(os.environ, UCB_PTXAS_VERBOSE="1", UCB_CUBIN_CACHE=str(cache))
    r = subprocess.run([sys.executable, "-c", CODE, str(n), str(block), str(cap)], env=env, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return int(re.search(r"entry function 'ucb_bif_kernel'.*?Used (\d+) registers", r.stderr, re.S).group(1))


@pytest.mark.parametrize("n", [1000, 20000])  # two warps for 32 points; one
@pytest.mark.parametrize("block", [0, 64])
def test_cap_is_kept(n, block, tmp_path):
    free = registers(tmp_path / "free", n, block, 0)
    cap = 64
    assert free > cap
    assert registers(tmp_path / "cap", n, block, cap) <= cap
